// Kirchhoff depth migration in the image domain (the reference's IDKDM,
// src/migration/KDM.cu:3-55 + IDKDM.cu:19-22) on traveltime tables kept on the
// device, and the wavelet cross-correlation of its input traces
// (Migration::set_wavelet + adjoint_convolution, migration.cu:54-71,
// :173-228).
//
// The reference launches image_domain_adjoint_kernel (migration.cu:398-483)
// once per source-receiver trace over the whole grid and adds each trace's
// term with atomicAdd; a cell is touched by one thread per launch, so the
// image is the FP32 sum of the traces' terms in trace order (source outer,
// receiver inner). Here what a term takes from one table is computed once per
// table and cell (k_table_terms), and a CTA owns 32 image cells: its warps form
// the traces' terms side by side and one of them adds them in that order
// (k_kirchhoff_image): the same sum, without atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "sf_engine.h"

using namespace sf;

#define CK(call)                                                          \
    do {                                                                  \
        int _st = sf_cuda_check(c, (call), #call);                        \
        if (_st != SF_OK) return _st;                                     \
    } while (0)

namespace {

constexpr float kEps = 1e-6f;  // EPS of migration.cuh:7
constexpr size_t kTermBytes = (size_t)4 << 30;  // workspace of the tables' terms (TermTable): blocks of cells or tables that fit

// The reference adds each term with a global float atomicAdd, which flushes
// subnormal operands and results to zero; the gather adds the same way.
__device__ __forceinline__ float add_ftz(float a, float b)
{
    float r;
    asm("add.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The part of a cell's weight that depends on one table only, as the
// reference's four Kirchhoff kernels compute it (migration.cu:418-466,
// :505-553, :592-640, :685-733) for the source's and the receiver's table of
// every trace: the time, the gradient norm, the Hessian's determinant, the
// angle to the vertical, the direction's cosine to it (signed), the spreading
// term, and the gradient.
struct CellTerms {
    float T, norm, detH, theta;
    float u, R, dx1, dz1;
};

// The terms of a call's tables at a block of model cells (rows iz0 .. iz0+nr-1
// of columns jx0 .., z fastest) are computed once (k_table_terms), 32 bytes per
// table and cell, 24 without the gradient: a trace then costs a cell the
// products of two tables' terms instead of both tables' stencils, roots,
// divisions and arc cosines.
struct TermTable {
    float4* a;         // T, norm, detH, theta; table t, cell q of the block at t * n + q
    float2* b;         // u, R
    float2* g;         // dx1, dz1 (the angle operators only)
    size_t n;          // cells of the block
    int iz0, nr, jx0;
};

template <bool GRAD>
__device__ __forceinline__ CellTerms load_terms(const TermTable& q, size_t t, size_t cell)
{
    const size_t o = t * q.n + cell;
    const float4 a = __ldg(q.a + o);
    const float2 b = __ldg(q.b + o), g = GRAD ? __ldg(q.g + o) : make_float2(0.0f, 0.0f);
    return CellTerms{a.x, a.y, a.z, a.w, b.x, b.y, g.x, g.y};
}

// Centred first and second differences of one table at padded node (i, j),
// gradient norm, unit direction (migration.cu:418-450). blockIdx.y strides over
// the tables (the sources' first), blockIdx.x over the cells. GRAD: the
// gradients too (the angle operators).
template <bool GRAD>
__global__ void k_table_terms(const float* __restrict__ S, const float* __restrict__ Ts, const float* __restrict__ Tr,
                              int nsrc, int ntab, int nxx, int nzz, int nb, float dx, float dz, bool fast, TermTable out)
{
    const size_t matsize = (size_t)nzz * nxx;
    for (int t = blockIdx.y; t < ntab; t += gridDim.y) {
        const float* T = (t < nsrc) ? Ts + matsize * t : Tr + matsize * (t - nsrc);
        for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < out.n; q += (size_t)gridDim.x * blockDim.x) {
            const unsigned col = (unsigned)q / (unsigned)out.nr;  // (a block's cells fit 32 bits)
            const int i = out.iz0 + (int)((unsigned)q - col * out.nr) + nb, j = out.jx0 + (int)col + nb;
            const float* c0 = T + i + (size_t)j * nzz;
            const float c = c0[0];
            const float zp = c0[1], zm = c0[-1];
            const float xp = c0[nzz], xm = c0[-nzz];
            float d_dz = 0.5f * (zp - zm) / dz;
            float d_dx = 0.5f * (xp - xm) / dx;
            float d2_dz2 = (zp - 2.0f * c + zm) / (dz * dz);
            float d2_dx2 = (xp - 2.0f * c + xm) / (dx * dx);
            float d2_dxdz = (c0[nzz + 1] - c0[nzz - 1] - c0[1 - nzz] + c0[-1 - nzz]) / (4.0f * dx * dz);
            // the multiply-adds the reference build fuses, written out
            const float norm = __fadd_rn(__fsqrt_rn(__fmaf_rn(d_dz, d_dz, __fmul_rn(d_dx, d_dx))), kEps);
            const float det = __fmaf_rn(d2_dx2, d2_dz2, -__fmul_rn(d2_dxdz, d2_dxdz));
            const float u = -(d_dz / norm);  // the direction's product with (0, -1)
            const float theta = acosf(min(1.0f, max(-1.0f, u)));
            const float Sc = S[i + (size_t)j * nzz];
            float R = max(c / Sc, kEps);
            const float detH = fabsf(det) + kEps;
            // every factor well inside FP32's range (their minima are EPS): the
            // weight's roots and quotients may take the fast form (fast: it was
            // found exact, fast_form). A negative R marks a cell where they may not.
            const bool regular = fast && norm < 1e6f && detH < 1e10f && R < 1e10f && fabsf(u) > 1e-12f && fabsf(u) < 2.0f &&
                                 fabsf(c) < 1e10f && Sc > 1e-9f && Sc < 1e9f;
            if (!regular) R = -R;
            const size_t o = (size_t)t * out.n + q;
            out.a[o] = make_float4(c, norm, detH, theta);
            out.b[o] = make_float2(u, R);
            if (GRAD) out.g[o] = make_float2(d_dx, d_dz);
        }
    }
}

// The exponent of a trace's taper at a cell: x - cmp over the aperture width
// tan(aperture) z + EPS (rwidth = RN(1/width); the fast quotient where both
// are in range).
__device__ __forceinline__ float taper_exponent(float x, float cmp, float width, float rwidth)
{
    const float d = __fsub_rn(x, cmp);
    const bool fast = width >= 1e-7f && width < 1e12f && fabsf(d) < 1e12f;  // a quotient below FP32's range gives taper 1 anyhow
    const float q = fast ? fdiv_k<false>(d, width, rwidth) : __fdiv_rn(d, width);
    return __fmul_rn(__fmul_rn(-0.5f, q), q);
}

// The cosine of the angle between two tables' gradients, with the multiply-add
// the reference build fuses.
__device__ __forceinline__ float gradient_cosine(const CellTerms& s, const CellTerms& r)
{
    const float dot = __fmaf_rn(s.dz1, r.dz1, __fmul_rn(s.dx1, r.dx1)), nn = __fmul_rn(s.norm, r.norm);
    return (fminf(s.R, r.R) > 0.0f) ? fdiv_k<false>(dot, nn, frcp_k(nn)) : __fdiv_rn(dot, nn);  // regular cells
}

// floor(angle / da): the angle bin (rda = RN(1/da), 0 where the quotient
// needs IEEE division).
__device__ __forceinline__ int angle_bin(float deg, float da, float rda)
{
    return __float2int_rd(rda > 0.0f ? fdiv_k<false>(deg, da, rda) : __fdiv_rn(deg, da));
}

// A cell's weight for a trace from both tables' terms. REGULAR: both cells are
// (k_table_terms); roots and quotients are Markstein corrections (sf_device.cuh)
// with IEEE's bits, without the branches of the general ones.
template <bool REGULAR>
__device__ __forceinline__ float kirchhoff_weight(const CellTerms& s, const CellTerms& r, float Sc, float texp)
{
    const float num = __fmul_rn(fsqrt_k<!REGULAR>(__fmul_rn(s.detH, r.detH)), Sc);
    const float nn = __fmul_rn(s.norm, r.norm), RR = __fmul_rn(s.R, r.R);
    const float Jterm = REGULAR ? fdiv_k<false>(num, nn, frcp_k(nn)) : __fdiv_rn(num, nn);
    const float cos_s = fabsf(s.u), cos_r = fabsf(r.u);
    const float obliquity = fsqrt_k<!REGULAR>(__fmul_rn(max(0.0f, cos_s), max(0.0f, cos_r)));
    const float rR = fsqrt_k<!REGULAR>(REGULAR ? RR : __fmul_rn(fabsf(s.R), fabsf(r.R)));
    const float G = REGULAR ? frcp_k(rR) : __fdiv_rn(1.0f, rR);
    const float theta = 0.5f * (s.theta + r.theta);
    const float R = 1.0f + 0.2f * cosf(theta);
    const float scale_const = 1.0f / (2.0f * M_PI);
    const float taper = expf(texp);
    return scale_const * Jterm * obliquity * G * R * taper;
}

// weight * v, the term that a trace adds at a cell x of aperture width `width`
// (rwidth: its reciprocal, at a regular cell by the fast form).
__device__ __forceinline__ float kirchhoff_term(const CellTerms& s, const CellTerms& r, float Sc, float x, float cmp,
                                                float width, float rwidth, float v)
{
    if (fminf(s.R, r.R) > 0.0f) {
        // expf underflows to 0 below this exponent (half the smallest subnormal is
        // exp(-103.98)): outside the trace's aperture, most of a shallow row, a
        // finite sample's term is 0
        const float texp = taper_exponent(x, cmp, width, rwidth);
        if (texp < -106.0f && fabsf(v) < 1e30f) return 0.0f;
        return __fmul_rn(kirchhoff_weight<true>(s, r, Sc, texp), v);
    }
    return __fmul_rn(kirchhoff_weight<false>(s, r, Sc, taper_exponent(x, cmp, width, __frcp_rn(width))), v);
}

// floor(T / dt): the sample of a time (rdt: sample_rate's).
__device__ __forceinline__ int sample_of(float T, float dt, float rdt)
{
    const float q = fdiv_k<false>(T, dt, rdt);
    return __float2int_rd((rdt > 0.0f && T > 1e-20f && T < 1e20f) ? q : T / dt);
}
// RN(1/dt), or 0 for steps so far out that the quotient needs IEEE division.
float sample_rate(float dt) { return (dt > 1e-15f && dt < 1e15f) ? 1.0f / dt : 0.0f; }

// RN(RN64(180 a / pi)), the angle in degrees as the reference's double
// expression rounds it, without the GPU's slow FP64 pipe: x / pi as x times a
// two-term reciprocal (relative error below 2^-45). Where the second term,
// moved by 2^-18 of itself either way, rounds differently, the quotient lies
// too near a rounding boundary and the double expression decides.
__device__ __forceinline__ float degrees_of(float a)
{
    const float x = 180.0f * a;
    const float hi = 0.318309873f;                    // RN(1/pi)
    const float lo = (float)(1.0 / M_PI - (double)0.318309873f);
    const float h = __fmul_rn(x, hi);
    const float e = __fmaf_rn(x, lo, __fmaf_rn(x, hi, -h));
    const float d = __fmul_rn(e, 3.8146973e-6f);      // 2^-18
    const float r1 = __fadd_rn(h, __fadd_rn(e, d)), r2 = __fadd_rn(h, __fsub_rn(e, d));
    if (r1 == r2) return r1;
    return (float)((double)x / M_PI);
}

struct KirchParams {
    const float* S;     // padded slowness
    TermTable tab;      // nsrc source tables, then nrec receiver tables
    const float* xs;    // nsrc
    const float* xr;    // nrec
    const float* data;  // nsrc x nrec x nt correlated traces
    float* image;       // nz x nx
    int nsrc, nrec, nt, nzz, nb;
    float dt, rdt, dx, dz, aperture, max_offset;  // rdt: sample_rate(dt)
};

// The image cells of the block (whole columns), 32 per CTA. The image is the
// sum of the traces' terms in trace order; a CTA's warps compute the terms of a
// source's receivers side by side (a warp takes every kImageWarps-th receiver
// for the 32 cells), and one of them adds them to the cells in receiver order
// while the others go on to the next. So few cells are in flight that the
// terms of their receivers stay in L1 and L2 from source to source: with a
// thread per cell every source streamed all tables' terms from DRAM (0.58 GB
// for 120 tables at 1001 x 201 cells; a migration of 20 x 100 traces there took
// 2.38 ms, 2.04 this way; 1.99 today, of which this kernel is 1.57).
constexpr int kImageWarps = 8;
constexpr int kImageRec = 128;   // receivers whose terms are buffered

__global__ void __launch_bounds__(32 * kImageWarps) k_kirchhoff_image(KirchParams p)
{
    __shared__ float term[2][kImageRec][32];
    __shared__ float sum[32];
    const int nz = p.nzz - 2 * p.nb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (size_t q0 = (size_t)blockIdx.x * 32; q0 < p.tab.n; q0 += (size_t)gridDim.x * 32) {
        const size_t q = min(q0 + lane, p.tab.n - 1);  // lanes past the end repeat the last cell
        const unsigned col = (unsigned)q / (unsigned)nz;
        const int i = (int)((unsigned)q - col * nz) + p.nb, j = p.tab.jx0 + (int)col + p.nb;
        const float z = __int2float_rd(i - p.nb) * p.dz;
        const float x = __int2float_rd(j - p.nb) * p.dx;
        const float Sc = p.S[(size_t)i + (size_t)j * p.nzz];
        const float width = __fmaf_rn(tanf(p.aperture * M_PI / 180.0f), z, kEps);  // fused in the reference's image kernel
        const float rwidth = __frcp_rn(width);
        if (warp == 0) sum[lane] = 0.0f;
        int buf = 0, turn = 0;
        for (int s = 0; s < p.nsrc; s++) {
            const CellTerms ts = load_terms<false>(p.tab, s, q);
            const float xs = p.xs[s];
            for (int r0 = 0; r0 < p.nrec; r0 += kImageRec) {
                const int n = min(kImageRec, p.nrec - r0);
#pragma unroll 2
                for (int k = warp; k < n; k += kImageWarps) {
                    const int r = r0 + k;
                    const float xr = p.xr[r];
                    float v = 0.0f;  // a trace left out adds nothing
                    if (fabsf((xs - xr)) < p.max_offset) {
                        const CellTerms tr = load_terms<false>(p.tab, (size_t)p.nsrc + r, q);
                        const int tId = sample_of(ts.T + tr.T, p.dt, p.rdt);
                        if ((unsigned)tId < (unsigned)p.nt)
                            v = kirchhoff_term(ts, tr, Sc, x, 0.5f * (xs + xr), width, rwidth,
                                               p.data[((size_t)s * p.nrec + r) * p.nt + tId]);
                    }
                    term[buf][k][lane] = v;
                }
                // the terms are complete, and the warp that added the last ones is done
                __syncthreads();
                if (warp == turn) {
                    float acc = sum[lane];
#pragma unroll 8
                    for (int k = 0; k < n; k++) acc = add_ftz(acc, term[buf][k][lane]);
                    sum[lane] = acc;
                }
                buf ^= 1;
                turn = (turn + 1) % kImageWarps;
            }
        }
        __syncthreads();
        if (warp == 0 && q0 + lane < p.tab.n) p.image[(size_t)p.tab.jx0 * nz + q] = sum[lane];
        __syncthreads();
    }
}

// Correlation and convolution of traces with the wavelet, both in FP64 with
// the reference's order of the sum, rounded once to FP32: a block of threads
// takes kFilterBlock output samples of one trace from its input samples in
// shared memory as doubles. A product of two FP32 values is exact in FP64, so
// one fused multiply-add gives the bits of the multiplication and addition
// each rounded once. Two FP64 lanes per SM bound them: converting every tap's
// sample anew and multiplying and adding apart took three FP64 instructions a
// tap (2000 traces of 1000 samples, 58 taps: 0.67 ms), this takes one.
constexpr int kFilterBlock = 256;
constexpr int kFilterTaps = 1024;  // taps staged at a time

// Correlation, as the reference's FFT product A conj(B) with FFTW's
// unnormalised inverse gives it: for output sample t >= shift, nfft * sum_m
// trace[t - shift + m] * w[m] (the zero padding to nfft >= nt + nw - 1 makes
// the circular sum a linear one); samples before the shift are 0.
// Convolution (FORWARD), the product A B (Migration::forward_convolution,
// migration.cu:230-261): nfft * sum_m trace[t + shift - m] * w[m] over the
// samples inside the trace, m ascending.
template <bool FORWARD>
__global__ void __launch_bounds__(kFilterBlock) k_filter(const float* __restrict__ in, float* __restrict__ out, int ntr,
                                                         int nt, const double* __restrict__ w, int nw, int shift,
                                                         double nfft)
{
    __shared__ double sw[kFilterTaps], sa[kFilterTaps + kFilterBlock];
    const int nblk = (nt + kFilterBlock - 1) / kFilterBlock;
    const size_t njob = (size_t)ntr * nblk;
    for (size_t job = blockIdx.x; job < njob; job += gridDim.x) {
        const float* a = in + (job / nblk) * nt;
        const int t0 = (int)(job % nblk) * kFilterBlock, t = t0 + threadIdx.x;
        // the output's taps: input sample c - m (FORWARD) or c + m
        const int c = FORWARD ? t + shift : t - shift;
        const int m0 = FORWARD ? max(0, c - nt + 1) : 0;
        const int m1 = (t >= nt || c < 0) ? 0 : min(nw, FORWARD ? c + 1 : nt - c);
        double acc = 0.0;
        for (int mc = 0; mc < nw; mc += kFilterTaps) {
            const int mn = min(kFilterTaps, nw - mc);
            // samples of these taps from sample lo
            const int lo = FORWARD ? t0 + shift - (mc + mn - 1) : t0 - shift + mc;
            __syncthreads();
            for (int q = threadIdx.x; q < mn; q += kFilterBlock) sw[q] = w[mc + q];
            for (int q = threadIdx.x; q < mn + kFilterBlock - 1; q += kFilterBlock) {
                const int k = lo + q;
                sa[q] = (k >= 0 && k < nt) ? (double)a[k] : 0.0;
            }
            __syncthreads();
            const int first = max(m0, mc), last = min(m1, mc + mn);
            if (FORWARD) {
                const double* x = sa + (c - lo);
#pragma unroll 4
                for (int m = first; m < last; m++) acc = __fma_rn(x[-m], sw[m - mc], acc);
            } else {
                const double* x = sa + (c - lo);
#pragma unroll 4
                for (int m = first; m < last; m++) acc = __fma_rn(x[m], sw[m - mc], acc);
            }
        }
        if (t < nt) out[(job / nblk) * nt + t] = (m1 > 0 || FORWARD || c >= 0) ? __double2float_rn(__dmul_rn(acc, nfft)) : 0.0f;
    }
}

constexpr int kMaxAngles = 256;

struct AngleParams {
    const float* S;
    TermTable tab;          // rows of every column; nsrc source tables, then nrec receiver tables
    const float* xs;
    const float* xr;
    const float* data;      // nsrc x nrec x nt correlated traces
    const int* cmp_ptr;     // traces of CMP bin b: [cmp_ptr[b], cmp_ptr[b+1]) of cmp_tr
    const int* cmp_tr;      // trace s * nrec + r, trace order within a bin
    float* gathers;         // nz x nang x ncmp
    int nsrc, nrec, nt, nxx, nzz, nb, nang, ncmp;
    float dt, rdt, dx, dz, da, rda, aperture;  // rdt: sample_rate(dt); rda: angle_bin's
};

// ADKDM's angle_domain_adjoint_kernel (migration.cu:572-663) as a gather: one
// thread per (depth row, CMP bin) walks the bin's traces in trace order and,
// for each, the row's cells left to right, adding each term to its
// reflection-angle bin. The reference adds with atomics from all columns of a
// launch at once, so its order within a bin is not fixed; the terms are the
// same.
__global__ void k_kirchhoff_angles(AngleParams p)
{
    const int nz = p.nzz - 2 * p.nb;
    const size_t nthr = (size_t)p.tab.nr * p.ncmp;
    float acc[kMaxAngles];
    for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < nthr; w += (size_t)gridDim.x * blockDim.x) {
        const int ir = (int)(w % p.tab.nr), b = (int)(w / p.tab.nr);
        const int iz = p.tab.iz0 + ir, i = iz + p.nb;
        for (int a = 0; a < p.nang; a++) acc[a] = 0.0f;
        const float z = __int2float_rd(i - p.nb) * p.dz;
        const float width = __fadd_rn(__fmul_rn(tanf(p.aperture * M_PI / 180.0f), z), kEps);
        const float rwidth = __frcp_rn(width);
        for (int e = p.cmp_ptr[b]; e < p.cmp_ptr[b + 1]; e++) {
            const int tr_id = p.cmp_tr[e];
            const int s = tr_id / p.nrec, r = tr_id % p.nrec;
            const float cmp = 0.5f * (p.xs[s] + p.xr[r]);
            const float* trace = p.data + (size_t)tr_id * p.nt;
#pragma unroll 2
            for (int j = p.nb; j < p.nxx - p.nb; j++) {
                const size_t m = (size_t)ir + (size_t)(j - p.nb) * p.tab.nr;
                const CellTerms ts = load_terms<true>(p.tab, s, m), tr = load_terms<true>(p.tab, (size_t)p.nsrc + r, m);
                const float x = __int2float_rd(j - p.nb) * p.dx;
                const float T = ts.T + tr.T;
                const int tId = sample_of(T, p.dt, p.rdt);
                if ((unsigned)tId >= (unsigned)p.nt) continue;
                const float Sc = p.S[(size_t)i + (size_t)j * p.nzz];
                const float term = kirchhoff_term(ts, tr, Sc, x, cmp, width, rwidth, trace[tId]);
                const float reflection_angle = 0.5f * acosf(gradient_cosine(ts, tr));
                const int aId = angle_bin(degrees_of(reflection_angle), p.da, p.rda);
                if (aId >= 0 && aId < p.nang) acc[aId] = add_ftz(acc[aId], term);
            }
        }
        for (int a = 0; a < p.nang; a++) p.gathers[(size_t)iz + (size_t)a * nz + (size_t)b * p.nang * nz] = acc[a];
    }
}

struct KirchFwdParams {
    const float* S;
    TermTable tab;       // every cell; nsrc source tables from s0, then receiver tables from r0
    const float* xs;
    const float* xr;
    const float* model;  // image (nz x nx) or angle gathers (nz x nang x ncmp)
    const int* trace;    // work trace e -> s * nrec + r, in trace order
    const int* cmp;      // work trace e -> CMP bin (angle domain)
    float* part;         // ntrace x nchunk x nt partial traces (nchunk > 1)
    float* data;         // nsrc x nrec x nt
    int nchunk, chunk, s0, r0, nsrc, nrec, nt, nxx, nzz, nb, nang, warps;
    float dt, rdt, dx, dz, da, rda, aperture;  // rdt: sample_rate(dt); rda: angle_bin's
};

// The forward (demigration) operator of the least-squares variants:
// image_domain_forward_kernel / angle_domain_forward_kernel
// (migration.cu:485-570, :665-756) add weight * model[cell] to sample
// floor((Ts + Tr)/dt) of the trace with a global atomicAdd per cell, in no
// fixed order. Here one CTA takes one chunk of one trace's cells. Each warp
// walks 32 consecutive cells (z fastest) at a time; lanes that hit the same
// sample are summed in lane order and the sum is added to the warp's own
// histogram of the trace in shared memory (one adder per sample, no
// atomics). The warps' histograms are summed in warp order, the chunks in
// chunk order: a fixed order that depends only on the sizes, so the traces
// are reproducible bit for bit.
template <bool ANGLE>
__global__ void k_kirchhoff_forward(KirchFwdParams p)
{
    extern __shared__ float smem[];
    const int W = p.warps, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* hist = smem + (size_t)warp * p.nt;
    float* st_v = smem + (size_t)W * p.nt + warp * 32;
    for (int q = threadIdx.x; q < W * p.nt; q += blockDim.x) smem[q] = 0.0f;
    __syncthreads();
    const int e = blockIdx.x / p.nchunk, ck = blockIdx.x % p.nchunk;
    const int tid = p.trace[e], s = tid / p.nrec, r = tid % p.nrec;
    const float cmp = 0.5f * (p.xs[s] + p.xr[r]);
    const int cmpId = ANGLE ? p.cmp[e] : 0;
    const int nz = p.nzz - 2 * p.nb;
    const float tan_ap = tanf(p.aperture * M_PI / 180.0f);
    const long ncell = (long)nz * (p.nxx - 2 * p.nb);
    const long m0 = (long)ck * p.chunk, m1 = min(m0 + (long)p.chunk, ncell);
    // the lane's cell as (row, column), moved on by 32 W cells at a time
    const int step_i = (32 * W) % nz, step_j = (32 * W) / nz;
    const long first = m0 + 32L * warp + lane;
    int iz = (int)(first % nz), jx = (int)(first / nz);
    for (long g = m0 + 32L * warp; g < m1; g += 32L * W) {
        const long m = g + lane;
        int tq = -1;
        float v = 0.0f;
        if (m < m1) {
            const CellTerms ts = load_terms<ANGLE>(p.tab, s - p.s0, (size_t)m);
            const CellTerms tr = load_terms<ANGLE>(p.tab, (size_t)p.nsrc + (r - p.r0), (size_t)m);
            const float T = ts.T + tr.T;
            const int tId = sample_of(T, p.dt, p.rdt);
            if (tId >= 0 && tId < p.nt) {
                const float z = __int2float_rd(iz) * p.dz;
                const float x = __int2float_rd(jx) * p.dx;
                const float Sc = p.S[(size_t)(iz + p.nb) + (size_t)(jx + p.nb) * p.nzz];
                const float width = __fadd_rn(__fmul_rn(tan_ap, z), kEps);
                size_t mId = (size_t)m;
                bool in = true;
                if (ANGLE) {
                    const float reflection_angle = 0.5f * acosf(gradient_cosine(ts, tr));
                    const int aId = angle_bin(degrees_of(reflection_angle), p.da, p.rda);
                    in = aId >= 0 && aId < p.nang;
                    mId = (size_t)iz + (size_t)aId * nz + (size_t)cmpId * p.nang * nz;
                }
                if (in) {
                    v = kirchhoff_term(ts, tr, Sc, x, cmp, width, frcp_k(width), p.model[mId]);
                    if (v != 0.0f) tq = tId;  // (NaN is kept)
                }
            }
        }
        iz += step_i;
        jx += step_j;
        if (iz >= nz) {
            iz -= nz;
            jx++;
        }
        st_v[lane] = v;
        __syncwarp();
        const unsigned grp = __match_any_sync(0xffffffffu, tq);
        if (tq >= 0 && lane == __ffs(grp) - 1) {
            float sum = v;
            for (unsigned rest = grp & (grp - 1); rest; rest &= rest - 1) sum = add_ftz(sum, st_v[__ffs(rest) - 1]);
            hist[tq] = add_ftz(hist[tq], sum);
        }
        __syncwarp();
    }
    __syncthreads();
    float* out = (p.nchunk == 1) ? p.data + (size_t)tid * p.nt : p.part + ((size_t)e * p.nchunk + ck) * p.nt;
    for (int t = threadIdx.x; t < p.nt; t += blockDim.x) {
        float a = smem[t];
        for (int w = 1; w < W; w++) a = add_ftz(a, smem[(size_t)w * p.nt + t]);
        out[t] = a;
    }
}

// Chunk partials of each work trace summed in chunk order.
__global__ void k_sum_chunks(const float* __restrict__ part, const int* __restrict__ trace, float* __restrict__ data,
                             int ntrace, int nchunk, int nt)
{
    const size_t n = (size_t)ntrace * nt;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
        const int e = (int)(q / nt), t = (int)(q % nt);
        const float* pp = part + (size_t)e * nchunk * nt + t;
        float a = pp[0];
        for (int c = 1; c < nchunk; c++) a = add_ftz(a, pp[(size_t)c * nt]);
        data[(size_t)trace[e] * nt + t] = a;
    }
}

}  // namespace

// Migration::set_wavelet (migration.cu:54-71) as its source computes it.
void sf_kirchhoff_wavelet(float fmax, float dt, std::vector<float>& w)
{
    const float t0 = 2.0f * sqrtf(M_PI) / fmax;
    const float fc = fmax / (3.0f * sqrtf(M_PI));
    const int nw = 2 * ((int)((t0 - 0.5f * dt) / dt));
    w.assign(std::max(nw, 0), 0.0f);
    for (int k = 0; k < nw; k++) {
        const float td = k * dt - t0;
        const float arg = M_PI * M_PI * M_PI * fc * fc * td * td;
        w[k] = (1.0f - 2.0f * arg) * expf(-arg);
    }
}

static int next_pow2(int n)
{
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// The wavelet correlation (forward = false) or convolution (forward = true)
// of ntr traces, as Migration::adjoint_convolution / forward_convolution.
static int wavelet_filter(sf_ctx* c, const float* traces, float* out, int ntr, int nt, float dt, float fmax, int mem,
                          void* stream, bool forward)
{
    if (!c || !traces || !out || ntr < 0 || nt < 1 || !(dt > 0.0f) || !(fmax > 0.0f))
        return sf_fail(c, SF_ERR_ARG, "bad convolution arguments");
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    std::vector<float> wf;
    sf_kirchhoff_wavelet(fmax, dt, wf);
    const int nw = (int)wf.size();
    if (nw < 1) return sf_fail(c, SF_ERR_ARG, "wavelet shorter than one sample (fmax too high for dt)");
    c->h_wav.assign(wf.begin(), wf.end());  // FP64 copy of the FP32 samples
    const size_t nb = (size_t)ntr * nt * sizeof(float);
    int rc = sf_dev_reserve(c, (void**)&c->d_wav, &c->cap_wav, c->h_wav.size() * sizeof(double));
    if (!rc && mem == SF_MEM_HOST) rc = sf_dev_reserve(c, (void**)&c->d_mig, &c->cap_mig, 2 * nb + 16);
    if (rc) return rc;
    CK(cudaMemcpyAsync(c->d_wav, c->h_wav.data(), c->h_wav.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    const float* din = traces;
    float* dout = out;
    if (mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(c->d_mig, traces, nb, cudaMemcpyHostToDevice, st));
        din = c->d_mig;
        dout = c->d_mig + (size_t)ntr * nt;
    }
    const size_t n = (size_t)ntr * nt;
    if (n) {
        const double nfft = (double)next_pow2(nt + nw - 1);
        const size_t njob = (size_t)ntr * ((nt + kFilterBlock - 1) / kFilterBlock);
        const unsigned grid = (unsigned)std::min<size_t>(njob, (size_t)c->sms * 16);
        if (forward)
            k_filter<true><<<grid, kFilterBlock, 0, st>>>(din, dout, ntr, nt, c->d_wav, nw, nw / 2 + nw / 10, nfft);
        else
            k_filter<false><<<grid, kFilterBlock, 0, st>>>(din, dout, ntr, nt, c->d_wav, nw, nw / 2 + nw / 10, nfft);
        CK(cudaGetLastError());
    }
    if (mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(out, dout, nb, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return SF_OK;
}

extern "C" int sf_adjoint_convolution(sf_ctx* c, const float* traces, float* out, int ntr, int nt, float dt,
                                      float fmax, int mem, void* stream)
{
    return wavelet_filter(c, traces, out, ntr, nt, dt, fmax, mem, stream, false);
}

extern "C" int sf_forward_convolution(sf_ctx* c, const float* traces, float* out, int ntr, int nt, float dt,
                                      float fmax, int mem, void* stream)
{
    return wavelet_filter(c, traces, out, ntr, nt, dt, fmax, mem, stream, true);
}

// Whether the roots and reciprocals made from the hardware's approximations
// are IEEE's on this device (checked at the context's creation).
static bool fast_form(const sf_ctx* c) { return (c->kc.mflags & 0x30) == 0x30; }

// Bytes of the terms of `tables` tables at `cells` cells, with the gradients or without.
static size_t term_bytes(bool grad, size_t tables, size_t cells)
{
    return tables * cells * (sizeof(float4) + (grad ? 2 : 1) * sizeof(float2));
}

// One operator's use of the context's buffers on its stream, the workspace of
// the terms among them: after the operator before it, whatever its stream. A
// captured operator, whose replays no event of the context could order, has a
// workspace of its graph's.
class KirchCall {
public:
    KirchCall(sf_ctx* c, cudaStream_t st) : c_(c), st_(st) {}
    KirchCall(const KirchCall&) = delete;
    KirchCall& operator=(const KirchCall&) = delete;
    ~KirchCall()
    {
        if (own_) cudaFreeAsync(own_, st_);
        if (open_ && !capturing_) cudaEventRecord(c_->kirch_ev, st_);
    }
    int open()
    {
        int rc = sf_capturing(c_, st_, &capturing_);
        if (!rc) rc = sf_wait_slowness(c_, st_);
        if (rc) return rc;
        open_ = true;
        return capturing_ ? SF_OK : sf_cuda_check(c_, cudaStreamWaitEvent(st_, c_->kirch_ev, 0), "cudaStreamWaitEvent");
    }
    // The workspace; it comes after the operator's other buffers, whose
    // allocation may give it up (sf_dev_reserve).
    int reserve(size_t bytes)
    {
        if (c_->kterm_limit && bytes > c_->kterm_limit) return sf_fail(c_, SF_ERR_NOMEM, "workspace limit of a test");
        if (capturing_) return sf_cuda_check(c_, cudaMallocAsync(&own_, bytes, st_), "cudaMallocAsync");
        return sf_dev_reserve(c_, &c_->d_kterm, &c_->cap_kterm, bytes);
    }
    // The largest count of `each` bytes, at most `all`, that kTermBytes and the
    // device's memory allow, reserved: halved until its allocation succeeds.
    int reserve_blocks(int all, size_t each, int* count)
    {
        int n = (int)std::min<size_t>(all, std::max<size_t>(kTermBytes / each, 1));
        int rc;
        while ((rc = reserve(n * each)) == SF_ERR_NOMEM && n > 1) n = (n + 1) / 2;
        *count = n;
        return rc;
    }
    void* workspace() const { return capturing_ ? own_ : c_->d_kterm; }

private:
    sf_ctx* c_;
    cudaStream_t st_;
    bool capturing_ = false, open_ = false;
    void* own_ = nullptr;
};

// Terms of the tables at rows iz0 .. iz0+nr-1 of columns jx0 .. jx0+nc-1 into
// the call's workspace, which is large enough. grad: with the gradients.
static int table_terms(sf_ctx* c, const KirchCall& call, bool grad, const float* Ts, const float* Tr, int nsrc, int nrec,
                       int iz0, int nr, int jx0, int nc, TermTable* q, cudaStream_t st)
{
    const size_t ntab = (size_t)nsrc + nrec, n = (size_t)nr * nc;
    q->a = reinterpret_cast<float4*>(call.workspace());
    q->b = reinterpret_cast<float2*>(q->a + ntab * n);
    q->g = grad ? q->b + ntab * n : nullptr;
    q->n = n;
    q->iz0 = iz0;
    q->nr = nr;
    q->jx0 = jx0;
    const unsigned gx = (unsigned)std::min<size_t>((n + 127) / 128, 65535);
    (grad ? k_table_terms<true> : k_table_terms<false>)<<<dim3(gx, (unsigned)std::min<size_t>(ntab, 65535)), 128, 0, st>>>(
        c->d_S, Ts, Tr, nsrc, (int)ntab, c->nxx, c->nzz, c->nb, c->dx, c->dz, fast_form(c), *q);
    CK(cudaGetLastError());
    return SF_OK;
}

extern "C" int sf_kirchhoff_image(sf_ctx* c, const float* Ts, const float* Tr, int nsrc, int nrec, const float* xsrc,
                                  const float* xrec, const float* data, int data_mem, int nt, float dt,
                                  float aperture, float max_offset, float* image, int image_mem, void* stream)
{
    if (!c || !Ts || !Tr || !xsrc || !xrec || !data || !image || nsrc < 1 || nrec < 1 || nt < 1 || !(dt > 0.0f))
        return sf_fail(c, SF_ERR_ARG, "bad Kirchhoff arguments");
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    KirchCall call(c, st);
    const size_t nd = (size_t)nsrc * nrec * nt, ni = (size_t)c->nx * c->nz;
    int rc = call.open();
    if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_kgeo, &c->cap_kgeo, (size_t)(nsrc + nrec) * sizeof(float));
    if (!rc && (data_mem == SF_MEM_HOST || image_mem == SF_MEM_HOST))
        rc = sf_dev_reserve(c, (void**)&c->d_mig, &c->cap_mig, (nd + ni) * sizeof(float));
    if (rc) return rc;
    c->h_kgeo.assign(xsrc, xsrc + nsrc);
    c->h_kgeo.insert(c->h_kgeo.end(), xrec, xrec + nrec);
    CK(cudaMemcpyAsync(c->d_kgeo, c->h_kgeo.data(), c->h_kgeo.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    const float* dd = data;
    float* di = image;
    if (data_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(c->d_mig, data, nd * sizeof(float), cudaMemcpyHostToDevice, st));
        dd = c->d_mig;
    }
    if (image_mem == SF_MEM_HOST) di = c->d_mig + nd;
    KirchParams p;
    p.S = c->d_S;
    p.xs = c->d_kgeo;
    p.xr = c->d_kgeo + nsrc;
    p.data = dd;
    p.image = di;
    p.nsrc = nsrc;
    p.nrec = nrec;
    p.nt = nt;
    p.nzz = c->nzz;
    p.nb = c->nb;
    p.dt = dt;
    p.rdt = sample_rate(dt);
    p.dx = c->dx;
    p.dz = c->dz;
    p.aperture = aperture;
    p.max_offset = max_offset;
    // blocks of whole columns whose terms fit the workspace
    int cols;
    rc = call.reserve_blocks(c->nx, term_bytes(false, (size_t)nsrc + nrec, c->nz), &cols);
    if (rc) return rc;
    for (int j0 = 0; j0 < c->nx; j0 += cols) {
        const int nc = std::min(cols, c->nx - j0);
        rc = table_terms(c, call, false, Ts, Tr, nsrc, nrec, 0, c->nz, j0, nc, &p.tab, st);
        if (rc) return rc;
        k_kirchhoff_image<<<(unsigned)std::min<size_t>((p.tab.n + 31) / 32, (size_t)1 << 30), 32 * kImageWarps, 0, st>>>(p);
        CK(cudaGetLastError());
    }
    if (image_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(image, di, ni * sizeof(float), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return SF_OK;
}

// Migration::set_gathers (migration.cu:73-97): CMP spacing half the smaller of
// the first source and receiver spacings, bins from the smallest CMP of all
// pairs. The reference starts the largest CMP from an uninitialised value
// (it assigns minCMP twice); here it starts from the first pair's CMP.
static int angle_dims(const float* xsrc, int nsrc, const float* xrec, int nrec, float max_angle, float da,
                      int* nang, int* ncmp, float* mincmp, float* dcmp)
{
    if (nsrc < 2 || nrec < 2 || !(da > 0.0f)) return SF_ERR_ARG;
    const float ds = xsrc[1] - xsrc[0], dr = xrec[1] - xrec[0];
    const float d = 0.5f * std::min(ds, dr);
    if (!(d > 0.0f)) return SF_ERR_ARG;
    float mn = 1e6f, mx = 0.5f * (xsrc[0] + xrec[0]);
    for (int s = 0; s < nsrc; s++)
        for (int r = 0; r < nrec; r++) {
            const float cmp = 0.5f * (xsrc[s] + xrec[r]);
            mn = (cmp < mn) ? cmp : mn;
            mx = (cmp > mx) ? cmp : mx;
        }
    *nang = (int)(max_angle / da) + 1;
    *ncmp = (int)((mx - mn) / d) + 1;
    *mincmp = mn;
    *dcmp = d;
    return SF_OK;
}

extern "C" int sf_kirchhoff_angle_gathers(sf_ctx* c, const float* Ts, const float* Tr, int nsrc, int nrec,
                                          const float* xsrc, const float* xrec, const float* data, int data_mem, int nt,
                                          float dt, float aperture, float max_offset, float max_angle, float da,
                                          float* gathers, int gathers_mem, int* nang_out, int* ncmp_out, void* stream)
{
    if (!c || !xsrc || !xrec) return sf_fail(c, SF_ERR_ARG, "null argument");
    int nang, ncmp;
    float mincmp, dcmp;
    if (angle_dims(xsrc, nsrc, xrec, nrec, max_angle, da, &nang, &ncmp, &mincmp, &dcmp))
        return sf_fail(c, SF_ERR_ARG, "angle gathers need two sources, two receivers, increasing positions, da > 0");
    if (nang > kMaxAngles) return sf_fail(c, SF_ERR_RANGE, "more than 256 angle bins");
    if (nang_out) *nang_out = nang;
    if (ncmp_out) *ncmp_out = ncmp;
    if (!gathers) return SF_OK;  // dimensions only
    if (!Ts || !Tr || !data || nt < 1 || !(dt > 0.0f)) return sf_fail(c, SF_ERR_ARG, "bad Kirchhoff arguments");
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    // traces by CMP bin, trace order kept (KDM.cu:28-53)
    std::vector<int> cnt(ncmp + 1, 0), ids;
    std::vector<std::pair<int, int>> tr;
    for (int s = 0; s < nsrc; s++)
        for (int r = 0; r < nrec; r++) {
            if (!(fabsf(xsrc[s] - xrec[r]) < max_offset)) continue;
            const float cmp = 0.5f * (xsrc[s] + xrec[r]);
            const int b = (int)((cmp - mincmp) / dcmp);
            if (b < 0 || b >= ncmp) continue;
            tr.push_back({b, s * nrec + r});
            cnt[b + 1]++;
        }
    for (int b = 0; b < ncmp; b++) cnt[b + 1] += cnt[b];
    ids.resize(tr.size());
    {
        std::vector<int> fill(cnt.begin(), cnt.end() - 1);
        for (auto& t : tr) ids[fill[t.first]++] = t.second;
    }
    const size_t nd = (size_t)nsrc * nrec * nt, ng = (size_t)(c->nzz - 2 * c->nb) * nang * ncmp;
    c->h_kgeo.assign(xsrc, xsrc + nsrc);
    c->h_kgeo.insert(c->h_kgeo.end(), xrec, xrec + nrec);
    c->h_kint.assign(cnt.begin(), cnt.end());
    c->h_kint.insert(c->h_kint.end(), ids.begin(), ids.end());
    KirchCall call(c, st);
    int rc = call.open();
    if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_kgeo, &c->cap_kgeo, c->h_kgeo.size() * sizeof(float));
    if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_kint, &c->cap_kint, c->h_kint.size() * sizeof(int));
    if (!rc && (data_mem == SF_MEM_HOST || gathers_mem == SF_MEM_HOST))
        rc = sf_dev_reserve(c, (void**)&c->d_mig, &c->cap_mig, (nd + ng) * sizeof(float));
    if (rc) return rc;
    CK(cudaMemcpyAsync(c->d_kgeo, c->h_kgeo.data(), c->h_kgeo.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(c->d_kint, c->h_kint.data(), c->h_kint.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    const float* dd = data;
    float* dg = gathers;
    if (data_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(c->d_mig, data, nd * sizeof(float), cudaMemcpyHostToDevice, st));
        dd = c->d_mig;
    }
    if (gathers_mem == SF_MEM_HOST) dg = c->d_mig + nd;
    AngleParams p;
    p.S = c->d_S;
    p.xs = c->d_kgeo;
    p.xr = c->d_kgeo + nsrc;
    p.data = dd;
    p.cmp_ptr = c->d_kint;
    p.cmp_tr = c->d_kint + ncmp + 1;
    p.gathers = dg;
    p.nsrc = nsrc;
    p.nrec = nrec;
    p.nt = nt;
    p.nxx = c->nxx;
    p.nzz = c->nzz;
    p.nb = c->nb;
    p.nang = nang;
    p.ncmp = ncmp;
    p.dt = dt;
    p.rdt = sample_rate(dt);
    p.dx = c->dx;
    p.dz = c->dz;
    p.da = da;
    p.rda = (da > 1e-6f && da < 1e6f) ? 1.0f / da : 0.0f;
    p.aperture = aperture;
    // blocks of whole rows whose terms fit the workspace
    int rows;
    rc = call.reserve_blocks(c->nz, term_bytes(true, (size_t)nsrc + nrec, c->nx), &rows);
    if (rc) return rc;
    for (int i0 = 0; i0 < c->nz; i0 += rows) {
        rc = table_terms(c, call, true, Ts, Tr, nsrc, nrec, i0, std::min(rows, c->nz - i0), 0, c->nx, &p.tab, st);
        if (rc) return rc;
        const size_t nthr = (size_t)p.tab.nr * ncmp;
        k_kirchhoff_angles<<<(unsigned)std::min<size_t>((nthr + 127) / 128, (size_t)c->sms * 64), 128, 0, st>>>(p);
        CK(cudaGetLastError());
    }
    if (gathers_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(gathers, dg, ng * sizeof(float), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return SF_OK;
}

// The warps of a forward CTA share kFwdSmem bytes, each a histogram of nt
// samples and kFwdWarp bytes, of which 32 staged terms take half: the count of
// warps decides the order of a trace's sums, so it does not follow what a warp
// happens to stage.
constexpr size_t kFwdSmem = 200 * 1024;
constexpr size_t kFwdWarp = 64 * sizeof(float);
// Work traces times chunks the forward aims at when traces are few; a fixed
// number, so the summation order depends on the sizes only.
constexpr long kFwdCtas = 2432;

// The forward operator over the pairs LSKDM::compute_gradient and
// compute_stepLength visit (LSKDM.cu:52-90, :168-201): every source, every
// receiver with |xsrc - xrec| < max_offset, in that order; the other traces
// of data are zero.
static int kirchhoff_forward(sf_ctx* c, bool angle, const float* Ts, const float* Tr, int nsrc, int nrec,
                             const float* xsrc, const float* xrec, const float* model, int model_mem, size_t nmodel,
                             int nt, float dt, float aperture, float max_offset, int nang, int ncmp, float mincmp,
                             float dcmp, float da, float* data, int data_mem, void* stream)
{
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    // the tables in groups whose terms fit the workspace (a trace needs its
    // source's and its receiver's): one group unless the grid or the survey is
    // large; each trace is summed in one launch whatever the groups
    struct Group { int s0, ns, r0, nr, first, n; };
    std::vector<Group> groups;
    std::vector<int> ids, bins;
    auto make_groups = [&](int fit) {  // fit >= 2 tables
        const int gs = std::max(1, std::min(nsrc, fit - std::min(nrec, fit / 2))), gr = std::max(1, std::min(nrec, fit - gs));
        groups.clear();
        ids.clear();
        bins.clear();
        for (int s0 = 0; s0 < nsrc; s0 += gs)
            for (int r0 = 0; r0 < nrec; r0 += gr) {
                Group g{s0, std::min(gs, nsrc - s0), r0, std::min(gr, nrec - r0), (int)ids.size(), 0};
                for (int s = s0; s < s0 + g.ns; s++)
                    for (int r = r0; r < r0 + g.nr; r++) {
                        if (!(fabsf(xsrc[s] - xrec[r]) < max_offset)) continue;
                        if (angle) {
                            const float cmp = 0.5f * (xsrc[s] + xrec[r]);
                            const int b = (int)((cmp - mincmp) / dcmp);
                            if (b < 0 || b >= ncmp) continue;
                            bins.push_back(b);
                        }
                        ids.push_back(s * nrec + r);
                    }
                g.n = (int)ids.size() - g.first;
                if (g.n) groups.push_back(g);
            }
    };
    const size_t per_table = term_bytes(angle, 1, (size_t)c->nx * c->nz);
    int fit = (int)std::max<size_t>(2, std::min<size_t>(kTermBytes / per_table, (size_t)nsrc + nrec));
    make_groups(fit);
    const int ntrace = (int)ids.size();
    const size_t per_warp = (size_t)nt * sizeof(float) + kFwdWarp;
    const int W = (int)std::min<size_t>(8, kFwdSmem / per_warp);
    if (W < 1) return sf_fail(c, SF_ERR_RANGE, "too many time samples for the forward operator");
    const int nz = c->nzz - 2 * c->nb;
    const long ncell = (long)nz * (c->nxx - 2 * c->nb);
    const int nchunk = (int)std::max<long>(
        1, std::min<long>((kFwdCtas + std::max(ntrace, 1) - 1) / std::max(ntrace, 1), (ncell + 4095) / 4096));
    const int chunk = (int)((ncell + nchunk - 1) / nchunk);
    const size_t nd = (size_t)nsrc * nrec * nt;
    KirchCall call(c, st);
    int rc = call.open();
    if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_kgeo, &c->cap_kgeo, ((size_t)nsrc + nrec) * sizeof(float));
    if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_kint, &c->cap_kint, std::max<size_t>(1, ids.size() + bins.size()) * sizeof(int));
    if (!rc && (model_mem == SF_MEM_HOST || data_mem == SF_MEM_HOST))
        rc = sf_dev_reserve(c, (void**)&c->d_mig, &c->cap_mig, (nd + nmodel) * sizeof(float));
    if (!rc && nchunk > 1)
        rc = sf_dev_reserve(c, (void**)&c->d_kpart, &c->cap_kpart, (size_t)ntrace * nchunk * nt * sizeof(float));
    if (rc) return rc;
    while (ntrace > 0 && (rc = call.reserve(fit * per_table)) == SF_ERR_NOMEM && fit > 2) {
        fit = std::max(2, (fit + 1) / 2);
        make_groups(fit);
    }
    if (rc) return rc;
    c->h_kgeo.assign(xsrc, xsrc + nsrc);
    c->h_kgeo.insert(c->h_kgeo.end(), xrec, xrec + nrec);
    c->h_kint.assign(ids.begin(), ids.end());
    c->h_kint.insert(c->h_kint.end(), bins.begin(), bins.end());
    CK(cudaMemcpyAsync(c->d_kgeo, c->h_kgeo.data(), c->h_kgeo.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    if (!c->h_kint.empty())
        CK(cudaMemcpyAsync(c->d_kint, c->h_kint.data(), c->h_kint.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    const float* dm = model;
    float* dd = data;
    if (model_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(c->d_mig + nd, model, nmodel * sizeof(float), cudaMemcpyHostToDevice, st));
        dm = c->d_mig + nd;
    }
    if (data_mem == SF_MEM_HOST) dd = c->d_mig;
    CK(cudaMemsetAsync(dd, 0, nd * sizeof(float), st));
    for (const Group& g : groups) {
        KirchFwdParams p;
        const size_t matsize = (size_t)c->nxx * c->nzz;
        rc = table_terms(c, call, angle, Ts + matsize * g.s0, Tr + matsize * g.r0, g.ns, g.nr, 0, c->nz, 0, c->nx, &p.tab, st);
        if (rc) return rc;
        p.S = c->d_S;
        p.xs = c->d_kgeo;
        p.xr = c->d_kgeo + nsrc;
        p.model = dm;
        p.trace = c->d_kint + g.first;
        p.cmp = c->d_kint + ntrace + g.first;
        p.part = c->d_kpart + (size_t)g.first * nchunk * nt;
        p.data = dd;
        p.nchunk = nchunk;
        p.chunk = chunk;
        p.s0 = g.s0;
        p.r0 = g.r0;
        p.nsrc = g.ns;
        p.nrec = nrec;
        p.nt = nt;
        p.nxx = c->nxx;
        p.nzz = c->nzz;
        p.nb = c->nb;
        p.nang = nang;
        p.warps = W;
        p.dt = dt;
        p.rdt = sample_rate(dt);
        p.dx = c->dx;
        p.dz = c->dz;
        p.da = da;
        p.rda = (da > 1e-6f && da < 1e6f) ? 1.0f / da : 0.0f;
        p.aperture = aperture;
        const size_t smem = (size_t)W * per_warp;
        const unsigned grid = (unsigned)((long)g.n * nchunk);
        const void* kern = angle ? (const void*)k_kirchhoff_forward<true> : (const void*)k_kirchhoff_forward<false>;
        CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        void* args[] = {&p};
        CK(cudaLaunchKernel(kern, dim3(grid), dim3(32 * W), args, smem, st));
    }
    if (ntrace > 0) {
        if (nchunk > 1) {
            const size_t n = (size_t)ntrace * nt;
            k_sum_chunks<<<(unsigned)std::min<size_t>((n + 255) / 256, (size_t)c->sms * 16), 256, 0, st>>>(
                c->d_kpart, c->d_kint, dd, ntrace, nchunk, nt);
            CK(cudaGetLastError());
        }
    }
    if (data_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(data, dd, nd * sizeof(float), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return SF_OK;
}

extern "C" int sf_kirchhoff_image_forward(sf_ctx* c, const float* Ts, const float* Tr, int nsrc, int nrec,
                                          const float* xsrc, const float* xrec, const float* image, int image_mem,
                                          int nt, float dt, float aperture, float max_offset, float* data,
                                          int data_mem, void* stream)
{
    if (!c || !Ts || !Tr || !xsrc || !xrec || !image || !data || nsrc < 1 || nrec < 1 || nt < 1 || !(dt > 0.0f))
        return sf_fail(c, SF_ERR_ARG, "bad Kirchhoff arguments");
    return kirchhoff_forward(c, false, Ts, Tr, nsrc, nrec, xsrc, xrec, image, image_mem, (size_t)c->nx * c->nz, nt,
                             dt, aperture, max_offset, 0, 0, 0.0f, 1.0f, 1.0f, data, data_mem, stream);
}

extern "C" int sf_kirchhoff_angle_forward(sf_ctx* c, const float* Ts, const float* Tr, int nsrc, int nrec,
                                          const float* xsrc, const float* xrec, const float* gathers,
                                          int gathers_mem, int nt, float dt, float aperture, float max_offset,
                                          float max_angle, float da, float* data, int data_mem, void* stream)
{
    if (!c || !xsrc || !xrec) return sf_fail(c, SF_ERR_ARG, "null argument");
    int nang, ncmp;
    float mincmp, dcmp;
    if (angle_dims(xsrc, nsrc, xrec, nrec, max_angle, da, &nang, &ncmp, &mincmp, &dcmp))
        return sf_fail(c, SF_ERR_ARG, "angle gathers need two sources, two receivers, increasing positions, da > 0");
    if (!Ts || !Tr || !gathers || !data || nt < 1 || !(dt > 0.0f))
        return sf_fail(c, SF_ERR_ARG, "bad Kirchhoff arguments");
    const size_t ng = (size_t)(c->nzz - 2 * c->nb) * nang * ncmp;
    return kirchhoff_forward(c, true, Ts, Tr, nsrc, nrec, xsrc, xrec, gathers, gathers_mem, ng, nt, dt, aperture,
                             max_offset, nang, ncmp, mincmp, dcmp, da, data, data_mem, stream);
}
