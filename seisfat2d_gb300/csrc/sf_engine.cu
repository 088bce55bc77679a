// C ABI of the GB300 eikonal engine (include/seisfat2d.h): context, buffers,
// launches of the forward kernels. Compiled for sm_103a only.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/seisfat2d.h"
#include "sf_engine.h"

using namespace sf;

// ------------------------------------------------------------------ helpers

const char* sf_status_string(int s)
{
    switch (s) {
    case SF_OK: return "ok";
    case SF_ERR_ARG: return "invalid argument";
    case SF_ERR_CUDA: return "CUDA error";
    case SF_ERR_TIMEOUT: return "in-kernel wait timed out";
    case SF_ERR_RANGE: return "source or window outside the grid";
    case SF_ERR_STATE: return "call out of order";
    case SF_ERR_NOMEM: return "device allocation failed";
    default: return "unknown status";
    }
}

int sf_fail(sf_ctx* c, int status, const std::string& msg)
{
    if (c) c->err = msg;
    return status;
}

int sf_cuda_check(sf_ctx* c, cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return SF_OK;
    std::string m = std::string(what) + ": " + cudaGetErrorString(e);
    if (e == cudaErrorMemoryAllocation) return sf_fail(c, SF_ERR_NOMEM, m);
    return sf_fail(c, SF_ERR_CUDA, m);
}

#define CK(call)                                                          \
    do {                                                                  \
        int _st = sf_cuda_check(c, (call), #call);                        \
        if (_st != SF_OK) return _st;                                     \
    } while (0)

int sf_dev_reserve(sf_ctx* c, void** p, size_t* cap, size_t bytes)
{
    if (bytes <= *cap && *p) return SF_OK;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    size_t want = std::max<size_t>(bytes, 256);
    cudaError_t e = cudaMalloc(p, want);
    if (e == cudaErrorMemoryAllocation && c->d_kterm) {
        // the Kirchhoff operators' workspace, which they can do with less of, makes room
        cudaGetLastError();
        cudaFree(c->d_kterm);
        c->d_kterm = nullptr;
        c->cap_kterm = 0;
        e = cudaMalloc(p, want);
    }
    if (e != cudaSuccess) {
        *p = nullptr;
        if (e == cudaErrorMemoryAllocation) cudaGetLastError();  // reported here, not by the next launch's check
        return sf_cuda_check(c, e, "cudaMalloc");
    }
    *cap = want;
    return SF_OK;
}

int sf_dev_reserve_zero(sf_ctx* c, void** p, size_t* cap, size_t bytes)
{
    const bool grow = !(bytes <= *cap && *p);
    int rc = sf_dev_reserve(c, p, cap, bytes);
    if (rc || !grow) return rc;
    return sf_cuda_check(c, cudaMemset(*p, 0, *cap), "cudaMemset");
}

unsigned sf_next_epoch(sf_ctx* c)
{
    // after a wrap an epoch's tags could meet pairs an earlier cycle left in
    // the handoff buffers: the next forward and adjoint launches clear them
    if (c->epoch == (1u << 22) - 1) {
        c->hand_stale_f = c->hand_stale_a = true;
        c->epoch = kGraphEpoch;
    }
    return ++c->epoch;
}

// ------------------------------------------------------------------ kernels

namespace {

// Checks fdiv_k against __fdiv_rn for b = divs[w] over all dividends of [1, 2)
// (both signs follow by symmetry); rbs[w] = RN(1/b), bad bit w set on any
// difference. Then (w = n) frcp_k on [1, 2), bad bit 5, and (w = n+1, n+2)
// fsqrt_k on [1, 4), bad bit 4.
__global__ void k_verify_div(const float* divs, int n, float* rbs, int* bad)
{
    const unsigned total = (unsigned)(n + 3) << 23;
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const int w = t >> 23;
        const float a = __uint_as_float(0x3f800000u | (t & 0x7fffffu));
        float got, want;
        int bit = w;
        if (w < n) {
            const float b = divs[w], rb = __frcp_rn(b);
            if ((t & 0x7fffffu) == 0) rbs[w] = rb;
            got = fdiv_k<false>(a, b, rb);
            want = __fdiv_rn(a, b);
        } else if (w == n) {
            got = frcp_k(a);
            want = __frcp_rn(a);
            bit = 5;
        } else {
            const float v = (w == n + 1) ? a : 2.0f * a;
            got = fsqrt_k<false>(v);
            want = __fsqrt_rn(v);
            bit = 4;
        }
        if (__float_as_uint(got) != __float_as_uint(want)) atomicOr(bad, 1 << bit);
    }
}

// Sets *flag when a slowness of the field (nzz x nxx) lies outside
// in_fast_range.
__global__ void k_check_range(const float* __restrict__ S, int nzz, int nxx, float dx, float dz, int* flag)
{
    bool ok = true;
    const size_t n = (size_t)nzz * nxx;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
        ok &= in_fast_range(S[q], dx, dz);
    if (!ok) *flag = 1;
}

// The context's padded slowness S from a model (expand_boundary,
// modeling.cu:204-232: clamp to the edge), or with a step dS added on the
// model's cells, or as it is; its copy Sp at the solver's column stride ld
// (rows past the grid repeat the last); and flags[2], whether a value lies
// outside in_fast_range. One launch: with a memset, an expansion or addition and
// a check of their own, an update of a small model took 10 us (of 60) longer. The
// CTAs join in flags[3] and count in flags[4]; the last one publishes and clears.
__global__ void k_solver_slowness(float* __restrict__ S, int nx, int nz, int nb, int ld, float dx, float dz,
                                  const float* __restrict__ model, const float* __restrict__ dS,
                                  float* __restrict__ Sp, int* flags)
{
    const int nzz = nz + 2 * nb, nxx = nx + 2 * nb;
    bool ok = true;
    for (int j = blockIdx.x; j < nxx; j += gridDim.x)
        for (int i = threadIdx.x; i < ld; i += blockDim.x) {
            const int r = min(i, nzz - 1);
            const size_t at = (size_t)r + (size_t)j * nzz;
            float s;
            if (model) {
                s = model[min(max(r - nb, 0), nz - 1) + (size_t)min(max(j - nb, 0), nx - 1) * nz];
            } else {
                s = S[at];
                if (dS && r >= nb && r < nzz - nb && j >= nb && j < nxx - nb)
                    s = fadd(s, dS[(r - nb) + (size_t)(j - nb) * nz]);
            }
            if ((model || dS) && i < nzz) S[at] = s;
            Sp[(size_t)i + (size_t)j * ld] = s;
            ok &= in_fast_range(s, dx, dz);
        }
    const int bad = __syncthreads_or(!ok);
    if (threadIdx.x == 0) {
        if (bad) atomicOr(flags + 3, 1);
        __threadfence();
        if (atomicAdd(flags + 4, 1) == (int)gridDim.x - 1) {
            flags[2] = atomicExch(flags + 3, 0);
            flags[4] = 0;
        }
    }
}

// A window of column stride ld as nzz x ncols values. Tables are copied one per
// call, a few microseconds each, so the launch of the next may begin while this
// one runs (a programmatic launch, see table_out); it waits for all work before it
// ahead of its first access.
__global__ void k_unpitch(const float* in, int nzz, int ncols, int ld, float* out)
{
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
    for (int j = blockIdx.x; j < ncols; j += gridDim.x)
        for (int i = threadIdx.x; i < nzz; i += blockDim.x) out[i + (size_t)j * nzz] = in[i + (size_t)j * ld];
}

// compute_seismogram on a device field (modeling.cu:161-194).
__global__ void k_picks(const float* __restrict__ T, int nzz, int ncols, int c0, int nb, float dx,
                        float dz, const float* __restrict__ rx, const float* __restrict__ rz,
                        int nrec, float* __restrict__ out)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrec) return;
    int i, j;
    float xd, zd;
    float v = __int_as_float(0x7fc00000);
    if (pick_geom(rx[r], rz[r], dx, dz, nb, nzz, ncols, c0, i, j, xd, zd))
        v = pick_value(T, nzz, i, j, xd, zd);
    out[r] = v;
}

}  // namespace

size_t sf_fwd_smem_bytes(int warps, bool comp)
{
    return ((sizeof(CtaShared) + 15) & ~size_t(15)) + (size_t)warps * (comp ? ring_bytes<true>() : ring_bytes<false>());
}

// ------------------------------------------------------------------ context

extern "C" const char* sf_ctx_last_error(const sf_ctx* c) { return c ? c->err.c_str() : "null context"; }

extern "C" int sf_ctx_create(sf_ctx** out, int nx, int nz, float dx, float dz, int device)
{
    if (!out) return SF_ERR_ARG;
    *out = nullptr;
    if (nx < 2 || nz < 2 || !(dx > 0.0f) || !(dz > 0.0f)) return SF_ERR_ARG;
    sf_ctx* c = new sf_ctx();
    c->dev = device;
    c->nx = nx;
    c->nz = nz;
    c->nb = 3;
    c->nxx = nx + 2 * c->nb;
    c->nzz = nz + 2 * c->nb;
    c->dx = dx;
    c->dz = dz;
    Consts& k = c->kc;
    k.dx = dx;
    k.dz = dz;
    k.dz2i = 1.0f / (dz * dz);  // modeling.cu:64-65 (host, no contraction)
    k.dx2i = 1.0f / (dx * dx);
    k.hyp = sqrtf(dx * dx + dz * dz);
    k.D = k.dz2i + k.dx2i;
    k.K = k.dz2i * k.dx2i;
    k.kA = k.dz2i - k.dx2i;
    k.kB = k.dx2i - k.dz2i;
    k.k2K = 2.0f * k.K;
    set_scaled(k);
    int st = sf_cuda_check(c, cudaSetDevice(device), "cudaSetDevice");
    if (st == SF_OK) {
        cudaDeviceProp prop;
        st = sf_cuda_check(c, cudaGetDeviceProperties(&prop, device), "cudaGetDeviceProperties");
        if (st == SF_OK) c->sms = prop.multiProcessorCount;
    }
    if (st == SF_OK) st = sf_verify_divisors(c);
    size_t cap = 0;
    if (st == SF_OK) st = sf_dev_reserve(c, (void**)&c->d_S, &cap, sizeof(float) * (size_t)c->nxx * c->nzz);
    cap = 0;
    if (st == SF_OK) st = sf_dev_reserve(c, (void**)&c->d_Sp, &cap, sizeof(float) * (size_t)c->nxx * strip_pitch(c->nzz));
    cap = 0;
    if (st == SF_OK) st = sf_dev_reserve(c, (void**)&c->d_flags, &cap, 256);
    if (st == SF_OK) st = sf_cuda_check(c, cudaMemset(c->d_flags, 0, 256), "cudaMemset");
    for (cudaEvent_t* ev : {&c->slowness_ev, &c->kirch_ev})
        if (st == SF_OK)
            st = sf_cuda_check(c, cudaEventCreateWithFlags(ev, cudaEventDisableTiming), "cudaEventCreateWithFlags");
    if (st == SF_OK) st = sf_fwd_setup(c);
    if (st != SF_OK) {
        sf_ctx_destroy(c);
        return st;
    }
    *out = c;
    return SF_OK;
}

extern "C" int sf_ctx_destroy(sf_ctx* c)
{
    if (!c) return SF_OK;
    cudaSetDevice(c->dev);
    sf_plan_release(c);
    sf_adjoint_release(c);
    void* bufs[] = {c->d_S, c->d_Sp, c->d_Tc, c->d_flags, c->d_shots, c->d_T, c->d_rx, c->d_rz, c->d_picks, c->d_Sq,
                    c->d_tcode, c->d_tc1, c->d_tc2, c->d_model, c->d_cij_all, c->d_hand, c->d_ctr,
                    c->d_skern, c->d_upd, c->d_wav, c->d_mig, c->d_kgeo, c->d_kint, c->d_kpart,
                    c->d_vfac, c->d_gcij, c->d_fuse, c->d_Tl, c->d_srange, c->d_kterm};
    for (void* b : bufs)
        if (b) cudaFree(b);
    for (cudaEvent_t ev : {c->slowness_ev, c->kirch_ev})
        if (ev) cudaEventDestroy(ev);
    delete c;
    return SF_OK;
}

extern "C" int sf_ctx_dims(const sf_ctx* c, int* nxx, int* nzz, int* nb)
{
    if (!c) return SF_ERR_ARG;
    if (nxx) *nxx = c->nxx;
    if (nzz) *nzz = c->nzz;
    if (nb) *nb = c->nb;
    return SF_OK;
}

extern "C" int sf_set_launch(sf_ctx* c, int warps, int gang_warps)
{
    if (!c) return SF_ERR_ARG;
    if (warps < 0 || warps > kMaxWarps) return sf_fail(c, SF_ERR_ARG, "warps per CTA must be 1..16");
    if (gang_warps < 0 || gang_warps > 1024) return sf_fail(c, SF_ERR_ARG, "gang warps must be 0..1024");
    if (warps) c->warps = warps;
    c->gang_warps = gang_warps;
    c->plan_dirty = true;  // a planned batch is reconfigured before its next iteration
    return SF_OK;
}

extern "C" int sf_set_wait_limit(sf_ctx* c, double seconds)
{
    if (!c) return SF_ERR_ARG;
    if (!(seconds >= 0.0 && seconds <= 60.0)) return sf_fail(c, SF_ERR_ARG, "wait limit must be in [0, 60] s");
    c->wait_ns = (unsigned long long)(seconds * 1e9);  // 0: the default of about 2 s
    c->plan_dirty = true;
    return SF_OK;
}

extern "C" int sf_test_stall_next_batch(sf_ctx* c)
{
    if (!c) return SF_ERR_ARG;
    c->stall_next = true;
    return SF_OK;
}

extern "C" int sf_test_workspace_limit(sf_ctx* c, size_t bytes)
{
    if (!c) return SF_ERR_ARG;
    c->kterm_limit = bytes;
    return SF_OK;
}

extern "C" int sf_set_arithmetic(sf_ctx* c, int mode)
{
    if (!c) return SF_ERR_ARG;
    if (mode != SF_ARITH_REFERENCE && mode != SF_ARITH_IEEE && mode != SF_ARITH_COMPENSATED)
        return sf_fail(c, SF_ERR_ARG, "unknown arithmetic");
    c->arith = mode;
    c->plan_dirty = true;
    return SF_OK;
}

extern "C" int sf_get_arithmetic(const sf_ctx* c, int* mode)
{
    if (!c || !mode) return SF_ERR_ARG;
    *mode = c->arith;
    return SF_OK;
}

extern "C" int sf_set_strip_loop(sf_ctx* c, int mode)
{
    if (!c) return SF_ERR_ARG;
    if (mode != SF_LOOP_AUTO && mode != SF_LOOP_GENERAL && mode != SF_LOOP_INTERIOR)
        return sf_fail(c, SF_ERR_ARG, "unknown strip-loop mode");
    c->strip_loop = mode;
    c->plan_dirty = true;
    return SF_OK;
}

extern "C" int sf_get_strip_loop(const sf_ctx* c, int* mode, int* last_interior)
{
    if (!c) return SF_ERR_ARG;
    if (mode) *mode = c->strip_loop;
    if (last_interior) *last_interior = c->batch_interior ? 1 : 0;
    return SF_OK;
}

extern "C" int sf_get_launch(const sf_ctx* c, int* warps, int* gang_warps)
{
    if (!c) return SF_ERR_ARG;
    if (warps) *warps = c->warps;
    if (gang_warps) *gang_warps = c->gang_warps;
    return SF_OK;
}

// Warps per shot ("slots"). The solve of a shot is a list of 4 nstrips strip
// tasks of which 2 nstrips can run at once (solve_window), so a shot gets up
// to that many warps when the device holds every shot that way. Otherwise the
// warps take the tasks in rounds, and a shot gets its equal share of the
// device's warps, or fewer where these divide the tasks of a pair of sweeps
// into as many full rounds: 100 shots of 12 strips took 3.94 ms with the 18
// warps each that fit, 3.76 with 12 (both two rounds of 24 tasks), 4.70 with
// 10 (three); 24 warps each, where they fit, 1.96 against 2.11 with 12. 200
// shots of 16 strips: 3.90 ms with the 12 warps each that fit, 4.04 with 8.
// With more shots than that leaves room for, a shot still gets four warps (or
// one per two strips) and the rest wait in the queue: fewer windows are then in
// use at a time, and the last shots end together. Taped forward and reverse
// sweeps of 1000 windows of about 1000 x 1001 cells 27.9 + 14.2 ms with four,
// 31.0 + 18.1 with two, 53 + 18 with one; 1000 shots of 801 x 351 9.7 + 5.0,
// 12.4 + 4.9, 11.7 + 6.4; 1500 shots of 401 x 101 (4 strips) 2.5 + 1.4 with
// four, 2.2 + 1.6 with two, 2.3 + 1.5 with one.
int sf_gang_shape(sf_ctx* c, const void* kernel, size_t smem, int nshots, int nstrips, int gang_warps, int* G,
                  int* NG)
{
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, c->warps * 32, smem));
    if (per_sm < 1) return sf_fail(c, SF_ERR_CUDA, "kernel does not fit on an SM");
    const long long cap_ctas = (long long)per_sm * c->sms;
    int slots = gang_warps;
    if (slots <= 0) {
        const long long cap_warps = cap_ctas * c->warps;
        const long long least = std::min(4, (nstrips + 1) / 2);
        const long long most = std::max(least, std::min<long long>(2LL * nstrips, cap_warps / std::max(1, nshots)));
        const int rounds = (int)((2 * nstrips + most - 1) / most);
        slots = (2 * nstrips) % rounds ? (int)most : 2 * nstrips / rounds;
    }
    int g = std::max(1, (slots + c->warps - 1) / c->warps);
    if (g > cap_ctas) g = (int)cap_ctas;
    *G = g;
    *NG = (int)std::max(1LL, std::min<long long>(nshots, cap_ctas / g));
    return SF_OK;
}

// Reciprocals of the four constant divisors and whether the fast division
// equals IEEE division for them (see fdiv_k).
int sf_verify_divisors(sf_ctx* c)
{
    Consts& k = c->kc;
    float h_div[4] = {k.dx, k.dz, k.hyp, k.D}, h_rb[4] = {0, 0, 0, 0};
    int h_bad = 0;
    float* d_div = nullptr;
    int* d_bad = nullptr;
    CK(cudaMalloc(&d_div, 8 * sizeof(float) + sizeof(int)));
    d_bad = reinterpret_cast<int*>(d_div + 8);
    cudaError_t e = cudaMemcpy(d_div, h_div, sizeof(h_div), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(d_bad, 0, sizeof(int));
    if (e == cudaSuccess) {
        k_verify_div<<<c->sms * 8, 256>>>(d_div, 4, d_div + 4, d_bad);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(h_rb, d_div + 4, sizeof(h_rb), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&h_bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d_div);
    CK(e);
    k.rdx = h_rb[0];
    k.rdz = h_rb[1];
    k.rhyp = h_rb[2];
    k.rD = h_rb[3];
    k.mflags = ((~h_bad) & 0x3f) | (range_ok(k.dx, k.dz) ? 0x40 : 0);
    return SF_OK;
}

namespace sf {
// accessors of the k_shots instantiations: tape, reference arithmetic,
// interior-block body, compensated arithmetic
const void* sf_kshots_0000();
const void* sf_kshots_0010();
const void* sf_kshots_0100();
const void* sf_kshots_0110();
const void* sf_kshots_1000();
const void* sf_kshots_1010();
const void* sf_kshots_1100();
const void* sf_kshots_1110();
const void* sf_kshots_0001();
const void* sf_kshots_0011();
const void* sf_kshots_1001();
const void* sf_kshots_1011();
const void* sf_kshots_noalloc();  // 0110 on windows of the caller's column stride
}  // namespace sf

// The compensated arithmetic has no reference-build variant.
const void* sf_kshots_kernel(bool tape, bool ref, bool interior, bool comp)
{
    if (comp) ref = false;
    switch (((int)tape << 3) | ((int)ref << 2) | ((int)interior << 1) | (int)comp) {
    case 0x0: return sf::sf_kshots_0000();
    case 0x2: return sf::sf_kshots_0010();
    case 0x4: return sf::sf_kshots_0100();
    case 0x6: return sf::sf_kshots_0110();
    case 0x8: return sf::sf_kshots_1000();
    case 0xa: return sf::sf_kshots_1010();
    case 0xc: return sf::sf_kshots_1100();
    case 0xe: return sf::sf_kshots_1110();
    case 0x1: return sf::sf_kshots_0001();
    case 0x3: return sf::sf_kshots_0011();
    case 0x9: return sf::sf_kshots_1001();
    case 0xb: return sf::sf_kshots_1011();
    default: return nullptr;
    }
}

// The qP pass kernels: arithmetic (reference / IEEE / compensated) x
// derivative factors (taped batches).
const void* sf_kqp_kernel(bool ref, bool comp, bool fact)
{
    if (comp) return fact ? (const void*)k_qp<false, true, true> : (const void*)k_qp<false, true, false>;
    if (ref) return fact ? (const void*)k_qp<true, false, true> : (const void*)k_qp<true, false, false>;
    return fact ? (const void*)k_qp<false, false, true> : (const void*)k_qp<false, false, false>;
}

// The interior-block body drops the bounds tests of the blocks whose marches
// all lie inside the window; a narrow window has few of them and runs both
// bodies. SF_LOOP_AUTO takes it when every window of the batch is at least
// kInteriorCols wide: 200 shots of 501 rows, untaped, 64 columns 0.703 ms either
// way, 96 0.748 general and 0.733 interior, 128 0.811 and 0.774, 196 0.923 and
// 0.847, 320 1.111 and 0.946; of 351 rows, taped compensated forward and
// reverse, 64 columns 1.221 and 1.273, 128 1.425 and 1.462, 196 1.611 and 1.608,
// 320 1.913 and 1.894.
constexpr int kInteriorCols = 128;
bool sf_interior_loops(const sf_ctx* c)
{
    if (c->strip_loop != SF_LOOP_AUTO) return c->strip_loop == SF_LOOP_INTERIOR;
    return !c->hshots.empty() && c->hshots.back().ncols >= kInteriorCols;  // sorted widest first
}

int sf_fwd_setup(sf_ctx* c)
{
    for (int k = 0; k < 16; k++) {
        const bool tape = k & 8, comp = k & 1;
        const size_t mx = sf_fwd_smem_bytes(comp ? kMaxWarpsComp : kMaxWarps, comp);
        const void* f = sf_kshots_kernel(tape, k & 4, k & 2, comp);
        if (f) CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mx));
    }
    return sf_adj_setup(c);
}

// ------------------------------------------------------------------ models

// The context's slowness from a model on the device, by a step dS or as it is
// (both null), with the solver's copy and the check for the fast form of the
// updates (k_solver_slowness).
int sf_solver_slowness(sf_ctx* c, const float* model, const float* dS, cudaStream_t st)
{
    const int ld = strip_pitch(c->nzz);
    k_solver_slowness<<<std::min(c->nxx, 2 * c->sms), std::min(ld, 512), 0, st>>>(c->d_S, c->nx, c->nz, c->nb, ld, c->dx, c->dz,
                                                                            model, dS, c->d_Sp, c->d_flags);
    CK(cudaGetLastError());
    return SF_OK;
}

int sf_capturing(sf_ctx* c, cudaStream_t st, bool* capturing)
{
    *capturing = false;
    if (!st || st == cudaStreamLegacy) return SF_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(st, &cs));
    *capturing = cs != cudaStreamCaptureStatusNone;
    return SF_OK;
}

int sf_launch_epoch(sf_ctx* c, void* hand, size_t bytes, cudaStream_t st, unsigned* epoch)
{
    bool capturing;
    int rc = sf_capturing(c, st, &capturing);
    if (rc) return rc;
    *epoch = capturing ? kGraphEpoch : sf_next_epoch(c);
    if (capturing) CK(cudaMemsetAsync(hand, 0, bytes, st));
    return SF_OK;
}

// Orders work on `st` that reads or updates the slowness after the last
// sf_set_slowness, which returns before its work on the legacy stream is done
// when its source is a padded device field. Blocking streams follow the legacy
// stream by themselves. A captured launch waits at every replay, for the
// sf_set_slowness called last by then.
int sf_wait_slowness(sf_ctx* c, cudaStream_t st)
{
    if (!st || st == cudaStreamLegacy) return SF_OK;
    bool capturing;
    int rc = sf_capturing(c, st, &capturing);
    if (rc) return rc;
    if (capturing) {
        CK(cudaStreamWaitEvent(st, c->slowness_ev, cudaEventWaitExternal));
        return SF_OK;
    }
    unsigned flags = 0;
    CK(cudaStreamGetFlags(st, &flags));
    if (flags & cudaStreamNonBlocking) CK(cudaStreamWaitEvent(st, c->slowness_ev, 0));
    return SF_OK;
}

extern "C" int sf_set_slowness(sf_ctx* c, const float* s, int layout, int mem)
{
    if (!c || !s) return SF_ERR_ARG;
    CK(cudaSetDevice(c->dev));
    const size_t npad = (size_t)c->nxx * c->nzz;
    if (layout == SF_LAYOUT_PADDED) {
        CK(cudaMemcpy(c->d_S, s, npad * sizeof(float),
                      mem == SF_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
        int rc = sf_solver_slowness(c, nullptr, nullptr, nullptr);
        if (rc) return rc;
        if (mem == SF_MEM_DEVICE) CK(cudaEventRecord(c->slowness_ev, nullptr));  // see sf_wait_slowness
        else CK(cudaStreamSynchronize(nullptr));  // a host copy is finished when the call returns: so is its check
        return SF_OK;
    }
    if (layout != SF_LAYOUT_MODEL) return sf_fail(c, SF_ERR_ARG, "unknown layout");
    const size_t nm = (size_t)c->nx * c->nz;
    int st = sf_dev_reserve(c, (void**)&c->d_model, &c->cap_model, nm * sizeof(float));
    if (st) return st;
    CK(cudaMemcpy(c->d_model, s, nm * sizeof(float),
                  mem == SF_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
    int rc = sf_solver_slowness(c, c->d_model, nullptr, nullptr);
    if (rc) return rc;
    CK(cudaDeviceSynchronize());
    return SF_OK;
}

extern "C" int sf_get_slowness(sf_ctx* c, float* out, int mem)
{
    if (!c || !out) return SF_ERR_ARG;
    CK(cudaSetDevice(c->dev));
    CK(cudaMemcpy(out, c->d_S, sizeof(float) * (size_t)c->nxx * c->nzz,
                  mem == SF_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost));
    return SF_OK;
}

// Deterministic quantisation of one padded field (modeling.cu:264-279).
static void compress_field(const float* in, size_t n, uint16_t* out, float* vmax, float* vmin)
{
    float mx = -1e20f, mn = 1e20f;
    for (size_t i = 0; i < n; i++) {
        mn = std::fmin(in[i], mn);
        mx = std::fmax(in[i], mx);
    }
    *vmax = mx;
    *vmin = mn;
    for (size_t i = 0; i < n; i++) {
        if (mx == mn) {
            out[i] = 1;
            continue;
        }
        float v = 1.0f + (float)(65535 - 1) * (in[i] - mn) / (mx - mn);
        out[i] = (uint16_t)v;
    }
}

static int upload_codes(sf_ctx* c, const uint16_t* const codes[6], int mem)
{
    const size_t npad = (size_t)c->nxx * c->nzz;
    int st = sf_dev_reserve(c, (void**)&c->d_cij_all, &c->cap_cij, 6 * npad * sizeof(uint16_t));
    if (st) return st;
    for (int q = 0; q < 6; q++) {
        CK(cudaMemcpy(c->d_cij_all + q * npad, codes[q], npad * sizeof(uint16_t),
                      mem == SF_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
    }
    c->have_cij = true;
    return SF_OK;
}

extern "C" int sf_set_stiffness(sf_ctx* c, const float* const cij[6], int mem)
{
    if (!c || !cij) return SF_ERR_ARG;
    for (int q = 0; q < 6; q++)
        if (!cij[q]) return SF_ERR_ARG;
    CK(cudaSetDevice(c->dev));
    const int nx = c->nx, nz = c->nz, nb = c->nb, nzz = c->nzz, nxx = c->nxx;
    const size_t nm = (size_t)nx * nz, npad = (size_t)nxx * nzz;
    std::vector<float> model(nm), padded(npad);
    std::vector<std::vector<uint16_t>> codes(6, std::vector<uint16_t>(npad));
    for (int q = 0; q < 6; q++) {
        if (mem == SF_MEM_DEVICE) CK(cudaMemcpy(model.data(), cij[q], nm * sizeof(float), cudaMemcpyDeviceToHost));
        else std::memcpy(model.data(), cij[q], nm * sizeof(float));
        for (int j = 0; j < nxx; j++)
            for (int i = 0; i < nzz; i++) {
                int si = std::min(std::max(i - nb, 0), nz - 1), sj = std::min(std::max(j - nb, 0), nx - 1);
                padded[i + (size_t)j * nzz] = model[si + (size_t)sj * nz];
            }
        compress_field(padded.data(), npad, codes[q].data(), &c->mm[2 * q + 1], &c->mm[2 * q]);
    }
    const uint16_t* ptrs[6];
    for (int q = 0; q < 6; q++) ptrs[q] = codes[q].data();
    return upload_codes(c, ptrs, SF_MEM_HOST);
}

extern "C" int sf_set_stiffness_codes(sf_ctx* c, const uint16_t* const codes[6], const float mm[12], int mem)
{
    if (!c || !codes || !mm) return SF_ERR_ARG;
    for (int q = 0; q < 6; q++)
        if (!codes[q]) return SF_ERR_ARG;
    CK(cudaSetDevice(c->dev));
    std::memcpy(c->mm, mm, sizeof(c->mm));
    return upload_codes(c, codes, mem);
}

// ------------------------------------------------------------------ shots

// Interior cells the reference's launch schedule (modeling.cu:123-159) never
// updates, for a grid of nzz x ncols, per sweep: the middle-band thread count
// (level-2) can fall one short of the diagonal when min(n)-2 is a multiple of
// the 256-thread block.
void sf_skip_cells(int ncols, int nzz, int si[4], int sj[4])
{
    const int nxx = ncols, total = nxx + nzz - 2, mn = std::min(nxx, nzz), mxl = std::max(nxx, nzz);
    for (int s = 0; s < 4; s++) {
        si[s] = sj[s] = -1;
        const int zd = (s == 2 || s == 3) ? -1 : 1;
        const int xd = (s == 0 || s == 2) ? -1 : 1;
        for (int level = 0; level < total; level++) {
            int zo, xo;
            switch (s) {
            case 0: zo = (level < nxx) ? 0 : level - nxx + 1; xo = (level < nxx) ? level : nxx - 1; break;
            case 1: zo = (level < nzz) ? nzz - level - 1 : 0; xo = (level < nzz) ? 0 : level - nzz + 1; break;
            case 2: zo = (level < nzz) ? level : nzz - 1; xo = (level < nzz) ? nxx - 1 : nxx - 1 - (level - nzz + 1); break;
            default: zo = (level < nxx) ? nzz - 1 : nzz - 1 - (level - nxx + 1); xo = (level < nxx) ? nxx - level - 1 : 0; break;
            }
            int n = (level < mn) ? level + 1 : (level >= mxl) ? total - level : total - mn - mxl + level;
            int nl = ((n + 255) / 256) * 256;
            int lo = 0, hi = 1 << 30;
            if (zd > 0) { lo = std::max(lo, 1 - zo); hi = std::min(hi, nzz - 2 - zo); }
            else { lo = std::max(lo, zo - (nzz - 2)); hi = std::min(hi, zo - 1); }
            if (xd > 0) { lo = std::max(lo, 1 - xo); hi = std::min(hi, nxx - 2 - xo); }
            else { lo = std::max(lo, xo - (nxx - 2)); hi = std::min(hi, xo - 1); }
            for (int e = std::max(lo, nl); e <= hi; e++) {
                si[s] = zo + zd * e;
                sj[s] = xo + xd * e;
            }
        }
    }
}

// Builds the device shot table (sorted widest window first for the work
// queue). Returns SF_ERR_RANGE for a source outside its window.
int sf_prepare_shots(sf_ctx* c, const sf_shot* shots, int nshots, bool tape)
{
    c->plan_valid = false;  // the planned batch's tables are replaced
    // a new generation unless the table comes out the same as before (an
    // early error return leaves it new)
    const std::vector<ShotDev> prev = c->hshots;
    const unsigned long long prev_gen = c->shots_gen++;
    c->hshots.resize(nshots);
    long long toff = 0, tape_off = 0, q_off = 0;
    const int nstrips = (c->nzz + 31) / 32;
    int maxcols = 0;
    for (int b = 0; b < nshots; b++) {
        const sf_shot& s = shots[b];
        ShotDev d;
        std::memset(&d, 0, sizeof(d));
        d.c0 = s.c0;
        d.ncols = (s.ncols <= 0) ? c->nxx - s.c0 : s.ncols;
        if (d.c0 < 0 || d.ncols < 3 || d.c0 + d.ncols > c->nxx)
            return sf_fail(c, SF_ERR_RANGE, "shot " + std::to_string(b) + ": window outside the grid");
        // modeling.cu:112-113 (host float arithmetic, no contraction)
        float fx = (s.sx + 0.5f * c->dx) / c->dx;
        float fz = (s.sz + 0.5f * c->dz) / c->dz;
        if (!(fx > -1e9f && fx < 1e9f && fz > -1e9f && fz < 1e9f))
            return sf_fail(c, SF_ERR_RANGE, "shot " + std::to_string(b) + ": source not finite");
        d.sIdx = (int)fx + c->nb;
        d.sIdz = (int)fz + c->nb;
        d.sx = s.sx;
        d.sz = s.sz;
        const int sloc = d.sIdx - d.c0;
        if (d.sIdz < 1 || d.sIdz > c->nzz - 2 || sloc < 1 || sloc > d.ncols - 2)
            return sf_fail(c, SF_ERR_RANGE, "shot " + std::to_string(b) + ": source outside its window");
        // the skipped cells depend on the window width alone (nzz is the
        // context's): computed once per width for the context's lifetime
        auto it = c->skip_cache.find(d.ncols);
        if (it == c->skip_cache.end()) {
            std::array<int, 8> v;
            sf_skip_cells(d.ncols, c->nzz, v.data(), v.data() + 4);
            it = c->skip_cache.emplace(d.ncols, v).first;
        }
        for (int q = 0; q < 4; q++) { d.skip_i[q] = it->second[q]; d.skip_j[q] = it->second[4 + q]; }
        d.orig = b;
        d.t_off = toff;  // per-shot traveltime windows (tables, anisotropic batches)
        toff += (long long)strip_pitch(c->nzz) * d.ncols;
        d.tape_off = tape_off;
        if (tape) tape_off += 4LL * nstrips * (d.ncols + 31) * 32;
        d.q_off = q_off;
        q_off += (long long)strip_pitch(c->nzz) * d.ncols;
        maxcols = std::max(maxcols, d.ncols);
        c->hshots[b] = d;
    }
    std::stable_sort(c->hshots.begin(), c->hshots.end(),
                     [](const ShotDev& a, const ShotDev& b) { return a.ncols > b.ncols; });
    c->batch_T_floats = toff;
    c->batch_tape_entries = tape_off;
    c->batch_q_cells = q_off;
    c->batch_maxcols = maxcols;
    c->tables_index.assign(nshots, 0);
    for (int q = 0; q < nshots; q++) c->tables_index[c->hshots[q].orig] = q;
    if (prev.size() == c->hshots.size() &&
        std::memcmp(prev.data(), c->hshots.data(), prev.size() * sizeof(ShotDev)) == 0)
        c->shots_gen = prev_gen;
    return SF_OK;
}

// One solve of every shot of the prepared batch: kernel, gang shape,
// buffers, parameters. per_shot_T: every shot keeps its own traveltime window
// (tables, anisotropic batches) instead of one window per gang. Sshots: the
// shots' own slowness windows (the qP slowness of an anisotropic batch's
// second solve), or nullptr for S.
int sf_fwd_configure(sf_ctx* c, int nrec, bool per_shot_T, bool tape, int gang_warps, cudaStream_t st,
                     FwdLaunch* L, const float* Sshots)
{
    const int nshots = (int)c->hshots.size();
    const int ld = strip_pitch(c->nzz);
    const int nstrips = (c->nzz + 31) / 32;
    const bool comp = c->arith == SF_ARITH_COMPENSATED;
    if (comp && c->warps > kMaxWarpsComp)
        return sf_fail(c, SF_ERR_ARG, "the compensated arithmetic runs at most 8 warps per CTA (sf_set_launch)");
    const bool ref = c->arith == SF_ARITH_REFERENCE;
    const size_t smem = sf_fwd_smem_bytes(c->warps, comp);
    // the interior-block kernels of taped batches are built for at most
    // kMaxWarpsTapedInterior warps per CTA
    c->batch_interior = !(tape && c->warps > kMaxWarpsTapedInterior) && sf_interior_loops(c);
    const void* kern = sf_kshots_kernel(tape, ref, c->batch_interior, comp);
    int G, NG;
    int rc = sf_gang_shape(c, kern, smem, nshots, nstrips, gang_warps, &G, &NG);
    if (rc) return rc;
    if ((long long)(nshots + NG - 1) / NG > kMaxSolves)
        return sf_fail(c, SF_ERR_ARG, "too many shots per gang for one launch; split the batch");
    c->last_G = G;
    c->last_NG = NG;
    rc = sf_dev_reserve(c, (void**)&c->d_shots, &c->cap_shots, nshots * sizeof(ShotDev));
    if (rc) return rc;
    CK(cudaMemcpyAsync(c->d_shots, c->hshots.data(), nshots * sizeof(ShotDev), cudaMemcpyHostToDevice, st));
    const long long t_per_gang = per_shot_T ? 0 : (long long)ld * c->batch_maxcols;
    const size_t tfloats = per_shot_T ? (size_t)c->batch_T_floats : (size_t)NG * t_per_gang;
    rc = sf_dev_reserve(c, (void**)&c->d_T, &c->cap_T, tfloats * sizeof(float));
    if (rc) return rc;
    if (comp) {
        rc = sf_dev_reserve(c, (void**)&c->d_Tl, &c->cap_Tl, tfloats * sizeof(float));
        if (rc) return rc;
    }
    const size_t hand_bytes =
        (size_t)NG * hand_words(nstrips, c->batch_maxcols, comp ? 2 : 1) * sizeof(unsigned long long);
    rc = sf_dev_reserve_zero(c, (void**)&c->d_hand, &c->cap_hand, hand_bytes);
    if (rc) return rc;
    const size_t nctr = gang_counters(NG);
    rc = sf_dev_reserve(c, (void**)&c->d_ctr, &c->cap_ctr, nctr * sizeof(unsigned));
    if (rc) return rc;
    if (tape) {
        size_t n = (size_t)c->batch_tape_entries;
        rc = sf_dev_reserve(c, (void**)&c->d_tcode, &c->cap_tcode, n);
        if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_tc1, &c->cap_tc1, n * sizeof(float));
        if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_tc2, &c->cap_tc2, n * sizeof(float));
        if (rc) return rc;
    }
    FwdParams& p = L->p;
    std::memset(&p, 0, sizeof(p));
    p.S = c->d_Sp;
    p.Sshots = Sshots;
    p.nzz = c->nzz;
    p.ld = ld;
    p.nxx = c->nxx;
    p.nb = c->nb;
    p.kc = c->kc;
    p.shots = c->d_shots;
    p.nshots = nshots;
    p.G = G;
    p.NG = NG;
    // The largest strip loop (taped, compensated) waits for instructions while
    // marches in both directions share an SM; one body for both then is the
    // faster, some 6% slower otherwise. Gangs march the same way at the same
    // time when each solves one shot and the windows are of one size (100
    // shots of 1701 x 351: 2.57 ms, 2.73 with one body), and hardly meet on an
    // SM when there are few (windows of about 1000 x 1001 cells: 40 shots 2.91
    // ms, with one body 3.18; 152 shots 8.20 and 6.70; from a queue, 400 shots
    // 21.0 and 17.1; 60 of about 430 x 351: 1.35 both).
    p.drift = nshots > NG || (c->hshots.back().ncols != c->batch_maxcols && 2 * NG > c->sms);
    p.maxcols = c->batch_maxcols;
    p.Tpool = c->d_T;
    p.Tlpool = comp ? c->d_Tl : nullptr;
    p.t_per_gang = t_per_gang;
    p.err = c->d_flags + 1;          // flags[1]: error flag
    p.wait_ns = c->wait_ns;
    p.hand = c->d_hand;
    p.bar = c->d_ctr;
    p.srange = Sshots ? c->d_srange : c->d_flags + 2;
    if (tape) {
        p.tcode = c->d_tcode;
        p.tc1 = c->d_tc1;
        p.tc2 = c->d_tc2;
    }
    p.rx = c->d_rx;
    p.rz = c->d_rz;
    p.nrec = nrec;
    L->kern = kern;
    L->grid = dim3(NG * G);
    L->block = dim3(c->warps * 32);
    L->smem = smem;
    L->nctr = nctr;
    L->hand_bytes = hand_bytes;
    return SF_OK;
}

int sf_kt_begin(sf_ctx* c, int k, cudaStream_t st)
{
    if (!c->timing) return SF_OK;
    c->kt_rec[k] = true;
    CK(cudaEventRecord(c->kt_ev[k][0], st));
    return SF_OK;
}

int sf_kt_end(sf_ctx* c, int k, cudaStream_t st)
{
    if (!c->timing) return SF_OK;
    CK(cudaEventRecord(c->kt_ev[k][1], st));
    return SF_OK;
}

// One forward launch (counters zeroed first), without the kernel timing.
int sf_fwd_launch(sf_ctx* c, FwdLaunch& L, float* d_picks, unsigned epoch, cudaStream_t st)
{
    L.p.picks = d_picks;
    L.p.epoch = epoch;
    CK(cudaMemsetAsync(L.p.bar, 0, L.nctr * sizeof(unsigned), st));
    if (c->hand_stale_f && epoch != kGraphEpoch) {
        CK(cudaMemsetAsync(c->d_hand, 0, c->cap_hand, st));
        c->hand_stale_f = false;
    }
    void* args[] = {&L.p};
    CK(cudaLaunchKernel(L.kern, L.grid, L.block, args, L.smem, st));
    return SF_OK;
}

int sf_fwd_enqueue(sf_ctx* c, FwdLaunch& L, float* d_picks, unsigned epoch, cudaStream_t st)
{
    int rc = sf_kt_begin(c, SF_KT_FORWARD, st);
    if (!rc) rc = sf_fwd_launch(c, L, d_picks, epoch, st);
    if (rc) return rc;
    return sf_kt_end(c, SF_KT_FORWARD, st);
}

// The qP pass of the prepared anisotropic batch (k_qp) over the traveltime
// windows of the first solves: the qP slowness windows into d_Sq, and with
// `fact` the derivative factors into d_vfac.
int sf_qp_launch(sf_ctx* c, bool fact, cudaStream_t st)
{
    QpParams q;
    std::memset(&q, 0, sizeof(q));
    q.S = c->d_S;
    q.nzz = c->nzz;
    q.ld = strip_pitch(c->nzz);
    q.nb = c->nb;
    q.kc = c->kc;
    q.shots = c->d_shots;
    q.nshots = (int)c->hshots.size();
    q.Tpool = c->d_T;
    q.Tlpool = c->d_Tl;
    const size_t npad = (size_t)c->nxx * c->nzz;
    for (int k = 0; k < 6; k++) q.cij[k] = c->d_cij_all + k * npad;
    std::memcpy(q.mm, c->mm, sizeof(q.mm));
    q.Sq = c->d_Sq;
    q.srange = c->d_srange;
    q.undef = c->d_srange + c->hshots.size();
    CK(cudaMemsetAsync(c->d_srange, 0, (c->hshots.size() + 1) * sizeof(int), st));
    q.vfac = fact ? c->d_vfac : nullptr;
    q.vfac_total = c->batch_q_cells;
    const bool comp = c->arith == SF_ARITH_COMPENSATED, ref = c->arith == SF_ARITH_REFERENCE;
    // x: the model's columns (grid-strided past 2048); y: groups of shots,
    // as many shots to a group as leave some 16 CTAs to every SM (their 64
    // warps; 12 shots of 1701 x 501 cells in groups of 8 take 102 us, of 16
    // 123 us, 4 shots in groups of 2 or 4 61-62 us)
    q.ncolumns = c->nxx;
    const long long want = 16LL * c->sms;
    q.chunk = (int)std::max(1LL, std::min<long long>(kQpChunk, (long long)c->nxx * q.nshots / want));
    const unsigned gx = (unsigned)std::min(c->nxx, 2048);
    const unsigned gy = (unsigned)std::min((q.nshots + q.chunk - 1) / q.chunk, 65535);
    void* args[] = {&q};
    CK(cudaLaunchKernel(sf_kqp_kernel(ref, comp, fact), dim3(gx, gy), dim3(128), args, 0, st));
    return SF_OK;
}

int sf_launch_shots(sf_ctx* c, int ani, int nrec, float* d_picks, bool keep_tables, bool tape, int gang_warps,
                    cudaStream_t st)
{
    const bool stall = c->stall_next;  // sf_test_stall_next_batch
    c->stall_next = false;
    int rc = sf_wait_slowness(c, st);
    if (rc) return rc;
    if (!ani) {
        FwdLaunch L;
        rc = sf_fwd_configure(c, nrec, keep_tables, tape, gang_warps, st, &L, nullptr);
        L.p.stall_handoff = stall ? 1 : 0;
        unsigned epoch = 0;
        if (!rc) rc = sf_launch_epoch(c, L.p.hand, L.hand_bytes, st, &epoch);
        if (!rc) rc = sf_fwd_enqueue(c, L, d_picks, epoch, st);
    } else {
        // eikonal_ani.cu:33-45: solve on S, qP pass, solve on the qP slowness;
        // every shot keeps its window between the launches
        rc = sf_dev_reserve(c, (void**)&c->d_Sq, &c->cap_Sq, (size_t)c->batch_q_cells * sizeof(float));
        if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_srange, &c->cap_srange, (c->hshots.size() + 1) * sizeof(int));
        if (!rc && tape)
            rc = sf_dev_reserve(c, (void**)&c->d_vfac, &c->cap_vfac, 3 * (size_t)c->batch_q_cells * sizeof(float));
        FwdLaunch L1, L2;
        if (!rc) rc = sf_fwd_configure(c, 0, true, false, gang_warps, st, &L1, nullptr);
        if (!rc) rc = sf_fwd_configure(c, nrec, true, tape, gang_warps, st, &L2, c->d_Sq);
        if (rc) return rc;
        // the second configuration may have grown the shared buffers
        L1.p.shots = c->d_shots;
        L1.p.Tpool = c->d_T;
        L1.p.Tlpool = L2.p.Tlpool;
        L1.p.hand = c->d_hand;
        L1.p.bar = c->d_ctr;
        L1.p.stall_handoff = L2.p.stall_handoff = stall ? 1 : 0;
        unsigned epoch = 0;
        rc = sf_kt_begin(c, SF_KT_FORWARD, st);
        if (!rc) rc = sf_launch_epoch(c, L1.p.hand, L1.hand_bytes, st, &epoch);
        if (!rc) rc = sf_fwd_launch(c, L1, nullptr, epoch, st);
        if (!rc) rc = sf_qp_launch(c, tape, st);
        if (!rc) rc = sf_launch_epoch(c, L2.p.hand, L2.hand_bytes, st, &epoch);
        if (!rc) rc = sf_fwd_launch(c, L2, d_picks, epoch, st);
        if (!rc) rc = sf_kt_end(c, SF_KT_FORWARD, st);
    }
    if (rc) return rc;
    c->tables_valid = keep_tables;
    c->tape_valid = tape;
    c->batch_nrec = nrec;
    c->batch_ani = ani;
    c->gcij_valid = false;
    return SF_OK;
}

int sf_upload_receivers(sf_ctx* c, const float* rx, const float* rz, int nrec, cudaStream_t st)
{
    if (nrec <= 0) return SF_OK;
    int rc = sf_dev_reserve(c, (void**)&c->d_rx, &c->cap_rx, nrec * sizeof(float));
    if (!rc) rc = sf_dev_reserve(c, (void**)&c->d_rz, &c->cap_rz, nrec * sizeof(float));
    if (rc) return rc;
    if (c->h_rx.size() == (size_t)nrec && std::equal(rx, rx + nrec, c->h_rx.begin()) &&
        std::equal(rz, rz + nrec, c->h_rz.begin()))
        return SF_OK;  // unchanged receivers stay on the device
    c->h_rx.assign(rx, rx + nrec);
    c->h_rz.assign(rz, rz + nrec);
    c->recv_gen++;
    CK(cudaMemcpyAsync(c->d_rx, c->h_rx.data(), nrec * sizeof(float), cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(c->d_rz, c->h_rz.data(), nrec * sizeof(float), cudaMemcpyHostToDevice, st));
    return SF_OK;
}

int sf_check_flags(sf_ctx* c, cudaStream_t st)
{
    CK(cudaStreamSynchronize(st));
    int err = 0;
    CK(cudaMemcpy(&err, c->d_flags + 1, sizeof(int), cudaMemcpyDeviceToHost));
    if (err) {
        cudaMemset(c->d_flags + 1, 0, sizeof(int));
        return sf_fail(c, SF_ERR_TIMEOUT, "an in-kernel wait gave up; results of the launch are void");
    }
    return SF_OK;
}

extern "C" int sf_synchronize(sf_ctx* c, void* stream)
{
    if (!c) return SF_ERR_ARG;
    CK(cudaSetDevice(c->dev));
    return sf_check_flags(c, (cudaStream_t)stream);
}

extern "C" int sf_batch_forward(sf_ctx* c, int ani, const sf_shot* shots, int nshots, const float* rx,
                                const float* rz, int nrec, float* picks, int picks_mem, int flags,
                                void* stream)
{
    if (!c || !shots || nshots <= 0 || nrec < 0 || (nrec > 0 && (!rx || !rz || !picks)))
        return sf_fail(c, SF_ERR_ARG, "bad batch arguments");
    if (ani && !c->have_cij) return sf_fail(c, SF_ERR_STATE, "anisotropic solve needs sf_set_stiffness");
    const bool tape = (flags & SF_KEEP_TAPE) != 0, tables = (flags & SF_KEEP_TABLES) != 0;
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    c->tape_valid = false;
    c->tables_valid = false;
    int rc = sf_prepare_shots(c, shots, nshots, tape);
    if (rc) return rc;
    rc = sf_upload_receivers(c, rx, rz, nrec, st);
    if (rc) return rc;
    float* dp = nullptr;
    if (nrec > 0) {
        if (picks_mem == SF_MEM_DEVICE) dp = picks;
        else {
            rc = sf_dev_reserve(c, (void**)&c->d_picks, &c->cap_picks, (size_t)nshots * nrec * sizeof(float));
            if (rc) return rc;
            dp = c->d_picks;
        }
    }
    rc = sf_launch_shots(c, ani, nrec, dp, tables, tape, c->gang_warps, st);
    if (rc) return rc;
    c->batch_nshots = nshots;
    c->batch_picks = dp;
    if (nrec > 0 && picks_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(picks, dp, (size_t)nshots * nrec * sizeof(float), cudaMemcpyDeviceToHost, st));
        return sf_check_flags(c, st);
    }
    return SF_OK;
}

// A traveltime window of the solver's column stride to the caller's nzz x ncols buffer.
static int table_out(sf_ctx* c, const float* window, int ncols, float* T, int mem, cudaStream_t st)
{
    const size_t n = (size_t)c->nzz * ncols;
    float* out = T;
    if (mem != SF_MEM_DEVICE) {
        int rc = sf_dev_reserve(c, (void**)&c->d_Tc, &c->cap_Tc, n * sizeof(float));
        if (rc) return rc;
        out = c->d_Tc;
    }
    // Programmatic (k_unpitch waits for the work before it itself), which takes
    // the launch latency out of a row of table copies: 121 tables of 1203 x 187
    // after their solve 1.37 -> 1.16 ms in all. Plain edges in a captured graph.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const bool plain = cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
    if (plain) cudaGetLastError();
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(ncols, 65535));
    cfg.blockDim = dim3(std::min(256, strip_pitch(c->nzz)));
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = plain ? 0 : 1;
    CK(cudaLaunchKernelEx(&cfg, k_unpitch, window, (int)c->nzz, ncols, (int)strip_pitch(c->nzz), out));
    if (mem == SF_MEM_DEVICE) return SF_OK;
    CK(cudaMemcpyAsync(T, out, n * sizeof(float), cudaMemcpyDeviceToHost, st));
    return sf_check_flags(c, st);
}

extern "C" int sf_batch_table(sf_ctx* c, int shot, float* T, int mem, void* stream)
{
    if (!c || !T) return SF_ERR_ARG;
    if (!c->tables_valid) return sf_fail(c, SF_ERR_STATE, "last batch did not keep tables");
    if (shot < 0 || shot >= (int)c->hshots.size()) return sf_fail(c, SF_ERR_ARG, "shot out of range");
    CK(cudaSetDevice(c->dev));
    const ShotDev& d = c->hshots[c->tables_index[shot]];
    cudaStream_t st = (cudaStream_t)stream;
    return table_out(c, c->d_T + d.t_off, d.ncols, T, mem, st);
}

// The tape is kept per (sweep, strip) in the strip's skewed step order: entry
// [step * 32 + lane] is the node of row 32k + lane (rows downward, sweeps 0
// and 2) or 32k + 31 - lane (upward, sweeps 1 and 3) and window column of
// march step - lane (columns rightward, sweeps 0 and 1, else leftward).
// This entry point unskews one shot's codes into [sweep][column][row].
extern "C" int sf_batch_tape_codes(sf_ctx* c, int shot, uint8_t* codes, int mem, void* stream)
{
    if (!c || !codes) return SF_ERR_ARG;
    if (!c->tape_valid) return sf_fail(c, SF_ERR_STATE, "last batch did not keep a tape");
    if (shot < 0 || shot >= (int)c->hshots.size()) return sf_fail(c, SF_ERR_ARG, "shot out of range");
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    const ShotDev& d = c->hshots[c->tables_index[shot]];
    const int nzz = c->nzz, ncols = d.ncols, nstrips = (nzz + 31) / 32;
    const size_t per_strip = (size_t)(ncols + 31) * 32;
    std::vector<uint8_t> raw(4 * (size_t)nstrips * per_strip), out(4 * (size_t)ncols * nzz, 0);
    CK(cudaMemcpyAsync(raw.data(), c->d_tcode + d.tape_off, raw.size(), cudaMemcpyDeviceToHost, st));
    int rc = sf_check_flags(c, st);
    if (rc) return rc;
    for (int sw = 0; sw < 4; sw++) {
        const bool zdown = (sw == 0 || sw == 2), xright = (sw == 0 || sw == 1);
        for (int k = 0; k < nstrips; k++) {
            const uint8_t* blk = raw.data() + ((size_t)sw * nstrips + k) * per_strip;
            for (int step = 0; step < ncols + 31; step++)
                for (int lane = 0; lane < 32; lane++) {
                    const int r = zdown ? 32 * k + lane : 32 * k + 31 - lane, m = step - lane;
                    if (r >= nzz || m < 0 || m >= ncols) continue;
                    const int j = xright ? m : ncols - 1 - m;
                    out[((size_t)sw * ncols + j) * nzz + r] = blk[(size_t)step * 32 + lane] & 0x1f;  // kKept is 0 here
                }
        }
    }
    CK(cudaMemcpyAsync(codes, out.data(), out.size(),
                       mem == SF_MEM_DEVICE ? cudaMemcpyHostToDevice : cudaMemcpyHostToHost, st));
    CK(cudaStreamSynchronize(st));
    return SF_OK;
}

extern "C" int sf_time_propagation(sf_ctx* c, int ani, float sx, float sz, float* T, int T_mem, void* stream)
{
    if (!c || !T) return sf_fail(c, SF_ERR_ARG, "null argument");
    if (ani && !c->have_cij) return sf_fail(c, SF_ERR_STATE, "anisotropic solve needs sf_set_stiffness");
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    sf_shot s{sx, sz, 0, c->nxx};
    int rc = sf_prepare_shots(c, &s, 1, false);
    if (rc) return rc;
    rc = sf_launch_shots(c, ani, 0, nullptr, true, false, c->gang_warps, st);
    if (rc) return rc;
    if (T_mem == SF_MEM_DEVICE) c->tables_valid = false;
    return table_out(c, c->d_T, c->nxx, T, T_mem, st);
}

extern "C" int sf_compute_seismogram(sf_ctx* c, const float* T_dev, const float* rx, const float* rz,
                                     int nrec, float* picks, int picks_mem, void* stream)
{
    if (!c || !T_dev || nrec < 0 || (nrec > 0 && (!rx || !rz || !picks))) return SF_ERR_ARG;
    if (nrec == 0) return SF_OK;
    CK(cudaSetDevice(c->dev));
    cudaStream_t st = (cudaStream_t)stream;
    int rc = sf_upload_receivers(c, rx, rz, nrec, st);
    if (rc) return rc;
    float* dp = picks;
    if (picks_mem == SF_MEM_HOST) {
        rc = sf_dev_reserve(c, (void**)&c->d_picks, &c->cap_picks, (size_t)nrec * sizeof(float));
        if (rc) return rc;
        dp = c->d_picks;
    }
    k_picks<<<(nrec + 127) / 128, 128, 0, st>>>(T_dev, c->nzz, c->nxx, 0, c->nb, c->dx, c->dz, c->d_rx,
                                                c->d_rz, nrec, dp);
    CK(cudaGetLastError());
    if (picks_mem == SF_MEM_HOST) {
        CK(cudaMemcpyAsync(picks, dp, (size_t)nrec * sizeof(float), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    return SF_OK;
}

// The allocation-free per-shot entry point shares this translation unit's
// instantiation of k_shots.
#include "sf_noalloc.cu"
