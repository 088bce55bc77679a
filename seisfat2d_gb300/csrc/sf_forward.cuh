// Whole-shot forward kernel: a gang of CTAs solves one shot window at a time
// (init, 4 sweeps, receiver picks) and takes the next shot of the queue. The same kernel with one shot and one CTA is the per-shot drop-in
// solver. An anisotropic batch (eikonal_ani.cu:33-45) is three launches: the
// solve of every shot on S, the qP pass over every shot's window (k_qp, a
// map over cells), and the solve of every shot on its own qP slowness.
#pragma once
#include "sf_sweep.cuh"

namespace sf {

// Device description of one shot (host computes it once per batch).
struct ShotDev {
    int c0, ncols;        // window: padded columns [c0, c0+ncols)
    int sIdx, sIdz;       // source node, global padded indices
    float sx, sz;         // source position (m)
    int skip_i[4];        // cells the reference schedule never updates
    int skip_j[4];        // (window coordinates, -1 = none), per sweep
    int orig;             // index of the shot in the caller's order
    int pad_;
    long long t_off;      // traveltime window offset (floats, column stride strip_pitch) when tables are kept
    long long tape_off;   // tape offset (entries)
    long long q_off;      // offset of its qP slowness window and derivative factors (floats, column stride strip_pitch)
};

struct FwdParams {
    const float* S;       // padded slowness, column stride ld
    const float* Sshots;  // per-shot slowness windows at q_off (same stride) instead of S, or nullptr
    int nzz, nxx, nb;
    int ld;               // column stride of the slowness and traveltime windows: strip_pitch(nzz) (VEC), or nzz
    Consts kc;
    const ShotDev* shots;
    int nshots;
    int G;                // CTAs per gang (one gang solves one shot at a time)
    int NG;               // gangs; gang k solves shot k first, then takes shots from a queue
    bool drift;           // gangs may be at sweeps of both march directions at the same time
    int maxcols;          // widest window of the batch
    float* Tpool;
    float* Tlpool;        // compensated: lo parts of the traveltimes, same layout as Tpool
    long long t_per_gang; // > 0: each gang reuses Tpool + gang * t_per_gang
    int* err;
    // per gang (hand_words): tagged strip handoff pairs [4 sweeps][nstrips]
    // [hand_pitch] (x2 compensated), then progress words [4 sweeps][nstrips]
    unsigned long long* hand;
    const int* srange;    // nonzero: the slowness has a value outside in_fast_range (per shot with Sshots)
    unsigned* bar;        // gang_counters(NG), zeroed
    unsigned epoch;       // launch number (tags: epoch << 10 | shot-solve number)
    unsigned long long wait_ns;  // time limit of the bounded waits
    int stall_handoff;    // test of the timeout path: consumers wait for a tag no producer writes
    // tape
    uint8_t* tcode;
    float* tc1;
    float* tc2;
    // receivers
    const float* rx;
    const float* rz;
    int nrec;
    float* picks;         // nshots x nrec, caller order
};

// 3x3 initial values of one solve into shared memory (modeling.cu:293-306):
// FP32 as the reference build computes them (REF) or in FP64, rounded once.
template <bool REF>
__device__ __forceinline__ void init_block(const FwdParams& p, const ShotDev& sh, const float* Sw,
                                           float* out)
{
    const int tid = threadIdx.x;
    if (tid < 9) {
        const int a = tid % 3, bb = tid / 3;
        const int zi = sh.sIdz + a - 1, xl = sh.sIdx - sh.c0 + bb - 1;
        const float s = Sw[zi + (size_t)xl * p.ld];
        if (REF)
            out[tid] = src_value_f32(s, zi, xl + sh.c0, p.nb, p.kc.dx, p.kc.dz, sh.sx, sh.sz);
        else
            out[tid] = __double2float_rn(
                __dmul_rn((double)s, src_dist(zi, xl + sh.c0, p.nb, p.kc.dx, p.kc.dz, sh.sx, sh.sz)));
    }
}

__device__ __forceinline__ size_t tape_strip_base(long long tape_off, int sweep, int k, int nstrips,
                                                  int ncols)
{
    return (size_t)tape_off + ((size_t)sweep * nstrips + k) * (size_t)(ncols + 31) * 32;
}

// Where a gang's warps sit: warp w of CTA g of the gang is slot w*G + g, so
// consecutive slots, which run consecutive strips, are on different CTAs and SMs.
struct GangPos {
    int gang, g, warp, slot, slots;
};

__device__ __forceinline__ GangPos gang_pos(int G)
{
    GangPos q;
    q.gang = blockIdx.x / G;
    q.g = blockIdx.x % G;
    q.warp = threadIdx.x >> 5;
    q.slots = G * (blockDim.x >> 5);
    q.slot = q.warp * G + q.g;
    return q;
}

// One strip of a sweep in the loop form the shot needs.
template <int DIR, bool TAPE, bool REF, bool INTERIOR, bool COMP, bool VEC>
__device__ __forceinline__ void strip(const StripArgs& a, bool exact)
{
    if (exact)
        run_strip<DIR, TAPE, REF, false, false, COMP, true, VEC>(a);
    else if (a.kc.dx == a.kc.dz)
        run_strip<DIR, TAPE, REF, INTERIOR, true, COMP, false, VEC>(a);
    else
        run_strip<DIR, TAPE, REF, INTERIOR, false, COMP, false, VEC>(a);
}

// The four sweeps of one solve of the current shot. Sweeps 0 (down) and 1
// (up) march to the right, 2 and 3 to the left. The strips of each such pair
// are one list of tasks in dependency order (sweep 0's strips top to bottom,
// then sweep 1's bottom to top), dealt to the gang's warps in turn: sweep 1's
// bottom strip starts as soon as a warp is free and sweep 0's bottom strip
// has written its first columns, instead of after the whole sweep. With a
// warp per task a pair of sweeps takes ncols + 2 nstrips lags steps instead
// of 2 (ncols + nstrips lags). Every task waits only on earlier ones (the
// strip before it in its sweep; its own rows in the sweep before), and each
// warp runs its tasks in order, so the schedule cannot deadlock. No barrier
// between sweeps. Square cells (dx and dz equal) run the strip loops'
// square-cell form. COMP: compensated arithmetic, lo parts in Tl, two handoff
// pairs per column.
template <bool TAPE, bool REF, bool INTERIOR, bool COMP, bool VEC>
__device__ void solve_window(const FwdParams& p, const ShotDev& sh, const GangPos& gp, const float* Sw, float* T, float* Tl, unsigned tag, bool exact, CtaShared* cs, unsigned char* rings)
{
    const int nzz = p.nzz, ncols = sh.ncols;
    const int nstrips = (nzz + 31) >> 5;
    constexpr size_t HS = COMP ? 2 : 1;
    const size_t row = (size_t)hand_pitch(p.maxcols) * HS;
    unsigned long long* hb = p.hand + (size_t)gp.gang * hand_words(nstrips, p.maxcols, HS);
    unsigned long long* prog = hb + 4 * (size_t)nstrips * row;
    StripArgs a;
    a.S = Sw;
    a.ld = p.ld;
    a.T = T;
    a.Tl = Tl;
    a.nzz = nzz;
    a.ncols = ncols;
    a.sIdz = sh.sIdz;
    a.sIdx = sh.sIdx - sh.c0;
    a.kc = p.kc;
    a.init = cs->init;
    a.ring = rings + (size_t)gp.warp * ring_bytes<COMP>();
    a.sh = cs;
    a.err = p.err;
    a.tcode = nullptr;
    a.tc1 = nullptr;
    a.tc2 = nullptr;
    a.tag = tag;
    a.tag_in = p.stall_handoff ? 1u : tag;  // epoch 0 is never used, zeroed pairs carry tag 0
#pragma unroll 1
    for (int task = gp.slot; task < 4 * nstrips; task += gp.slots) {
        const int sw = task / nstrips, pidx = task - sw * nstrips;
        a.k = (sw & 1) ? nstrips - 1 - pidx : pidx;
        a.right = sw < 2;
        a.down = !(sw & 1);
        a.sw0 = sw == 0;
        a.skip_i = sh.skip_i[sw];
        a.skip_j = sh.skip_j[sw];
        unsigned long long* hs = hb + ((size_t)sw * nstrips + pidx) * row;
        a.h_in = (pidx > 0) ? hs : nullptr;
        a.h_out = (pidx < nstrips - 1) ? hs + row : nullptr;
        a.prog_in = (sw > 0) ? prog + (size_t)(sw - 1) * nstrips + a.k : nullptr;
        a.follow = sw & 1;
        a.prog_out = (sw < 3) ? prog + (size_t)sw * nstrips + a.k : nullptr;
        a.publish = (sw & 1) ? 0 : publish_every(nstrips - 1 - pidx);
        if (TAPE) {
            size_t base = tape_strip_base(sh.tape_off, sw, a.k, nstrips, ncols);
            a.tcode = p.tcode + base;
            a.tc1 = p.tc1 + base;
            a.tc2 = p.tc2 + base;
        }
        if (TAPE && COMP && INTERIOR && p.drift)
            strip<(TAPE && COMP && INTERIOR) ? 0 : 1, TAPE, REF, INTERIOR, COMP, VEC>(a, exact);
        else if (sw < 2)
            strip<1, TAPE, REF, INTERIOR, COMP, VEC>(a, exact);
        else
            strip<-1, TAPE, REF, INTERIOR, COMP, VEC>(a, exact);
    }
}

// Persistent gangs of G CTAs: gang k solves shot k, then the next of the queue
// (shots are sorted widest window first). The grid never exceeds what the device can
// hold at once, so every gang's CTAs are resident together. INTERIOR: the
// strip loops' bounds-test-free body for interior blocks (see run_strip).
// COMP: compensated arithmetic (node_update_comp; the 3x3 initial values are
// the FP64 ones rounded once).
template <bool TAPE, bool REF, bool INTERIOR, bool COMP = false, bool VEC = true>
// Register bounds: 168 keep three warps per scheduler (and 8 per CTA); the
// plain FP32 kernels run CTAs of up to 16 warps, hence 128.
__global__ void __maxnreg__((COMP || (TAPE && INTERIOR)) ? 168 : 128)
    k_shots(FwdParams p)
{
    static_assert(!(COMP && REF), "the compensated arithmetic has no reference-build variant");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CtaShared* cs = reinterpret_cast<CtaShared*>(smem_raw);
    unsigned char* rings = smem_raw + ((sizeof(CtaShared) + 15) & ~size_t(15));
    const int tid = threadIdx.x;
    const GangPos gp = gang_pos(p.G);
    const int nzz = p.nzz;
    unsigned* bar = p.bar + gp.gang;
    unsigned nbar = 0;
    if (tid == 0) {
        cs->abort_flag = 0;
        cs->wait_ns = p.wait_ns ? p.wait_ns : kSpinNs;
    }
    __syncthreads();
    int it = 0;
#pragma unroll 1
    for (int b = gp.gang; b < p.nshots; it++) {
        const ShotDev sh = p.shots[b];
        float* T = (p.t_per_gang > 0) ? p.Tpool + (size_t)gp.gang * p.t_per_gang : p.Tpool + sh.t_off;
        float* Tl = !COMP ? nullptr
                          : (p.t_per_gang > 0) ? p.Tlpool + (size_t)gp.gang * p.t_per_gang : p.Tlpool + sh.t_off;
        // the shot's slowness window: columns c0.. of S, or its own qP slowness
        const float* Sw = p.Sshots ? p.Sshots + sh.q_off : p.S + (size_t)sh.c0 * p.ld;
        const unsigned tag = (p.epoch << 10) | (unsigned)(it & 1023);
        init_block<REF>(p, sh, Sw, cs->init);
        __syncthreads();
        const bool exact = p.kc.mflags != kFastFlags || p.srange[p.Sshots ? b : 0] != 0;
        solve_window<TAPE, REF, INTERIOR, COMP, VEC>(p, sh, gp, Sw, T, Tl, tag, exact, cs, rings);
        // receivers (modeling.cu:161-194), spread over the gang once the field is final
        if (p.nrec > 0 && p.picks) {
            gang_barrier(bar, (++nbar) * p.G, cs, p.err);
            for (int r = (gp.g * (blockDim.x >> 5) + gp.warp) * 32 + (tid & 31); r < p.nrec; r += gp.slots * 32) {
                int i, j;
                float xd, zd;
                float v = __int_as_float(0x7fc00000);
                if (pick_geom(p.rx[r], p.rz[r], p.kc.dx, p.kc.dz, p.nb, nzz, sh.ncols, sh.c0, i, j, xd, zd))
                    v = pick_value(T, p.ld, i, j, xd, zd);
                p.picks[(size_t)sh.orig * p.nrec + r] = v;
            }
        }
        b = next_shot(p.bar, p.NG, p.G, gp.gang, gp.g, it, nbar, cs, p.err);
    }
}

// The qP pass of an anisotropic batch, get_quasi_slowness
// (eikonal_ani.cu:47-111), on every shot's window once the first solves are
// done: the qP slowness of each window cell from the central differences of
// the window's traveltimes (of their pairs in the compensated arithmetic)
// and the decoded stiffness; the window's edge cells (nb of them) and the
// source node keep S. FACT (taped batches): also the derivative factors dSq/dS,
// dSq/dC11, dSq/dC13 of each cell. A map over the model's cells and the shots:
// 128 threads over a column's rows (coalesced, z fastest), blockIdx.x strides
// over the columns, blockIdx.y over groups of p.chunk shots. The pass is bound
// by its instructions (IEEE quotients), and 18 of the 23 of a cell and shot
// (decoding and normalising the six stiffnesses) depend on the cell alone, so
// a thread does them once and goes through the group's shots: 100 shots of
// 1701 x 501 cells 1.47 -> 0.55 ms (compensated, no factors).
constexpr int kQpChunk = 16;  // shots per group at most
struct QpParams {
    const float* S;       // padded slowness, column stride nzz (as the codes)
    int nzz, nb;
    int ld;               // column stride of the shots' windows
    Consts kc;
    const ShotDev* shots;
    int nshots, ncolumns, chunk;  // chunk <= kQpChunk
    const float* Tpool;   // per-shot traveltime windows at t_off
    const float* Tlpool;  // their lo parts (compensated)
    const uint16_t* cij[6];
    float mm[12];
    float* Sq;            // per-shot qP slowness windows at q_off
    int* srange;          // per shot: set when its qP slowness has a value outside in_fast_range
    int* undef;           // FACT: set when a derivative factor is not finite
    float* vfac;          // FACT: dSq/dS, dSq/dC11, dSq/dC13 per window cell (3 x vfac_total)
    long long vfac_total;
};

template <bool REF, bool COMP, bool FACT>
__global__ void __launch_bounds__(128) k_qp(QpParams p)
{
    const int nzz = p.nzz, nb = p.nb, ld = p.ld;
    // the group's windows: columns [c0, c0 + ncols), source node, pool offsets
    __shared__ int4 win[kQpChunk];
    __shared__ longlong2 off[kQpChunk];
#pragma unroll 1
    for (int b0 = blockIdx.y * p.chunk; b0 < p.nshots; b0 += gridDim.y * p.chunk) {
        const int nsh = min(p.chunk, p.nshots - b0);
        __syncthreads();
        if ((int)threadIdx.x < nsh) {
            const ShotDev& sh = p.shots[b0 + threadIdx.x];
            win[threadIdx.x] = make_int4(sh.c0, sh.ncols, sh.sIdx, sh.sIdz);
            off[threadIdx.x] = make_longlong2(sh.t_off, sh.q_off);
        }
        __syncthreads();
#pragma unroll 1
        for (int jg = blockIdx.x; jg < p.ncolumns; jg += gridDim.x) {
            bool any = false;
            for (int k = 0; k < nsh; k++) any |= (unsigned)(jg - win[k].x) < (unsigned)win[k].y;
            if (!any) continue;
#pragma unroll 1
            for (int i = threadIdx.x; i < nzz; i += blockDim.x) {
                const size_t g = (size_t)i + (size_t)jg * nzz;
                const float s = p.S[g];
                const float c11 = decode_c(p.cij[0][g], p.mm[0], p.mm[1]);
                const float c13 = decode_c(p.cij[1][g], p.mm[2], p.mm[3]);
                const float c15 = decode_c(p.cij[2][g], p.mm[4], p.mm[5]);
                const float c33 = decode_c(p.cij[3][g], p.mm[6], p.mm[7]);
                const float c35 = decode_c(p.cij[4][g], p.mm[8], p.mm[9]);
                const float c55 = decode_c(p.cij[5][g], p.mm[10], p.mm[11]);
                const QpCell cell = qp_cell(s, c11, c13, c15, c33, c35, c55);
                const bool row = i >= nb && i < nzz - nb;
#pragma unroll 2
                for (int k = 0; k < nsh; k++) {
                    const int4 w = win[k];
                    const int j = jg - w.x;
                    if ((unsigned)j >= (unsigned)w.y) continue;
                    const longlong2 o = off[k];
                    const size_t idx = (size_t)i + (size_t)j * ld;
                    float out = s;
                    float fS = 1.0f, f11 = 0.0f, f13 = 0.0f;
                    if (row && j >= nb && j < w.y - nb && !(i == w.w && jg == w.z)) {
                        const float* Tc = p.Tpool + o.x + idx;
                        // central differences; of the pairs in the compensated arithmetic
                        float dzr, dxr;
                        if (COMP) {
                            const float* Lc = p.Tlpool + o.x + idx;
                            dzr = ff_diff(Tc[1], Lc[1], Tc[-1], Lc[-1]);
                            dxr = ff_diff(Tc[ld], Lc[ld], Tc[-(long)ld], Lc[-(long)ld]);
                        } else {
                            dzr = fsub(Tc[1], Tc[-1]);
                            dxr = fsub(Tc[ld], Tc[-(long)ld]);
                        }
                        out = qp_slowness<REF>(dzr, dxr, p.kc.dx, p.kc.dz, cell);
                        if (FACT)
                            qp_factors(dzr, dxr, s, p.kc.dx, p.kc.dz, c11, c13, c15, c33, c35, c55, fS, f11, f13);
                    }
                    p.Sq[o.y + idx] = out;
                    if (!in_fast_range(out, p.kc.dx, p.kc.dz)) p.srange[b0 + k] = 1;
                    if (FACT) {
                        float* f = p.vfac + o.y + idx;
                        f[0] = fS;
                        f[p.vfac_total] = f11;
                        f[2 * p.vfac_total] = f13;
                        if (!(fabsf(fS) + fabsf(f11) + fabsf(f13) < INFINITY)) *p.undef = 1;
                    }
                }
            }
        }
    }
}

}  // namespace sf
