// Adjoint-state gradient: reverse sweeps over the forward tape.
//
// The forward pass (k_shots<true>) records, for every node of every sweep,
// which candidate set the node (code bits 0-2), which slowness cell that
// candidate read (bits 3-4) and two derivative coefficients c1, c2 (see
// include/seisfat2d.h). The discrete adjoint of one sweep is then the linear
// recurrence, in pull form, for node n = (i, j) of a sweep with signs (sz, sx):
//
//   mu(n)  = (lam(n) + (pv(i+sz, j) + pev(i+sz, j+sx))) + pe(i, j+sx)
//   lam(n) <- mu(n) if the node kept its value (code 0), else 0
//   pv/pe/pev(n) = mu(n) * dT(n)/d{tv, te, tev}   (pushed to the upwind nodes)
//   v(n)   = mu(n) * c2                           (term of the node's slowness cell)
//
// swept in the reverse order. It is the forward's dependency pattern with the
// march reversed, so the same strip-systolic schedule runs it: lane l owns a
// row, the lane above supplies the sum of its pv of the previous step and its
// pev of the step before by one shfl (the two pushes of the upwind row are
// summed by their sender), the lane's own previous pe is kept in a register.
// The tape was written in the forward strip's skewed step order, which makes
// the reverse read of one step 32 consecutive entries (lane l of the reverse
// march is lane 31-l of the forward one), and of a block of four steps one
// contiguous run. The reverse sweeps overlap in pairs as the forward's do.
//
// A step is a handful of multiply-adds on a short chain (one shfl, four
// dependent operations), so its cost is its instruction stream: the block's
// tape rows come in by three 16-byte copies per lane, the pushes are mu times
// three coefficients selected from the code without branches, and the pair
// for the next strip is one 16-byte store.
//
// The node terms v overwrite the tape's c2; the gradient gather (gather_tile)
// sums them per slowness cell, either in its own launch (k_gather) or inside
// the reverse-sweep launch (k_adjoint_gather), where each tile starts as soon
// as the last reverse sweep of every shot has finished it.
#pragma once
#include <cooperative_groups.h>

#include "sf_adjoint_params.cuh"
#include "sf_forward.cuh"

namespace sf {

constexpr int kGT = 32;    // gather tile columns (the column blocks of the gradient gather)
// Strip loop of the reverse sweeps: steps per block, staging leads of the
// columns with their tape rows and of the upwind strip's pairs, ring lengths
// (columns; blocks of tape rows; pairs). A block's prefetches never refill a
// slot that this block or the one before it reads.
constexpr int kU = 4;
constexpr int kLookA = 12;
constexpr int kPairLookA = 8;
constexpr int kAheadA = kPairLookA + kU;  // a consumer's fall-back distance after a stall
constexpr int kRingA = 52;
constexpr int kTapeBlocks = kLookA / kU + 2;
constexpr int kPairsA = 16;
static_assert(kLookA % kU == 0 && kPairLookA % kU == 0 && kPairLookA <= kLookA && kRingA % kU == 0 &&
              kRingA >= 31 + kLookA + 2 * kU && kPairsA >= kPairLookA + kU && kPairsA % kU == 0, "adjoint rings too small");
static_assert(kU == 4, "a block's tape rows are one 16-byte copy per lane");

struct AdjTape {
    float c1[kU * 32], c2[kU * 32];
    uint8_t code[kU * 32];
};
struct __align__(16) AdjRing {
    float L[kRingA * 32];             // lambda, one column of the strip's rows per slot
    AdjTape tape[kTapeBlocks];        // forward step order: row U-1-u is the block's step u
    uint4 pair[kPairsA];              // {pv, tag, pev, tag} of march q at q mod kPairsA
};

struct AdjStripArgs {
    float* lam;        // window adjoint field (column stride strip_pitch(nzz)), in place
    int nzz, ncols, k;
    bool down, right;  // directions of the reverse march
    const uint8_t* tcode;  // tape of this (sweep, strip): entries [fstep*32 + flane]
    const float* tc1;
    float* tc2;            // overwritten with v = mu * c2
    uint8_t* vflag;        // one per 1024 tape entries of the batch: set when a term is not zero
    size_t tape_base;      // the strip's first tape entry
    AdjRing* ring;
    CtaShared* sh;
    const unsigned long long* h_in;  // {pv,tag},{pev,tag} of the upwind strip's row (nullptr: first strip)
    unsigned long long* h_out;       // pairs this strip feeds to the next one (nullptr: last strip)
    unsigned tag;
    // columns of the strip finished by the reverse sweep before this one, and by this one (see StripArgs)
    const unsigned long long* prog_in;
    bool follow;
    unsigned long long* prog_out;
    int publish;
    int* err;
    // last reverse sweep inside a fused launch: count each column block of
    // kGT padded columns once all lanes have finished its columns
    unsigned* ready;   // this strip's row of counters (nullptr: no counting)
    int c0;            // the window's first padded column
};

// INTERIOR: blocks whose marches all lie inside the window run a body without
// bounds tests. One body serves the four sweeps (see run_strip).
template <bool INTERIOR>
__device__ __forceinline__ void adj_strip(const AdjStripArgs& a)
{
    const int lane = threadIdx.x & 31;
    const int nzz = a.nzz, ncols = a.ncols;
    const int rb = 32 * a.k;
    const int r = a.down ? rb + lane : rb + 31 - lane;
    const bool vrow = r < nzz;
    const int tix = r - rb;
    const int flane = 31 - lane;  // this row's lane in the forward strip
    AdjRing& R = *a.ring;
    CtaShared* sh = a.sh;
    const bool consumer = a.h_in != nullptr;
    const bool lane0 = lane == 0;
    const bool feeds = (lane == 31) && (a.h_out != nullptr);
    const int nsteps = ncols + 31;
    auto col_of = [&](int m) { return a.right ? m : ncols - 1 - m; };
    // lane 8 u + c copies 16 bytes, rows rb+4c .. rb+4c+3, of the block's column u
    const int vu = lane >> 3, vc = 4 * (lane & 7);
    const long long ld = strip_pitch(nzz), dL = a.right ? ld : -ld;
    const long long first = (long long)col_of(0) * ld + vu * dL + rb + vc;
    const float* pL = a.lam + first;
    // the lane's 16 bytes of a block's tape rows (rows of steps q+U-1 .. q, forward step order)
    const long long fs0 = (long long)(ncols + 31 - kU) * 32;
    const float* pT1 = a.tc1 + fs0 + 4 * lane;
    const float* pT2 = a.tc2 + fs0 + 4 * lane;
    const uint8_t* pTc = a.tcode + fs0 + 16 * lane;
    // marches q .. q+U-1: columns into the next slots, tape rows into block slot tb
    // FAST: every march of the call is inside the window (no bounds tests)
    unsigned so = vu * 32, wo = (kRingA - 31 - kU + vu) * 32;  // ring offsets of the columns staged and written back
    auto stage = [&](int q, int tb, auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        if (FAST || q + vu < ncols) cp_async16_cg(&R.L[so + vc], pL);
        so = ring_next<kU * 32, kRingA * 32>(so);
        pL += kU * dL;
        AdjTape& t = R.tape[tb];
        if (FAST || q + kU - 1 - (lane >> 3) < nsteps) {
            cp_async16_cg(&t.c1[4 * lane], pT1);
            cp_async16_cg(&t.c2[4 * lane], pT2);
        }
        if (lane < 8 && (FAST || q + kU - 1 - (lane >> 1) < nsteps)) cp_async16_cg(&t.code[16 * lane], pTc);
        pT1 -= 32 * kU;
        pT2 -= 32 * kU;
        pTc -= 32 * kU;
    };
    const bool pair_lane = consumer && lane < kU;
    const unsigned long long* pP = a.h_in + 2 * lane;
    unsigned po = lane % kPairsA, pi = 0;  // ring slots of the pairs staged and read
    if (!consumer && lane < kPairsA) R.pair[lane] = make_uint4(0, 0, 0, 0);
    auto stage_pairs = [&](int q, auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        if (pair_lane && (FAST || q + lane < ncols)) cp_async16_cg(&R.pair[po], pP);
        pP += 2 * kU;
        po = (po + kU) % kPairsA;
    };
    int avail = a.prog_in ? 0 : 0x7fffffff;
    auto ensure = [&](int q) {  // marches below q may be staged
        if (q > avail) {
            avail = wait_progress(a.prog_in, a.tag, a.follow ? min(q, ncols) : ncols, sh, a.err);
            if (avail >= ncols) avail = 0x7fffffff;
        }
    };
    ensure(kLookA);
#pragma unroll 1
    for (int q = 0; q < kLookA; q += kU) {
        stage(q, q / kU, std::false_type{});
        // let the previous strip get kAheadA columns ahead before the first pairs
        if (q == 0 && consumer && lane0) wait_pair(a.h_in + 2 * (size_t)min(kAheadA, ncols - 1) + 1, a.tag, sh, a.err);
        __syncwarp();
        if (q < kPairLookA) stage_pairs(q, std::false_type{});
        cp_commit();
    }

    // running destinations: the term v of forward tape step ncols+30-s, the
    // columns written back by a block (march s0-kU-31 for its first), the pair of march s-31
    float* pV = a.tc2 + (long long)(ncols + 30) * 32 + flane;
    float* pW = a.lam + first - (31 + kU) * dL;
    unsigned long long* pH = a.h_out - 2 * 31;

    float my_x = 0.0f, my_pe = 0.0f, my_pev = 0.0f, pev_hold = 0.0f;
    int tb0 = 0, tf0 = kLookA / kU;  // ring slots of the block's tape rows and of those staged next
    int next_pub = a.publish ? a.publish : -1;  // the block that publishes the progress next
    unsigned ro = ((kRingA - lane) % kRingA) * 32;  // ring offset of the lane's march s0 - lane
    float* const Lr = R.L + tix;

    // Blocks of kU steps, as in the forward: one wait per block, the block's
    // ring reads, its kU linear updates (the only serial chain), its stores.
    auto block = [&](int s0, auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        cp_wait<(kLookA < kPairLookA ? kLookA : kPairLookA) / kU - 1>();
        __syncwarp();

        const AdjTape& t = R.tape[tb0];
        unsigned off[kU];
        int br[kU];
        float lam_in[kU], c2[kU], av[kU], ae[kU], aev[kU], hx[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) {
            off[u] = ro;
            ro = ring_next<32, kRingA * 32>(ro);
            lam_in[u] = Lr[off[u]];
            const int e = (kU - 1 - u) * 32 + flane;
            const float c = t.c1[e], cm = fsub(1.0f, c);
            c2[u] = t.c2[e];
            // dT/d{tv, te, tev} of the candidate: (1,0,0), (0,1,0), (c,-c,1), (0,1-c,c), (1-c,0,c);
            // c is zero for the first two, so 1 goes with 5 and 2 with 4; the zeros are selected below
            br[u] = t.code[e] & 7;
            const bool two = br[u] == 3;
            av[u] = two ? c : cm;
            ae[u] = two ? -c : cm;
            aev[u] = two ? 1.0f : c;
        }
        // write back the columns every lane had finished before this block (marches s0-kU-31 ..)
        {
            const int m = s0 + vu - kU - 31;
            if (FAST || (m >= 0 && m < ncols))
                *reinterpret_cast<float4*>(pW) = *reinterpret_cast<const float4*>(&R.L[wo + vc]);
            wo = ring_next<kU * 32, kRingA * 32>(wo);
            pW += kU * dL;
        }
        {
            // the upwind row of lane 0: the previous strip's pairs, or nothing
            // (every lane reads them, lane 0 uses them)
            uint4 e[kU];
            unsigned stale = 0;
#pragma unroll
            for (int u = 0; u < kU; u++) {
                e[u] = R.pair[pi + u];
                if (FAST || s0 + u < ncols) stale |= (e[u].y ^ a.tag) | (e[u].w ^ a.tag);
            }
            pi = (pi + kU) % kPairsA;
            // the rare cases of a block behind one branch
            if ((consumer && stale != 0) || s0 + kLookA + kU > avail || s0 == next_pub) {
                if (consumer && stale != 0) {
                    // pairs the previous strip had not written when they were prefetched:
                    // wait for them, then fall kAheadA columns behind so later prefetches hit
                    if (lane0) {
#pragma unroll
                        for (int u = 0; u < kU; u++)
                            if (FAST || s0 + u < ncols) {
                                e[u].x = __float_as_uint(wait_pair(a.h_in + 2 * (size_t)(s0 + u), a.tag, sh, a.err));
                                e[u].z = __float_as_uint(wait_pair(a.h_in + 2 * (size_t)(s0 + u) + 1, a.tag, sh, a.err));
                            }
                        wait_pair(a.h_in + 2 * (size_t)min(s0 + kU - 1 + kAheadA, ncols - 1) + 1, a.tag, sh, a.err);
                    }
                    __syncwarp();
                }
                ensure(s0 + kLookA + kU);
                if (s0 == next_pub) {
                    publish_progress(a.prog_out, a.tag, min(s0 - 31, ncols));
                    next_pub += a.publish;
                }
            }
#pragma unroll
            for (int u = 0; u < kU; u++) {
                hx[u] = fadd(__uint_as_float(e[u].x), pev_hold);
                pev_hold = __uint_as_float(e[u].z);
            }
        }

        // next columns, tape rows and pairs (the ring reads above are in flight meanwhile)
        {
            stage(s0 + kLookA, tf0, fast_tag);
            if (++tf0 >= kTapeBlocks) tf0 = 0;
            stage_pairs(s0 + kPairLookA, fast_tag);
            cp_commit();
        }

        float lo[kU], vv[kU], opv[kU], opev[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) {
            const int m = s0 + u - lane;
            // pv of the upwind row's node in this column plus pev of its node in
            // the previous column, summed by the lane above
            const float x_up = __shfl_up_sync(0xffffffffu, my_x, 1);
            float mu = fadd(fadd(lam_in[u], lane0 ? hx[u] : x_up), my_pe);
            if (!FAST && !(vrow && (m >= 0) && (m < ncols))) mu = 0.0f;
            lo[u] = br[u] ? 0.0f : mu;
            vv[u] = fmul(mu, c2[u]);
            opv[u] = (br[u] & 1) ? fmul(mu, av[u]) : 0.0f;
            opev[u] = (br[u] >= 3) ? fmul(mu, aev[u]) : 0.0f;
            my_x = fadd(opv[u], my_pev);  // this node's pv + the previous node's pev
            my_pe = ((unsigned)(br[u] - 2) < 3u) ? fmul(mu, ae[u]) : 0.0f;
            my_pev = opev[u];
        }

#pragma unroll
        for (int u = 0; u < kU; u++) {
            const int m = s0 + u - lane;
            if (FAST ? vrow : (vrow && (m >= 0) && (m < ncols))) {
                Lr[off[u]] = lo[u];
                pV[-32 * u] = vv[u];
                if (feeds)
                    st_pairs(pH + 2 * u, opv[u], opev[u], a.tag);
            }
        }
        // mark the block's tape entries if a term is not zero (read by the gather)
        bool nz = false;
#pragma unroll
        for (int u = 0; u < kU; u++) nz |= vv[u] != 0.0f;
        if (__any_sync(0xffffffffu, nz) && lane < 2) {
            const int fs = ncols + 30 - s0 - (lane ? kU - 1 : 0);
            a.vflag[(a.tape_base + (size_t)max(fs, 0) * 32) >> 10] = 1;
        }
        pV -= 32 * kU;
        pH += 2 * kU;
        if (++tb0 >= kTapeBlocks) tb0 = 0;
    };
    // column blocks in the order the march finishes them: the counted sweep
    // is the reverse of sweep 0, which marches down the columns, so
    // block b is done once lane 31 has passed its first window column (the
    // tile's extra node column, the next block's first, came earlier)
    const int blo = a.c0 / kGT, bhi = (a.c0 + ncols - 1) / kGT;
    int next_b = bhi;
    auto count_done = [&](int s_end) {
        while (next_b >= blo) {
            const int wcol = max(next_b * kGT, a.c0) - a.c0;
            const int m = ncols - 1 - wcol;  // march of that column
            if (m + 31 > s_end) break;
            __threadfence();  // this lane's terms before the count
            __syncwarp();
            if (lane == 0) atomicAdd(a.ready + next_b, 1u);
            next_b--;
        }
    };
    // one block past the last step writes the last columns back
    [[maybe_unused]] const unsigned nfast = max(ncols + 1 - kLookA - kU - (31 + kU), 0);  // first steps of interior blocks: 31 + kU ..
#pragma unroll 1
    for (int s0 = 0; s0 < nsteps + kU; s0 += kU) {
        if constexpr (INTERIOR) {
            if ((unsigned)(s0 - (31 + kU)) < nfast)
                block(s0, std::true_type{});
            else
                block(s0, std::false_type{});
        } else {
            block(s0, std::false_type{});
        }
        if (a.ready) count_done(s0 + kU - 1);
    }
    if (a.prog_out) publish_progress(a.prog_out, a.tag, ncols);
    cp_wait<0>();
    __syncwarp();
}

// The reverse sweeps of every shot (persistent gangs, as the forward). f:
// inside a fused launch, count finished column blocks in the last reverse
// sweep and flag each shot's initialisation term.
template <bool INTERIOR>
__device__ void adjoint_body(const AdjParams& p, const FuseParams* f)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CtaShared* cs = reinterpret_cast<CtaShared*>(smem_raw);
    AdjRing* rings = reinterpret_cast<AdjRing*>(smem_raw + ((sizeof(CtaShared) + 15) & ~size_t(15)));
    const int tid = threadIdx.x;
    const GangPos gp = gang_pos(p.G);
    const int nzz = p.nzz, nstrips = p.nstrips, ld = strip_pitch(nzz);
    float* lam = p.lam + (size_t)gp.gang * p.lam_per_gang;
    const size_t row = 2 * (size_t)hand_pitch(p.maxcols);
    unsigned long long* hb = p.hand + (size_t)gp.gang * hand_words(nstrips, p.maxcols, 2);
    unsigned long long* prog = hb + 4 * (size_t)nstrips * row;
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
        const int ncols = sh.ncols;
        const unsigned tag = (p.epoch << 10) | (unsigned)(it & 1023);
        // seed: adjoint of the final field from the pick gradients. The window
        // is zeroed by the whole gang, then each seeded node sums its
        // receivers' terms in receiver order (the order of a receiver-by-
        // receiver accumulation, hence the same bits).
        {
            const int gt = gp.g * blockDim.x + tid, gn = p.G * blockDim.x;
            const size_t nw = (size_t)ld * ncols;  // rows past the grid stay zero
#pragma unroll 4
            for (size_t q = gt; q < nw; q += gn) lam[q] = 0.0f;
            gang_barrier(bar, (++nbar) * p.G, cs, p.err);
            const float* pg = p.pick_grad + (size_t)sh.orig * p.nrec;
            for (int n = gt; n < p.nseed; n += gn) {
                const int col = p.seed_col[n] - sh.c0;
                if (col < 0 || col >= ncols) continue;
                float acc = 0.0f;
                bool any = false;
                for (int e = p.seed_ptr[n]; e < p.seed_ptr[n + 1]; e++) {
                    const int rr = p.seed_rec[e];
                    const int jl = p.rec_jg[rr] - sh.c0;
                    const float g = pg[rr];
                    if (jl - 1 < 1 || jl + 2 > ncols - 2 || !(g == g)) continue;
                    acc = fadd(acc, fmul(g, p.seed_w[e]));
                    any = true;
                }
                if (any) lam[(size_t)p.seed_row[n] + (size_t)col * ld] = acc;
            }
        }
        gang_barrier(bar, (++nbar) * p.G, cs, p.err);
        // reverse sweeps 3, 2, 1, 0 as one list of strip tasks dealt to the
        // warps in turn (see solve_window): 3 and 2 march to the right, 1 and 0
        // to the left; 3 and 1 take the strips top to bottom, 2 and 0 upwards
        AdjStripArgs a;
        a.lam = lam;
        a.nzz = nzz;
        a.ncols = ncols;
        a.ring = rings + gp.warp;
        a.sh = cs;
        a.err = p.err;
        a.tag = tag;
        a.c0 = sh.c0;
        a.vflag = p.vflag;
#pragma unroll 1
        for (int task = gp.slot; task < 4 * nstrips; task += gp.slots) {
            const int rs = task / nstrips, pidx = task - rs * nstrips, sw = 3 - rs;
            a.k = (rs & 1) ? nstrips - 1 - pidx : pidx;
            a.down = !(rs & 1);
            a.right = rs < 2;
            unsigned long long* hs = hb + ((size_t)rs * nstrips + pidx) * row;
            a.h_in = (pidx > 0) ? hs : nullptr;
            a.h_out = (pidx < nstrips - 1) ? hs + row : nullptr;
            a.prog_in = (rs > 0) ? prog + (size_t)(rs - 1) * nstrips + a.k : nullptr;
            a.follow = rs & 1;
            a.prog_out = (rs < 3) ? prog + (size_t)rs * nstrips + a.k : nullptr;
            a.publish = (rs & 1) ? 0 : publish_every(nstrips - 1 - pidx);
            const size_t tb = tape_strip_base(sh.tape_off, sw, a.k, nstrips, ncols);
            a.tcode = p.tcode + tb;
            a.tc1 = p.tc1 + tb;
            a.tc2 = p.tc2 + tb;
            a.tape_base = tb;
            a.ready = (f && sw == 0) ? f->ready + (size_t)a.k * f->nblk : nullptr;
            adj_strip<INTERIOR>(a);
        }
        gang_barrier(bar, (++nbar) * p.G, cs, p.err);
        if (gp.g == 0 && tid < 9) {
            const int aa = tid % 3, bb = tid / 3;
            const int zi = sh.sIdz + aa - 1, xl = sh.sIdx - sh.c0 + bb - 1;
            p.lam_init[(size_t)sh.orig * 9 + tid] = lam[(size_t)zi + (size_t)xl * ld];
        }
        if (f && gp.g == 0) {
            __threadfence();
            __syncthreads();
            if (tid == 0) st_release_gpu(f->shot_done + sh.orig, f->done_tag);
        }
        b = next_shot(p.bar, p.NG, p.G, gp.gang, gp.g, it, nbar, cs, p.err);
    }
}

// (kMaxWarps * 32, 1): the block size alone as the bound caps the kernel at
// 64 registers and spills the strip loop's state.
template <bool INTERIOR>
__global__ void __launch_bounds__(kMaxWarps * 32, 1) k_adjoint(AdjParams p)
{
    adjoint_body<INTERIOR>(p, nullptr);
}

// g(a, b) = sum over shots (caller order, FP64) of the shot's FP32 sum over
// sweeps 0..3 and corners (dr, dc) = (0,0),(0,1),(1,0),(1,1) of the matching
// node terms, plus the 3x3 initialisation term lam_init * dist.
//
// One CTA per tile of 32 rows (one strip) x kGT columns. The terms of node
// (i, j) in a sweep sit in the tape in the forward strip's skewed step order,
// so the nodes a tile reads (its rows and the first row of the next strip,
// its columns and one more) are, per shot and sweep, one contiguous run of
// kGT + 32 tape steps of the strip plus kGT + 1 entries of the next strip.
// These runs stream through kGStages shared-memory stages (cp.async) while
// the threads sum their cells' terms in the order above. The shots covering
// the tile's columns come from a per-column-block list built on the host,
// staged in shared memory kGChunk at a time. Runs without a nonzero term (the
// rays of a shot pass through a part of its window only) are left out: the
// reverse sweeps mark every 1024 tape entries that hold one (vflag). A shot
// without a term is then not summed at all, unless a factor of its zero is not
// finite (undef).
constexpr int kGSteps = kGT + 32;   // tape steps a tile's strip spans per sweep
constexpr int kGStages = 3;
constexpr int kGChunk = 128;

struct __align__(16) GatherStage {
    float v[kGSteps * 32];
    uint32_t code[kGSteps * 8];      // code bytes
    float v2[kGT + 1];               // next strip, first row
    uint32_t code2[kGT + 1];         // the aligned words holding its code bytes
};

struct GatherSmem {
    GatherStage stg[kGStages];
    GatherShot shots[kGChunk];
    uint16_t list[4 * kGChunk];      // runs to sum: shot of the chunk * 4 + sweep
    int wcount[kMaxWarps];
};

// One run's node terms for the thread's NQ cells: row a = rb + lane, NQ
// consecutive columns from window column bl0. A node column is read once (its
// rows a and a+1) and serves the cells on both its sides: corner (dr, dc) of
// cell (a, b) is node (a + 1 - dr, b + 1 - dc). A kept node's code has bit 5
// set and matches no corner. EDGE: node columns outside the window have no terms.
template <int NQ, bool EDGE>
__device__ __forceinline__ void gather_run(const GatherStage& S, float* g, int bl0, int ncols, int fmlo, bool szpos,
                                           bool sxpos, bool next_strip)
{
    const int lane = threadIdx.x & 31;
    const bool last = lane == 31;   // its node row a+1 is the next strip's first
    const int dir = sxpos ? 1 : -1;
    const int fm0 = (sxpos ? bl0 : ncols - 1 - bl0) - fmlo;
    const int fl0 = szpos ? lane : 31 - lane, fl1 = szpos ? lane + 1 : 30 - lane;
    const uint8_t* cb = reinterpret_cast<const uint8_t*>(S.code);
    const uint8_t* cb2 = reinterpret_cast<const uint8_t*>(S.code2);
    const float* pv0 = S.v + ((fm0 + fl0) * 32 + fl0);
    const uint8_t* pc0 = cb + ((fm0 + fl0) * 32 + fl0);
    const float* pv1 = last ? S.v2 + fm0 : S.v + ((fm0 + fl1) * 32 + fl1);
    const uint8_t* pc1 = last ? cb2 + (4 * fm0 + (szpos ? 0 : 3)) : cb + ((fm0 + fl1) * 32 + fl1);
    const int s0 = 32 * dir, sv1 = last ? dir : s0, sc1 = last ? 4 * dir : s0;
    const bool has1 = !last || next_strip;
    float v0p = 0.0f, v1p = 0.0f;
    int c0p = 0x20, c1p = 0x20;
#pragma unroll
    for (int q = 0; q <= NQ; q++) {
        const bool in = !EDGE || (bl0 + q >= 0 && bl0 + q < ncols);
        float v0 = 0.0f, v1 = 0.0f;
        int c0 = 0x20, c1 = 0x20;
        if (in) {
            v0 = pv0[q * s0];
            c0 = pc0[q * s0] & 0x38;
            if (has1) {
                v1 = pv1[q * sv1];
                c1 = pc1[q * sc1] & 0x38;
            }
        }
        if (q > 0) {
            float& x = g[q - 1];
            if (c1 == 0x00) x = fadd(x, v1);
            if (c1p == 0x10) x = fadd(x, v1p);
            if (c0 == 0x08) x = fadd(x, v0);
            if (c0p == 0x18) x = fadd(x, v0p);
        }
        v0p = v0;
        v1p = v1;
        c0p = c0;
        c1p = c1;
    }
}

// Bounded wait of one thread until *p >= target (acquire); false after the
// limit, with the error flag set.
__device__ __forceinline__ bool wait_count(const unsigned* p, unsigned target, int* err, unsigned long long wait_ns)
{
    if (ld_acquire_gpu(p) >= target) return true;
    const unsigned long long t0 = global_ns();
    const unsigned long long lim = wait_ns ? wait_ns : kSpinNs;
    long long n = 0;
    while (ld_acquire_gpu(p) < target) {
        if (*(volatile int*)err) return false;
        __nanosleep(256);
        if (++n > kSpinLimit || ((n & 255) == 0 && global_ns() - t0 > lim)) {
            atomicExch(err, 2);
            return false;
        }
    }
    return true;
}

// g(a, b) of one tile (strip k, column block cb) by 32 W threads: thread
// (warp w, lane l) owns the 32 / W cells (32 k + l, 32 cb + w 32/W ..).
// VTI: the batch was anisotropic; each shot's summed terms (its gradient with
// respect to its own qP slowness) are multiplied by the shot's derivative
// factors of the qP slowness before the FP64 sum over shots, giving dJ/dS,
// dJ/dC11 and dJ/dC13. FUSED: the tile runs inside the reverse-sweep launch
// while other shots may still be writing terms; it reads the tape through L2
// only (cp.async.cg, ld.global.cg) and waits for a shot's flag before using
// its initialisation term. Returns false when a wait gave up.
template <int W, bool VTI, bool FUSED>
__device__ bool gather_tile(const GatherParams& p, GatherSmem& sm, int k, int cb)
{
    constexpr int NQ = 32 / W;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = cb * kGT;
    const int rb = 32 * k;
    const bool next_strip = k + 1 < p.nstrips;
    const int a = rb + lane, cw = c + warp * NQ;  // the thread's cells: row a, columns cw ..

    // node-column range of run (shot t, sweep sw) in march order
    auto fm_range = [&](const GatherShot& t, int sw, int& fmlo, int& fmhi) {
        const int jlo = max(c - t.c0, 0);
        const int jhi = min(c + kGT - t.c0, t.ncols - 1);   // covered cells' columns and one more
        fmlo = (sw < 2) ? jlo : t.ncols - 1 - jhi;
        fmhi = (sw < 2) ? jhi : t.ncols - 1 - jlo;
    };
    // the tile holds cells of the shot's 3x3 initialisation
    auto has_source = [&](const GatherShot& t) {
        return t.sIdz + 1 >= rb && t.sIdz - 1 < rb + 32 && t.sIdx + 1 >= c && t.sIdx - 1 < c + kGT;
    };
    auto marked = [&](size_t lo, size_t hi) {  // a nonzero term among tape entries lo .. hi
        unsigned any = 0;
        for (size_t q = lo >> 10; q <= hi >> 10; q++) any |= __ldcg(p.vflag + q);
        return any != 0;
    };
    // the sum of a shot that may be left out: 0, or none (NaN) as zero times a
    // factor that is not finite is NaN
    const float skip = VTI && *p.undef != 0 ? __int_as_float(0x7fc00000) : 0.0f;
    auto wanted = [&](const GatherShot& t, int sw) {
        if (sw == 3 && ((VTI && skip != skip) || has_source(t))) return true;
        int fmlo, fmhi;
        fm_range(t, sw, fmlo, fmhi);
        const size_t base = tape_strip_base(t.tape_off, sw, k, p.nstrips, t.ncols);
        if (marked(base + (size_t)fmlo * 32, base + (size_t)(fmhi + 31) * 32 + 31)) return true;
        const int fl2 = (sw == 1 || sw == 3) ? 31 : 0;
        const size_t base2 = base + (size_t)(t.ncols + 31) * 32;
        return next_strip && marked(base2 + (size_t)(fmlo + fl2) * 32, base2 + (size_t)(fmhi + fl2) * 32 + 31);
    };
    auto issue = [&](int x, GatherStage& S) {
        const GatherShot& t = sm.shots[x >> 2];
        const int sw = x & 3;
        int fmlo, fmhi;
        fm_range(t, sw, fmlo, fmhi);
        const int nst = t.ncols + 31;
        const size_t base = tape_strip_base(t.tape_off, sw, k, p.nstrips, t.ncols);
        for (int q = tid; q < kGSteps * 8; q += 32 * W) {
            const int st = fmlo + (q >> 3);
            if (st < nst) cp_async16_cg(&S.v[q * 4], p.vrec + base + (size_t)st * 32 + (q & 7) * 4);
        }
        for (int q = tid; q < kGSteps * 2; q += 32 * W) {
            const int st = fmlo + (q >> 1);
            if (st < nst) cp_async16_cg(&S.code[q * 4], p.tcode + base + (size_t)st * 32 + (q & 1) * 16);
        }
        if (next_strip) {
            const size_t base2 = base + (size_t)nst * 32;
            const int fl2 = (sw == 1 || sw == 3) ? 31 : 0;
            for (int q = tid; q <= fmhi - fmlo; q += 32 * W) {
                const size_t e = base2 + (size_t)(fmlo + q + fl2) * 32 + fl2;
                if (FUSED) {
                    S.v2[q] = __ldcg(p.vrec + e);
                } else {
                    cp_async4(&S.v2[q], p.vrec + e);
                }
                cp_async4(&S.code2[q], p.tcode + (e & ~(size_t)3));
            }
        }
        cp_commit();
    };

    double total[NQ], t11[VTI ? NQ : 1], t13[VTI ? NQ : 1];
    float g[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        total[q] = 0.0;
        g[q] = 0.0f;
        if (VTI) t11[q] = t13[q] = 0.0;
    }
    bool ok = true;
    // a shot's sum is complete: its initialisation term, then the sum over shots
    auto close_shot = [&](const GatherShot& t) {
        const bool src = has_source(t);
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const int bc = cw + q, bl = bc - t.c0;
            if (src) {
                const int da = a - t.sIdz + 1, db = bc - t.sIdx + 1;
                if (da >= 0 && da < 3 && db >= 0 && db < 3) {
                    const double d = src_dist(a, bc, p.nb, p.dx, p.dz, t.sx, t.sz);
                    const float* li = p.lam_init + (size_t)t.orig * 9 + da + 3 * db;
                    g[q] = fadd(g[q], fmul(FUSED ? __ldcg(li) : *li, __double2float_rn(d)));
                }
            }
            if (g[q] != (VTI ? skip : 0.0f) && a < p.nzz && bc < p.nxx && bl >= 0 && bl < t.ncols) {
                if (VTI) {
                    const float* f = p.vfac + t.q_off + (size_t)a + (size_t)bl * strip_pitch(p.nzz);
                    total[q] += (double)g[q] * (double)f[0];
                    t11[q] += (double)g[q] * (double)f[p.vfac_total];
                    t13[q] += (double)g[q] * (double)f[2 * p.vfac_total];
                } else {
                    total[q] += (double)g[q];
                }
            }
            g[q] = 0.0f;
        }
    };
    const int e_end = p.blk_ptr[cb + 1];
#pragma unroll 1
    for (int e0 = p.blk_ptr[cb]; e0 < e_end; e0 += kGChunk) {
        const int n = min(kGChunk, e_end - e0);
        __syncthreads();  // the previous chunk's list and stages are no longer read
        for (int q = tid; q < n; q += 32 * W) sm.shots[q] = p.blk_shots[e0 + q];
        __syncthreads();
        // the chunk's runs with terms, in order
        int nrun = 0;
#pragma unroll 1
        for (int x0 = 0; x0 < 4 * n; x0 += 32 * W) {
            const int x = x0 + tid;
            const bool keep = x < 4 * n && wanted(sm.shots[x >> 2], x & 3);
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) sm.wcount[warp] = __popc(m);
            __syncthreads();
            int before = nrun;
#pragma unroll
            for (int w = 0; w < W; w++) {
                before += (w < warp) ? sm.wcount[w] : 0;
                nrun += sm.wcount[w];
            }
            if (keep) sm.list[before + __popc(m & ((1u << lane) - 1))] = (uint16_t)x;
            __syncthreads();
        }
        for (int i = 0; i < kGStages - 1 && i < nrun; i++) issue(sm.list[i], sm.stg[i]);
#pragma unroll 1
        for (int i = 0; i < nrun; i++) {
            const int ahead = min(kGStages - 1, nrun - 1 - i);  // stages issued after stage i
            if (i + kGStages - 1 < nrun) {
                const int j = i + kGStages - 1;
                issue(sm.list[j], sm.stg[j % kGStages]);
                cp_wait<kGStages - 1>();
            } else if (ahead == 1) {
                cp_wait<1>();
            } else {
                cp_wait<0>();
            }
            const int x = sm.list[i];
            const GatherShot& t = sm.shots[x >> 2];
            const int sw = x & 3;
            if (FUSED && sw == 3 && tid == 0) {
                // the shot's initialisation term is written when its reverse sweeps end
                if (has_source(t) && !wait_count(p.shot_done + t.orig, p.done_tag, p.err, p.wait_ns)) ok = false;
            }
            __syncthreads();
            int fmlo, fmhi;
            fm_range(t, sw, fmlo, fmhi);
            const bool szpos = !(sw & 1), sxpos = sw < 2;
            const int bl0 = cw - t.c0;
            if (c >= t.c0 && c + kGT - t.c0 <= t.ncols - 1)
                gather_run<NQ, false>(sm.stg[i % kGStages], g, bl0, t.ncols, fmlo, szpos, sxpos, next_strip);
            else
                gather_run<NQ, true>(sm.stg[i % kGStages], g, bl0, t.ncols, fmlo, szpos, sxpos, next_strip);
            if (i + 1 == nrun || (sm.list[i + 1] >> 2) != (x >> 2)) close_shot(t);
            __syncthreads();  // stage i's buffer is refilled by stage i + kGStages
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        const int bc = cw + q;
        if (a < p.nzz && bc < p.nxx) {
            p.grad[(size_t)a + (size_t)bc * p.nzz] = __double2float_rn(total[q]);
            if (VTI) {
                p.grad_c11[(size_t)a + (size_t)bc * p.nzz] = __double2float_rn(t11[q]);
                p.grad_c13[(size_t)a + (size_t)bc * p.nzz] = __double2float_rn(t13[q]);
            }
        }
    }
    return ok;
}

// The gather as its own launch: one CTA of 8 warps per tile.
template <bool VTI>
__global__ void __launch_bounds__(256) k_gather(GatherParams p)
{
    extern __shared__ __align__(16) unsigned char gsm_raw[];
    GatherSmem& sm = *reinterpret_cast<GatherSmem*>(gsm_raw);
    const int ntx = (p.nxx + kGT - 1) / kGT;
    gather_tile<8, VTI, false>(p, sm, blockIdx.x / ntx, blockIdx.x % ntx);
}

// Residuals r = pick - t_obs (NaN picks or observations contribute nothing)
// and the misfit 1/2 sum r^2 in FP64 in a fixed order: 1024 sums, the t-th of
// elements t, t + 1024, ..., then a tree over them. Bound by the FP64 pipe
// (r^2 is exact there, so one multiply-add per element, and the half waits
// for the end) and the latency of each sum's chain, so the sums are spread
// over the 8 CTAs of one cluster, which leave them in the first CTA's shared
// memory; one CTA of 1024 threads took 0.70 ms for 801000 picks, the cluster
// takes 0.18 ms.
constexpr int kResCtas = 8, kResThreads = 1024 / kResCtas, kResUnroll = 8;
__global__ void __cluster_dims__(kResCtas, 1, 1) __launch_bounds__(kResThreads)
    k_residual(const float* picks, const float* tobs, size_t n, float* res, double* misfit)
{
    __shared__ double part[1024];
    const unsigned t = blockIdx.x * kResThreads + threadIdx.x;
    double acc = 0.0;
    for (size_t k0 = t; k0 < n; k0 += 1024 * kResUnroll) {
        float pk[kResUnroll], ob[kResUnroll];
#pragma unroll
        for (int u = 0; u < kResUnroll; u++) {
            const size_t k = k0 + 1024 * u;
            pk[u] = k < n ? picks[k] : 0.0f;
            ob[u] = k < n ? tobs[k] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kResUnroll; u++) {
            const size_t k = k0 + 1024 * u;
            if (k >= n) break;
            float r = fsub(pk[u], ob[u]);
            if (!(r == r)) r = __int_as_float(0x7fc00000);
            res[k] = r;
            if (r == r) acc = fma((double)r, (double)r, acc);
        }
    }
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    cl.sync();  // the first CTA has started before its memory is written
    cl.map_shared_rank(part, 0)[t] = acc;
    cl.sync();
    if (cl.block_rank() != 0) return;
    for (int s = 512; s > 0; s >>= 1) {
        for (int k = threadIdx.x; k < s; k += kResThreads) part[k] += part[k + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *misfit = 0.5 * part[0];
}

}  // namespace sf

namespace sf {

// Reverse sweeps and gather in one launch of 32 W-thread CTAs (see
// FuseParams). Every CTA of the launch is resident at once (the host sizes
// the grid to the device), the reverse sweeps never wait on the gather, and
// every gather wait is bounded.
template <bool INTERIOR, int W>
__global__ void __launch_bounds__(kMaxWarps * 32, 1) k_adjoint_gather(AdjParams p, GatherParams g, FuseParams f)
{
    if ((int)blockIdx.x < f.nadj) {
        adjoint_body<INTERIOR>(p, &f);
        return;
    }
    extern __shared__ __align__(16) unsigned char fsm_raw[];
    GatherSmem& sm = *reinterpret_cast<GatherSmem*>(fsm_raw);
    __shared__ int tile_s, ok_s;
    const int ntiles = p.nstrips * f.nblk;
#pragma unroll 1
    while (true) {
        if (threadIdx.x == 0) {
            const int t = (int)atomicAdd(f.tile_ctr, 1u);
            int ok = 1;
            if (t < ntiles) {
                // bottom strips first, columns right to left: the order the last
                // reverse sweep finishes them
                const int k = p.nstrips - 1 - t / f.nblk, cb = f.nblk - 1 - t % f.nblk;
                const unsigned cover = (unsigned)(g.blk_ptr[cb + 1] - g.blk_ptr[cb]);
                ok = wait_count(f.ready + (size_t)k * f.nblk + cb, cover, g.err, g.wait_ns);
                if (ok && k + 1 < p.nstrips) ok = wait_count(f.ready + (size_t)(k + 1) * f.nblk + cb, cover, g.err, g.wait_ns);
            }
            tile_s = t;
            ok_s = ok;
        }
        __syncthreads();
        const int t = tile_s, ok = ok_s;
        __syncthreads();
        if (t >= ntiles || !ok) break;
        if (!gather_tile<W, false, true>(g, sm, p.nstrips - 1 - t / f.nblk, f.nblk - 1 - t % f.nblk)) break;
    }
}

}  // namespace sf
