// Strip-systolic fast sweeping (GB300, sm_103a).
//
// A shot window of nzz rows x ncols columns is cut into 32-row strips; a warp
// sweeps a strip with lane l owning one row and marching across the columns,
// lane l running l steps behind lane 0. At step s lane l updates node (row(l),
// column of march index s-l), so the three upwind values of the reference
// update (modeling.cu:324-326) are: the lane above's result of the previous
// step (shfl), the lane's own previous result, and the lane's own previous
// upwind value. Consecutive strips (usually on other SMs) are chained through
// global memory without fences: the last lane of strip p writes each value of
// its row together with a tag (launch epoch and shot number) as one 64-bit
// store (two pairs in one 16-byte store in the compensated arithmetic); strip
// p+1 prefetches the pairs (through L2 only, so that a line of which the
// producer had written a part is never found again in L1) and checks the tags. A stale pair (the producer has not got there yet) sends
// lane 0 into a bounded spin on the pair itself, after which it waits until
// the producer is some columns further on, so later prefetches find their
// data. Producers never wait on consumers, so every wait points to an earlier
// strip and the schedule cannot deadlock however strips are spread over warps
// and CTAs.
//
// The two sweeps of a march direction overlap: the upward sweep's first strip
// starts once the downward sweep's last strip is under way (solve_window). A
// strip's traveltimes then pass from one warp to another, so the earlier
// sweep's strip publishes how many columns it has written back (a fence and
// a tagged counter, every 32 to 256 columns) and the later one stays behind it.
//
// Columns are staged into a per-warp shared-memory ring by cp.async, a few
// march columns ahead, and lane l reads its own row of column s-l from the
// ring. A ring slot holds one column: slowness rows rb-1..rb+31 at 3..35,
// traveltimes at 36..67 and, in the compensated arithmetic, their lo parts at
// 68..99; one address serves all fields of a node, and with odd differences
// of pitch and row stride the skewed reads are (but for the lanes past the
// ring's end) bank-conflict free. The solver's own slowness and traveltime
// windows have a column stride of whole strips (VEC), so a strip's column is
// one aligned 128-byte line and the four columns of a block are one 16-byte
// copy per lane and field; finished columns go back the same way, one
// 16-byte load and store per lane. (Columns at the caller's stride, every one
// at another alignment, took a 4-byte copy per lane and column, two lines per
// column and L1 to merge them.) The march runs in blocks of a few steps: one wait for the
// staged columns per block, the block's ring reads, its node updates
// (the only serial chain), then its stores.
//
// Any order of node updates that respects the sweep's dependency DAG gives the
// same bits as the reference's anti-diagonal launches, so this schedule is a
// bit-exact replacement of eikonal_solver (modeling.cu:123-159).
#pragma once
#include <type_traits>

#include "sf_device.cuh"

namespace sf {

// Block size U, staging leads (march columns, multiples of the block) of the
// columns (LOOK) and of the upwind strip's pairs (PLOOK), and ring length of
// the forward strip loop. After a stall a consumer lets its producer get AHEAD
// columns ahead. The ring holds the 32 marches the lanes work on, the block
// still to be written back, the lead and a block. Blocks of four steps with
// eight columns staged ahead measured best: blocks of two (lead four) took
// 15% longer for the plain solve and 14% for the taped one (100 shots of
// 1707 x 357: 1.82 and 3.21 ms), a lead of four 25%, pairs eight ahead 3% (they
// lengthen the lag between strips).
template <bool COMP>
struct FwdBlock {
    static constexpr int U = 4;
    static constexpr int LOOK = 8;
    static constexpr int PLOOK = 4;
    static constexpr int AHEAD = PLOOK + U;
    static constexpr int RING = 47;
    static constexpr int SLOT = COMP ? 100 : 68;  // floats per slot
    static constexpr int PAIRS = 8;               // columns of the pair ring
    static_assert(LOOK % U == 0 && PLOOK % U == 0 && PLOOK <= LOOK && RING >= 31 + LOOK + 2 * U, "ring too small");
    static_assert(PAIRS % U == 0 && PAIRS >= PLOOK + U && U % 2 == 0, "pair ring too small");
    static_assert(SLOT % 4 == 0, "16-byte copies");
    static_assert(U == 4, "a block's columns are one 16-byte copy per lane");
};
constexpr int kS0 = 3, kT0 = 36, kL0 = 68;  // slowness rows rb-1.., traveltimes, their lo parts in a slot
// Columns between two publications of the progress of a sweep's strip with
// `after` strips behind it in the sweep. The fence waits for all of the
// warp's stores (7% of the reverse sweeps' stalls at 32 columns everywhere),
// and only the last strip's reader, the next sweep's first strip, follows at
// once; each strip before it has two more lags of over 40 columns in hand.
// Against 32 everywhere: reverse sweeps of 100 shots of 1701 x 351 cells 1.415 ->
// 1.36 ms, of 1000 windows of about 1000 x 1001 14.7 -> 14.3 ms, a lone shot
// of 201 x 101 279 -> 270 us.
__device__ __forceinline__ int publish_every(int after) { return 32 << min(after, 3); }
constexpr int kMaxWarps = 16;
// compensated kernels keep a second traveltime ring (the lo parts): at most
// 8 warps per CTA fit in shared memory
constexpr int kMaxWarpsComp = 8;
// the taped interior-block forward kernels have up to 168 registers a thread
// (k_shots), of which an SM holds three warps per scheduler: CTAs of 8 warps
constexpr int kMaxWarpsTapedInterior = 8;
constexpr long long kSpinLimit = 1ll << 30;          // iterations
constexpr unsigned kPollNs = 100;                    // pause between two polls of a wait
constexpr unsigned long long kSpinNs = 2000000000ull;  // and at most ~2 s (default; sf_set_wait_limit)

// A warp's forward ring: RING column slots, then the pair ring (a tagged
// pair per column, two in the compensated arithmetic). Multiples of 16 bytes.
template <bool COMP>
constexpr size_t ring_bytes()
{
    using B = FwdBlock<COMP>;
    return sizeof(float) * (size_t)B::RING * B::SLOT + 8 * (size_t)B::PAIRS * (COMP ? 2 : 1);
}

// Column stride of the solver's own windows: whole strips.
__host__ __device__ constexpr int strip_pitch(int nzz) { return (nzz + 31) & ~31; }

// Columns a row of handoff pairs is padded to: whole 16-byte pairs of pairs
// past the last column.
__host__ __device__ constexpr int hand_pitch(int maxcols) { return (maxcols + 3) & ~1; }
// 64-bit words of one gang's handoff region: the pairs of four sweeps (hs
// per column), then one progress word per sweep and strip.
__host__ __device__ constexpr size_t hand_words(int nstrips, int maxcols, int hs)
{
    return 4 * (size_t)nstrips * ((size_t)hand_pitch(maxcols) * hs) + ((4 * (size_t)nstrips + 1) & ~(size_t)1);
}

// Per-CTA shared state (static part), followed by the CTA's warp rings in
// dynamic shared memory.
struct CtaShared {
    int abort_flag;
    int item;              // the gang's next shot
    unsigned long long wait_ns;  // time limit of every bounded wait of the CTA
    float init[9];
};

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem)
{
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16_cg(void* smem, const void* gmem)
{
    unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }
__device__ __forceinline__ void st_volatile(int* p, int v) { *(volatile int*)p = v; }
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned* p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_u64(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Two pairs {v, tag}, {w, tag} in one 16-byte store, each one 64-bit element of it.
__device__ __forceinline__ void st_pairs(unsigned long long* p, float v, float w, unsigned tag)
{
    asm volatile("{\n.reg .b64 a, b;\nmov.b64 a, {%1, %3};\nmov.b64 b, {%2, %3};\nst.global.v2.b64 [%0], {a, b};\n}\n" ::"l"(p),
                 "r"(__float_as_uint(v)), "r"(__float_as_uint(w)), "r"(tag)
                 : "memory");
}
__device__ __forceinline__ unsigned long long pack_tag(float v, unsigned tag)
{
    return ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(v);
}
__device__ __forceinline__ unsigned tag_of(unsigned long long e) { return (unsigned)(e >> 32); }
__device__ __forceinline__ float val_of(unsigned long long e) { return __uint_as_float((unsigned)e); }

// The ring offset STEP further on in a ring of END words (x < END, STEP <= END).
template <int STEP, int END>
__device__ __forceinline__ unsigned ring_next(unsigned x)
{
    x += STEP;
    return min(x, x - END);  // x - END wraps past 2^31 while x < END
}

// Everything one warp needs for one strip of one sweep.
struct StripArgs {
    const float* S;   // slowness of the window
    float* T;         // traveltimes of the window
    int ld;           // column stride of both: strip_pitch(nzz) (VEC), or nzz
    float* Tl;        // compensated: their lo parts, same layout
    int nzz, ncols;
    int k;            // strip index: rows [32k, 32k+32)
    bool right;       // columns to the right (sweeps 0 and 1)
    bool down;        // rows downward (sweeps 0 and 2)
    bool sw0;         // first sweep: every node starts at kBig but the source's 3x3 block
    int sIdz, sIdx;   // source node (window coordinates)
    int skip_i, skip_j;
    Consts kc;
    const float* init;  // 9 values in shared memory
    unsigned char* ring;  // this warp's ring (ring_bytes<COMP>())
    CtaShared* sh;
    const unsigned long long* h_in;  // {value, tag} of the upwind strip's row by march column (nullptr: first strip)
    unsigned long long* h_out;       // pairs this strip feeds to the next one (nullptr: last strip)
    unsigned tag;                    // tag of this shot's pairs
    unsigned tag_in;                 // tag a consumer waits for (= tag; 1, which no launch writes, to test the timeout path)
    // columns written back by the previous sweep of this strip (nullptr in
    // the first sweep): all of them before the march starts, or (follow) a
    // few more than the march has reached
    const unsigned long long* prog_in;
    bool follow;
    unsigned long long* prog_out;    // this strip's own count (nullptr: nobody reads it)
    int publish;                     // columns between publications (publish_every), 0: only at the end
    // tape (TAPE only): base of this sweep/strip, entries [step*32 + lane]
    uint8_t* tcode;
    float* tc1;
    float* tc2;
    int* err;
};

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// One round of a bounded wait: sleeps, and now and then looks whether the
// wait must end: the launch's error flag or the CTA's abort flag is up, or its
// own limit has run out, which raises both. Every later wait of the CTA (or of
// any CTA once the launch's flag is up) then ends at once, so the kernel always
// finishes (its results are void and the host reports SF_ERR_TIMEOUT). The
// flags are read every eighth round only: the polling of warps that wait for
// their turn was a third of all instructions of the reverse sweeps.
struct WaitRound {
    unsigned long long t0 = 0;
    long long n = 0;
    __device__ __forceinline__ bool give_up(CtaShared* sh, int* err)
    {
        if ((n & 7) == 0) {
            if (ld_volatile(&sh->abort_flag) || *(volatile int*)err) return true;
            const unsigned long long now = global_ns();
            if (n == 0) t0 = now;
            if (n > kSpinLimit || now - t0 > sh->wait_ns) {
                st_volatile(&sh->abort_flag, 1);
                atomicExch(err, 2);
                return true;
            }
        }
        n++;
        __nanosleep(kPollNs);
        return false;
    }
};

// Bounded wait until the pair at p carries `tag`; returns its value (0 when
// it gives up).
__device__ __forceinline__ float wait_pair(const unsigned long long* p, unsigned tag, CtaShared* sh, int* err)
{
    unsigned long long e = ld_relaxed_u64(p);
    WaitRound w;
    while (tag_of(e) != tag) {
        if (w.give_up(sh, err)) return 0.0f;
        e = ld_relaxed_u64(p);
    }
    return val_of(e);
}

// Bounded wait of the whole warp until the progress word at p carries `tag`
// and at least `need` columns (acquire, by lane 0); returns the columns seen
// (`need` when it gives up).
__device__ __forceinline__ int wait_progress(const unsigned long long* p, unsigned tag, int need, CtaShared* sh, int* err)
{
    int cols = need;
    if ((threadIdx.x & 31) == 0) {
        WaitRound w;
        while (true) {
            unsigned long long e;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(e) : "l"(p) : "memory");
            if (tag_of(e) == tag && (int)(unsigned)e >= need) {
                cols = (int)(unsigned)e;
                break;
            }
            if (w.give_up(sh, err)) break;
        }
    }
    cols = __shfl_sync(0xffffffffu, cols, 0);
    __syncwarp();  // orders the other lanes' copies after lane 0's acquire
    return cols;
}

// Publishes that this warp's strip has written `cols` columns back: every
// lane's stores, ordered by the warp barrier and lane 0's fence, before the word.
__device__ __forceinline__ void publish_progress(unsigned long long* p, unsigned tag, int cols)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)tag << 32) | (unsigned)cols)
                     : "memory");
    }
}

// Bounded wait until the counter at p reaches `target` (acquire).
__device__ __forceinline__ void wait_counter(const unsigned* p, unsigned target, CtaShared* sh, int* err)
{
    WaitRound w;
    while (ld_acquire_gpu(p) < target)
        if (w.give_up(sh, err)) return;
}

// INTERIOR: blocks whose marches all lie inside the window (and touch neither
// the source's 3x3 block nor a skipped cell) run a body without those tests
// (fewer instructions per step, more code); otherwise every block runs the
// general body. SQ: square cells (node_update). EXACT: IEEE division and
// roots on any operand (a slowness outside in_fast_range). All forms give
// the same bits. COMP: compensated arithmetic (node_update_comp): every
// traveltime the loop carries, stages, hands on and writes back is a pair
// (hi, lo); the second handoff pair of a column carries lo.
//
// DIR: the march's direction, right (1), left (-1) or a runtime value (0, one
// body for both, where FwdParams::drift is set). The row direction and the
// first sweep's start values are runtime values, so the two sweeps that run at the same time share
// their code: with a copy per sweep, loops of up to 14 KB were in flight on
// an SM and instruction fetch was 16% of the stalls. The node's cells need no
// more for it than a select: of the two slowness columns a lane holds, the
// carried one is the cell column on the upwind side (j1) in either direction,
// and the new one the other. Marches to the left read one column ahead.
// VEC: the windows' column stride is strip_pitch(nzz).
template <int DIR, bool TAPE, bool REF, bool INTERIOR, bool SQ, bool COMP, bool EXACT, bool VEC>
__device__ __forceinline__ void run_strip(const StripArgs& a)
{
    using B = FwdBlock<COMP>;
    constexpr int U = B::U, LOOK = B::LOOK, PLOOK = B::PLOOK, RING = B::RING, P = B::SLOT;
    constexpr int HS = COMP ? 2 : 1;         // handoff pairs per column
    const int lane = threadIdx.x & 31;
    const int nzz = a.nzz, ncols = a.ncols;
    const int rb = 32 * a.k;
    const bool right = DIR > 0 || (DIR == 0 && a.right), down = a.down, sw0 = DIR >= 0 && a.sw0;
    const int r = down ? rb + lane : rb + 31 - lane;
    const bool vrow = r < nzz;
    const bool irow = (r >= 1) && (r <= nzz - 2);
    const bool row1 = r == 1;
    const int tix = r - rb;    // the row's place among the strip's rows
    const int cz = down ? 0 : 8, cx = right ? 0 : 16;  // tape bits of the cell (i1, j1)
    const int dr2a = (r - 1 >= 1) ? 0 : 8;

    float* ring = reinterpret_cast<float*>(a.ring);
    float* pring = ring + RING * P;          // handoff pairs of march q at (q mod PAIRS) * 2 HS

    CtaShared* sh = a.sh;
    const bool consumer = a.h_in != nullptr;
    const bool lane0 = lane == 0;
    const bool feeds = (lane == 31) && (a.h_out != nullptr);
    // the strip holds rows of the source's 3x3 block (first sweep only)
    const bool src_rows = sw0 && (a.sIdz + 1 >= rb) && (a.sIdz - 1 <= rb + 31);
    auto col_of = [&](int m) { return right ? m : ncols - 1 - m; };
    // blocks whose first step lies in [g0, g0 + gn] need the general body for
    // the source block (first sweep) or a skipped cell
    int g0 = 0, gn = -1;
    if (src_rows) {
        const int ms = col_of(a.sIdx);  // its own inverse
        g0 = ms - 1;
        gn = 2;
    }
    if (a.skip_i >= rb && a.skip_i <= rb + 31) {
        const int ms = col_of(a.skip_j);
        const int lo = (gn < 0) ? ms : min(g0, ms), hi = (gn < 0) ? ms : max(g0 + gn, ms);
        g0 = lo;
        gn = hi - lo;
    }
    // from marches to a block's first step (none: a range no step reaches)
    g0 = (gn < 0) ? -(1 << 30) : g0 - (U - 1);
    gn = (gn < 0) ? 0 : gn + U - 1 + 31;

    // running source addresses of the next march columns to stage. VEC: lane
    // 8 u + c copies 16 bytes, rows rb+4c .. rb+4c+3, of the block's column u;
    // lanes 0..U-1 the row above of column `lane`. Else lane l copies row
    // rb-1+l (traveltimes rb+l) of every column, lanes 0..U-1 also row rb+31.
    const int vu = lane >> 3, vc = 4 * (lane & 7);
    const long long dT = (right ? 1 : -1) * (long long)a.ld;
    const long long c00 = (long long)col_of(0) * (long long)a.ld;
    const int ls_row = rb - 1 + lane;
    const bool ls_ok = VEC || ((ls_row >= 0) && (ls_row < nzz));
    const bool lt_ok = VEC || (rb + lane) < nzz;
    const bool lx_ok = (lane < U) && (VEC ? a.k > 0 : rb + 31 < nzz);
    const long long first = VEC ? c00 + vu * dT + rb + vc : c00 + rb + lane;
    const float* pS = a.S + (VEC ? first : first - 1);
    const float* pX = a.S + (c00 + lane * dT + (VEC ? rb - 1 : rb + 31));
    const float* pT = a.T + first;
    const float* pTl = COMP ? a.Tl + first : nullptr;
    // ring offsets of the slots these go to, and of the columns written back
    unsigned so = vu * P, xo = lane * P, wo = (RING - 31 - U + vu) * P;
    // columns q .. q+U-1 into the slots from `slot`
    // FAST: every march the call touches lies inside the window (no bounds tests)
    auto stage_cols = [&](int q, int slot, auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        auto wrap = [](int sl) { return sl >= RING ? sl - RING : sl; };
        if constexpr (VEC) {
            float* d = ring + so + vc;
            so = ring_next<U * P, RING * P>(so);
            const bool in = FAST || q + vu < ncols;
            if (in) cp_async16_cg(d + kS0 + 1, pS);
            if (sw0) {
                *reinterpret_cast<float4*>(d + kT0) = make_float4(kBig, kBig, kBig, kBig);
                if (COMP) *reinterpret_cast<float4*>(d + kL0) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            } else if (in) {
                cp_async16_cg(d + kT0, pT);
                if (COMP) cp_async16_cg(d + kL0, pTl);
            }
            pS += U * dT;
            pT += U * dT;
            if (COMP) pTl += U * dT;
        } else {
#pragma unroll
            for (int u = 0; u < U; u++) {
                float* d = ring + wrap(slot + u) * P + lane;
                const bool in = FAST || q + u < ncols;
                if (in && ls_ok) cp_async4(d + kS0, pS);
                if (sw0) {
                    d[kT0] = kBig;
                    if (COMP) d[kL0] = 0.0f;
                } else if (in && lt_ok) {
                    cp_async4(d + kT0, pT);
                    if (COMP) cp_async4(d + kL0, pTl);
                }
                pS += dT;
                pT += dT;
                if (COMP) pTl += dT;
            }
        }
        if (lx_ok && (FAST || q + lane < ncols)) cp_async4(ring + xo + (VEC ? kS0 : kS0 + 32), pX);
        xo = ring_next<U * P, RING * P>(xo);
        pX += U * dT;
    };
    // the upwind row's pairs of marches q .. q+U-1; the ring holds two blocks
    static_assert(B::PAIRS == 2 * U, "pair slots alternate");
    constexpr int kPairWords = U * 2 * HS;
    const bool pair_lane = consumer && lane < (COMP ? U : U / 2);  // 16-byte copies
    const unsigned long long* pP = a.h_in + 2 * lane;
    unsigned po = 4 * lane, pi = 0;  // ring offsets of the pairs staged and read
    auto stage_pairs = [&](int q, auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        if (pair_lane && (FAST || q + (COMP ? lane : 2 * lane) < ncols)) cp_async16_cg(pring + po, pP);
        pP += U * HS;
        po ^= kPairWords;
    };

    // columns of the previous sweep known to be written back
    int avail = sw0 ? 0x7fffffff : 0;
    auto ensure = [&](int q) {  // marches below q may be staged
        if (q > avail) {
            avail = wait_progress(a.prog_in, a.tag, a.follow ? min(q, ncols) : ncols, sh, a.err);
            if (avail >= ncols) avail = 0x7fffffff;
        }
    };

    // prologue: march columns 0 .. LOOK-1, pairs 0 .. PLOOK-1; the previous
    // strip gets AHEAD columns ahead before the first prefetches of its values
    ensure(LOOK);
#pragma unroll 1
    for (int q = 0; q < LOOK; q += U) {
        stage_cols(q, q, std::false_type{});
        if (q == 0 && consumer && lane0) wait_pair(a.h_in + HS * min(B::AHEAD, ncols - 1), a.tag_in, sh, a.err);
        __syncwarp();
        if (q < PLOOK) stage_pairs(q, std::false_type{});
        cp_commit();
    }

    // running destinations: the columns written back by a block (march s0-U-31
    // for its first), the next pair, the tape entry s*32+lane
    const long long wfirst = VEC ? first - (31 + U) * dT : c00 + r - (31 + U) * dT;
    float* pW = a.T + wfirst;
    float* pWl = COMP ? a.Tl + wfirst : nullptr;
    unsigned long long* pH = a.h_out - 31 * HS;
    uint8_t* pcode = TAPE ? a.tcode + lane : nullptr;
    float* pc1 = TAPE ? a.tc1 + lane : nullptr;
    float* pc2 = TAPE ? a.tc2 + lane : nullptr;

    float tn = 0.0f, tvp = 0.0f;                          // own last result, last upwind value
    float tnl = 0.0f, tvpl = 0.0f;                        // their lo parts (compensated)
    float cU = 0.0f, cI = 0.0f, cN = 0.0f;                // carried S of rows r-1, r and i1 (the one of the two on the upwind side)
    const int nsteps = ncols + 31;
    int next_pub = a.publish ? a.publish : -1;            // the block that publishes the progress next
    int b0 = 0;                                           // ring slot of march s0
    // ring offset of the lane's march s0 - lane; the lane's row of a slot
    unsigned ro = ((RING - lane) % RING) * P;
    float* const ringr = ring + tix;

    // Blocks of U steps: one wait for the staged columns per block, then the
    // block's ring reads, its U node updates, and its stores. Within a block
    // the node updates are the only serial chain; the loads before and the
    // stores after it are independent of it.
    auto block = [&](int s0, auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        auto stage_next = [&]() {
            int pf0 = b0 + LOOK;
            if (pf0 >= RING) pf0 -= RING;
            stage_cols(s0 + LOOK, pf0, fast_tag);
            stage_pairs(s0 + PLOOK, fast_tag);
            cp_commit();
        };
        // staged: columns up to s0+U-1 (a leftward march reads one more), pairs up to s0+U-1
        constexpr int kCols = LOOK / U - (DIR > 0 ? 1 : 2), kPairs = PLOOK / U - 1;
        cp_wait<(kCols < kPairs) ? kCols : kPairs>();
        __syncwarp();

        unsigned off[U];
        float nU[U], nI[U], told[U], toldl[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            off[u] = ro;
            ro = ring_next<P, RING * P>(ro);
            // S of the new column: march m (rightward) or m+1
            const unsigned ns = right ? off[u] : ro;
            nU[u] = ringr[ns + kS0];
            nI[u] = ringr[ns + kS0 + 1];
            told[u] = ringr[off[u] + kT0];
            toldl[u] = COMP ? ringr[off[u] + kL0] : 0.0f;
        }
        // write back the columns every lane had finished before this block (marches s0-U-31 ..)
        {
            if constexpr (VEC) {
                const int m = s0 + vu - U - 31;
                const float* q = ring + wo + vc;
                wo = ring_next<U * P, RING * P>(wo);
                if (FAST || (m >= 0 && m < ncols)) {
                    *reinterpret_cast<float4*>(pW) = *reinterpret_cast<const float4*>(q + kT0);
                    if (COMP) *reinterpret_cast<float4*>(pWl) = *reinterpret_cast<const float4*>(q + kL0);
                }
            } else {
                int wb = b0 + (RING - 31 - U);
                if (wb >= RING) wb -= RING;
                const float* q = ring + kT0 + tix;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int m = s0 + u - U - 31;
                    int ws = wb + u;
                    if (ws >= RING) ws -= RING;
                    if (vrow && (FAST || (m >= 0 && m < ncols))) {
                        pW[u * dT] = q[ws * P];
                        if (COMP) pWl[u * dT] = q[ws * P + kL0 - kT0];
                    }
                }
            }
            pW += U * dT;
            if (COMP) pWl += U * dT;
        }
        // the upwind strip's values of the block (every lane reads them, lane 0 uses them)
        float hv[U], hvl[U];
        {
            const float* q = pring + pi;
            pi ^= kPairWords;
            unsigned stale = 0;
            if (COMP) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint4 e = *reinterpret_cast<const uint4*>(q + 4 * u);
                    hv[u] = __uint_as_float(e.x);
                    hvl[u] = __uint_as_float(e.z);
                    if (FAST || s0 + u < ncols) stale |= (e.y ^ a.tag_in) | (e.w ^ a.tag_in);
                }
            } else {
#pragma unroll
                for (int u = 0; u < U; u += 2) {
                    const uint4 e = *reinterpret_cast<const uint4*>(q + 2 * u);
                    hv[u] = __uint_as_float(e.x);
                    hv[u + 1] = __uint_as_float(e.z);
                    hvl[u] = hvl[u + 1] = 0.0f;
                    if (FAST || s0 + u < ncols) stale |= e.y ^ a.tag_in;
                    if (FAST || s0 + u + 1 < ncols) stale |= e.w ^ a.tag_in;
                }
            }
            // the rare cases of a block behind one branch
            if ((consumer && stale != 0) || s0 + LOOK + U > avail || s0 == next_pub) {
                if (consumer && stale != 0) {
                    // a pair the previous strip had not written when it was prefetched:
                    // wait for it, then fall AHEAD columns behind so later prefetches hit
                    if (lane0) {
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int s = s0 + u;
                            if (FAST || s < ncols) {
                                hv[u] = wait_pair(a.h_in + HS * s, a.tag_in, sh, a.err);
                                if (COMP) hvl[u] = wait_pair(a.h_in + HS * s + 1, a.tag_in, sh, a.err);
                            }
                        }
                        wait_pair(a.h_in + HS * min(s0 + U - 1 + B::AHEAD, ncols - 1), a.tag_in, sh, a.err);
                    }
                    __syncwarp();
                }
                ensure(s0 + LOOK + U);
                if (s0 == next_pub) {
                    publish_progress(a.prog_out, a.tag, min(s0 - 31, ncols));
                    next_pub += a.publish;
                }
            }
        }

        stage_next();  // the ring reads above are in flight meanwhile

        float tnw[U], tnwl[U], sr[U];
        Rec rec[U];
        bool any_far = false;
        // Step u's tape entry. The plain arithmetic writes it in the step; the
        // compensated, whose batches are short of issue slots, after the block,
        // where one vote skips the coefficients of a block without a far
        // candidate (1000 windows of about 1000 x 1001 cells 30.2 -> 29.0 ms;
        // 7 shots of 333 x 97 in the plain arithmetic 0.38 -> 0.40 that way).
        [[maybe_unused]] auto write_entry = [&](int u, int code, float c1, float c2) {
            if (FAST || s0 + u < nsteps) {
                pcode[32 * u] = (uint8_t)code;
                pc1[32 * u] = c1;
                pc2[32 * u] = c2;
            }
        };
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int s = s0 + u;
            const int m = s - lane;
            const int j = col_of(m);
            const bool act = FAST || (vrow && (m >= 0) && (m < ncols));
            // upwind value from the lane above (or the previous strip)
            float tv = __shfl_up_sync(0xffffffffu, tn, 1);
            float tvl = COMP ? __shfl_up_sync(0xffffffffu, tnl, 1) : 0.0f;
            if (lane0) {
                tv = hv[u];
                if (COMP) tvl = hvl[u];
            }
            const float te = tn, tev = tvp;
            [[maybe_unused]] const float tel = tnl, tevl = tvpl;

            float to = told[u], tol = toldl[u];
            if (!FAST && src_rows) {
                const int da = r - a.sIdz + 1, db = j - a.sIdx + 1;
                if (da >= 0 && da < 3 && db >= 0 && db < 3) {
                    to = a.init[da + 3 * db];
                    tol = 0.0f;
                }
            }
            const bool inner = FAST ? irow
                                    : act && irow && (j >= 1) && (j <= ncols - 2) && !(r == a.skip_i && j == a.skip_j);
            // row i1 (downward r-1, else r), columns j-1 (clamped to 1) and j; the
            // order matters to the tape only
            const float nN = down ? nU[u] : nI[u];
            float s1a = cN, s1b = nN;
            if (TAPE || !FAST) {
                s1a = right ? cN : nN;
                s1b = right ? nN : cN;
                if (!FAST && j == 1) s1a = s1b;
            }
            // column j1: rows max(i-1,1) and i
            const float s2a = row1 ? cI : cU;
            const int dc1a = (FAST || j - 1 >= 1) ? 0 : 16;
            float tnew, tnewl = 0.0f;
            if constexpr (COMP)
                node_update_comp<TAPE, EXACT, SQ>(to, tol, tv, tvl, te, tel, tev, tevl, s1a, s1b, s2a, cI, cN,
                                                  a.kc, cz, cx, dc1a, dr2a, tnew, tnewl, rec[u]);
            else
                tnew = node_update<TAPE, REF, EXACT, SQ>(to, tv, te, tev, s1a, s1b, s2a, cI, cN, a.kc,
                                                         cz, cx, dc1a, dr2a, rec[u]);
            tnw[u] = inner ? tnew : to;
            tnwl[u] = COMP ? (inner ? tnewl : tol) : 0.0f;
            if (TAPE) {
                rec[u].code = inner ? rec[u].code : kKept;
                rec[u].upd &= inner;
                rec[u].far &= inner;
                any_far |= rec[u].far;
                sr[u] = cN;
                if constexpr (!COMP) {
                    float c1, c2;
                    node_record<COMP, EXACT, SQ>(rec[u], cN, a.kc, c1, c2);
                    write_entry(u, rec[u].code, c1, c2);
                }
            }
            // carry state
            if (act) {
                tn = tnw[u];
                tnl = tnwl[u];
            }
            tvp = tv;
            tvpl = tvl;
            cU = nU[u];
            cI = nI[u];
            cN = nN;
        }

        if constexpr (TAPE) {
            if constexpr (COMP) {
                float c1[U], c2[U];
                if (__any_sync(0xffffffffu, any_far)) {
#pragma unroll
                    for (int u = 0; u < U; u++) node_record<COMP, EXACT, SQ>(rec[u], sr[u], a.kc, c1[u], c2[u]);
                } else {
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        c1[u] = 0.0f;
                        c2[u] = rec[u].upd ? (SQ || rec[u].w11 ? a.kc.dz : a.kc.dx) : 0.0f;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; u++) write_entry(u, rec[u].code, c1[u], c2[u]);
            }
            pcode += 32 * U;
            pc1 += 32 * U;
            pc2 += 32 * U;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int m = s0 + u - lane;
            const bool act = FAST || (vrow && (m >= 0) && (m < ncols));
            if (act) {
                ringr[off[u] + kT0] = tnw[u];
                if (COMP) ringr[off[u] + kL0] = tnwl[u];
            }
            // feed the next strip: lane 31 just finished march s-31
            if (feeds && act) {
                if constexpr (COMP)
                    st_pairs(pH + HS * u, tnw[u], tnwl[u], a.tag);
                else
                    st_u64(pH + HS * u, pack_tag(tnw[u], a.tag));
            }
        }
        pH += HS * U;
        b0 += U;
        if (b0 >= RING) b0 -= RING;
    };
    // one block past the last step writes the last columns back
    [[maybe_unused]] const unsigned nfast = max(ncols - LOOK - U - (31 + U), 0);  // first steps of interior blocks: 31 + U ..
#pragma unroll 1
    for (int s0 = 0; s0 < nsteps + U; s0 += U) {
        if constexpr (INTERIOR) {
            if ((unsigned)(s0 - (31 + U)) < nfast && (unsigned)(s0 - g0) > (unsigned)gn)
                block(s0, std::true_type{});
            else
                block(s0, std::false_type{});
        } else {
            block(s0, std::false_type{});
        }
    }
    if (a.prog_out) publish_progress(a.prog_out, a.tag, ncols);
    cp_wait<0>();
    __syncwarp();
}

// Gang-wide barrier: every CTA of the gang arrives once per barrier instance;
// `target` = (instance + 1) * gang size. Bounded like every wait.
__device__ __forceinline__ void gang_barrier(unsigned* ctr, unsigned target, CtaShared* sh, int* err)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(ctr, 1u);
        wait_counter(ctr, target, sh, err);
        __threadfence();
    }
    __syncthreads();
}

// Counters of a persistent launch of NG gangs: a barrier counter per gang,
// the queue (shots taken past the gangs' first ones), two next-shot words per gang.
__host__ __device__ constexpr size_t gang_counters(int NG) { return 3 * (size_t)NG + 1; }
constexpr int kMaxSolves = 1023;  // shots one gang takes in a launch (the tags' 10-bit shot-solve number)

// Ends the gang's shot number `it` (its buffers are free for the next) and
// returns the next one from the queue, for every thread of the gang. Shots
// are sorted widest first, so taking them as gangs fall free balances uneven
// windows: 1000 windows of 400 to 1600 columns on 456 gangs took 52.9 ms
// (forward) and 26.0 ms (reverse) dealt in turn, where the gangs' sums range
// from 0.7 to 1.4 of their mean.
__device__ __forceinline__ int next_shot(unsigned* ctr, int NG, int G, int gang, int g, int it, unsigned& nbar,
                                         CtaShared* sh, int* err)
{
    // two words in turn: a CTA may still read the last one
    unsigned* slot = ctr + NG + 1 + 2 * (size_t)gang + (it & 1);
    if (g == 0 && threadIdx.x == 0)
        *(volatile unsigned*)slot = (it + 1 < kMaxSolves) ? (unsigned)NG + atomicAdd(ctr + NG, 1u) : 0x7fffffffu;
    gang_barrier(ctr + gang, (++nbar) * G, sh, err);
    if (threadIdx.x == 0) {
        const bool stop = ld_volatile(&sh->abort_flag) || *(volatile int*)err;  // a wait gave up: results are void
        sh->item = stop ? 0x7fffffff : (int)*(volatile unsigned*)slot;
    }
    __syncthreads();
    return sh->item;
}

}  // namespace sf
