// Device code of the full-pairwise distance stage for sm_103a.
//
// One warp aligns one sequence pair end to end, the way
// FullPairwiseAlign::pairwiseAlign does it per (si, sj)
// (CPU/clustalw-2.0.11/src/pairwise/FullPairwiseAlign.cpp:112-183):
//   1. forwardPass  (:280-341)  local Gotoh sweep, max score, first max cell
//   2. reversePass  (:343-416)  reverse sweep from the end cell, start cell
//   3. diff         (:418-612)  Myers-Miller recursion on the [sb..se] box
//   4. tracePath    (:231-278)  identity count, folded into diff's M==1 leaves
//   5. distance     (:172-181)  float arithmetic identical to the reference
//
// All dynamic-programming sweeps of steps 1-3 run on one primitive, `sweep`:
// a row-striped anti-diagonal wavefront. Lane l of a W-lane segment owns R
// consecutive rows of the current stripe and processes column c = t - l + 1 at
// step t. H and E of the row above arrive from lane l-1 by __shfl_up_sync; the
// segment's first lane takes them from the previous stripe's last row, which
// the segment reads W columns at a time with one coalesced load and hands to
// that lane by shuffle, or from the closed-form boundary of the first stripe.
//
// A cell costs five integer instructions, three of them on the ALU pipe (64
// lanes per SM and clock, the pipe that bounds every sweep):
//   t = H(r-1,c-1) + s                          dp2a (picks one int16 score and adds: FMA pipe)
//   H = max(E, F, t [, 0])                      __vimax3_s32[_relu]
//   g = H - (gapOpen + gapExtend)               add (either pipe)
//   E(r+1,c) = max(E(r,c) - ge, g)              __viaddmax_s32
//   F(r,c+1) = max(F(r,c) - ge, g)              __viaddmax_s32
// which is the reference's recurrence with E and F carried one cell ahead.
// Measured with all operands in registers: 20.2 cells per SM and clock, against
// 12.7 for the form with two more ALU instructions (an unpack of the score and
// a second two-way max in place of the three-way one); the 200 x 1523 protein
// family 110.4 -> 89.0 ms.
//
// Scores come from a per-stripe int16 profile in shared memory,
// prof[code][lane][row], one conflict-free 16-byte load per step and lane
// (8 bytes in the short-pair kernel, whose lanes hold 4 rows).
// Residues are remapped on the host to the K codes that occur (K <= 32), so
// the profile holds K rows of codes.
//
// Myers-Miller frames small enough (M <= tiny_m, N <= tiny_n) are not swept
// by the warp: they are queued, and 32 of them at a time are solved one per
// lane with the reference's sequential loops, rows kept in the lane's column
// of the warp's shared scratch.
#pragma once

#include <climits>
#include <stdint.h>

#include "cwgpu.h"
#include "cwgpu_layout.h"

namespace cwgpu {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kR = 8;              // rows per lane in every sweep of long pairs
constexpr int kRShort = 4;         // rows per lane in the short-pair kernel
constexpr int kTinyMaxN = 16;      // tiny frames: N <= kTinyMaxN (shared-memory rows)
constexpr int kTinyStride = kTinyMaxN + 1;
constexpr int kTinyWords = 4 * kTinyStride * 32;  // HH, DD, RR, SS for 32 lanes
constexpr int kTinyStack = 16;

// Bytes of the per-warp shared region: the stripe profile or the tiny-frame rows.
__host__ __device__ constexpr int warp_region_bytes(int K) {
    return (K * 32 * kR * 2 > kTinyWords * 4) ? K * 32 * kR * 2 : kTinyWords * 4;
}

// One rectangular sweep. Row r (0-based) uses residue rseq[r]; column c
// (1-based) uses residue cseq[c - 1]. Sweeps that run backwards over a
// sequence read its reversed copy, so every sweep reads its residues in
// ascending address order. cseq[-kGuard .. cols + kGuard) must be readable.
// Closed-form boundaries, which is what every sweep of the reference uses:
//   H(-1, c) = ht0 - c*hts        E(-1, c) = H(-1, c) - eo      (c >= 1)
//   H(r, 0)  = hl0 - (r+1)*hls    F(r, 0)  = H(r, 0) - fo
//   H(-1, 0) = corner
// buf[c] (c = 1..cols) carries (H, E) of the last row of a stripe to the next
// stripe, and in MODE_GLOBAL holds the final row on return.
struct Task {
    const int8_t* rseq;
    const int8_t* cseq;
    int2* buf;
    int rows, cols;
    int ht0, hts, eo;
    int hl0, hls, fo;
    int corner;
    int pad;  // padding rows above the first (less than the rows of a lane)
};

// MODE_LOCAL_FWD: H floored at 0, the first maximum in row-major order tracked
// (forwardPass's strict `hh > maxScore`). reversePass runs in the same loops,
// on H + 1: the corner is 1, and its boundary of -1 becomes the floor. The
// floor also holds inside the sweep there, which reversePass's does not; that
// only adds paths that start at -1, whose remainder is a local alignment of at
// most maxScore, so the first cell to reach maxScore is the same. The general
// form (GEN, any penalties) cannot argue so and has MODE_LOCAL_REV: no floor,
// and the first cell of the maximum of min(H, thresh) tracked (reversePass's
// strict `hh > cost` and its break at cost >= maxScore).
enum { MODE_LOCAL_FWD = 0, MODE_LOCAL_REV = 1, MODE_GLOBAL = 2 };

struct Best {
    int val;
    unsigned key;  // (row << 16) | col of the winning cell
};

// Rows of the shared matrix: 32 codes and a padding row of kPadScore.
constexpr int kPadRow = 32;
constexpr int kSmatWords = (kPadRow + 1) * 32;
constexpr int kPadScore = -32768;

// Per-block constants the device functions read.
struct Env {
    unsigned smat_at;    // shared matrix over remapped codes: 32x32, then the padding row
    unsigned region_at;  // this warp's shared region (profile, tiny rows, box edges or frame stack)
    int K;               // number of remapped codes
    int gp1, gp2;        // remapped gapPos1 / gapPos2 (-1 if absent)
    int tiny_m, tiny_n;  // tiny-frame thresholds
    int* err;

    // Kept as addresses in shared memory, so that functions that are not
    // inlined still read them with shared-memory loads.
    __device__ __forceinline__ void set_shared(const int* smat, uint16_t* region) {
        smat_at = (unsigned)__cvta_generic_to_shared(smat);
        region_at = (unsigned)__cvta_generic_to_shared(region);
    }
    __device__ __forceinline__ const int* smat() const {
        return static_cast<const int*>(__cvta_shared_to_generic(smat_at));
    }
    __device__ __forceinline__ uint16_t* region() const {
        return static_cast<uint16_t*>(__cvta_shared_to_generic(region_at));
    }
};

template <int R>
struct SweepState {
    int hl[R];  // H(r, c-1)
    int fp[R];  // F(r, c)
    int diag;   // H of the row above the lane's first row, column c-1
    int hout, eout;  // H of the lane's last row, E of the row below it
    int thr;         // the lane's tracked maximum: columns that reach it are examined
    int bv;          // the maximum of the lane's rows in this stripe
    unsigned bk;     // its first cell in row-major order: (row in lane << 16) | column
    int ch, ce, nh, ne;  // boundary chunks (H above, E of the stripe's first row): current and next W columns
};

// Residue load. NC: through the read-only data path (codes written before the
// kernel started); otherwise a plain load (codes the kernel itself wrote).
template <bool NC>
__device__ __forceinline__ int ldres(const int8_t* p) {
    if constexpr (NC)
        return (int)__ldg(p);
    else
        return (int)*p;
}

// The R int16 scores of one (code, lane) profile entry, two per word: one
// 16-byte (R == 8) or 8-byte (R == 4) shared load.
template <int R>
__device__ __forceinline__ void load_scores(const uint16_t* p, int (&w)[R / 2]) {
    static_assert(R == 8 || R == 4, "profile entries hold 4 or 8 rows");
    if constexpr (R == 8) {
        const int4 v = *reinterpret_cast<const int4*>(p);
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
    } else {
        const int2 v = *reinterpret_cast<const int2*>(p);
        w[0] = v.x;
        w[1] = v.y;
    }
}

// d + one of the two int16 scores of w, in one instruction: the dot product
// of w's halves with (1, 0) or (0, 1).
template <bool HI>
__device__ __forceinline__ int add_score(int w, int d) {
    return __dp2a_lo(w, HI ? 0x0100 : 0x0001, d);
}

__device__ __forceinline__ unsigned pack2(int lo, int hi) {
    return ((unsigned)lo & 0xffffu) | ((unsigned)hi << 16);
}

// prof[(b*32 + lane)*R + k] = matrix[a[k]][b] for the K codes b. Lane l starts
// at code l % K so that its shared-matrix reads spread over the banks.
template <int R>
__device__ __forceinline__ void build_profile(uint16_t* prof, const int* smat, const int (&a)[R], int lane,
                                              int K) {
    int b = lane % K;
    for (int i = 0; i < K; ++i) {
        if constexpr (R == 8) {
            uint4 w;
            w.x = pack2(smat[a[0] * 32 + b], smat[a[1] * 32 + b]);
            w.y = pack2(smat[a[2] * 32 + b], smat[a[3] * 32 + b]);
            w.z = pack2(smat[a[4] * 32 + b], smat[a[5] * 32 + b]);
            w.w = pack2(smat[a[6] * 32 + b], smat[a[7] * 32 + b]);
            *reinterpret_cast<uint4*>(prof + (b * 32 + lane) * 8) = w;
        } else {
            uint2 w;
            w.x = pack2(smat[a[0] * 32 + b], smat[a[1] * 32 + b]);
            w.y = pack2(smat[a[2] * 32 + b], smat[a[3] * 32 + b]);
            *reinterpret_cast<uint2*>(prof + (b * 32 + lane) * 4) = w;
        }
        b = (b + 1 == K) ? 0 : b + 1;
    }
}

// ---------------------------------------------------- warps sharing one sweep

// Device-side status values of the pair kernels' status word (nonzero = error).
enum { kStatusStackLimit = 1, kStatusTimeout = 2 };

// Hand-over of stripe boundary rows between the warps of a CTA that sweep one
// task together (stripes dealt round-robin). Warp w writes the last row of
// each of its stripes into its own row buffer and publishes how far it got in
// its progress word: epoch | stripe << 17 | columns written, which only grows
// (columns <= 65535, stripes <= 511, epochs count the CTA's sweeps). The warp
// with the next stripe waits for that word before it loads a chunk of the
// row. Every wait is bounded: past `limit_ns` it records kStatusTimeout, sets
// `abort`, and every later wait of the CTA returns at once, so the kernel
// ends (with wrong values that the host does not return).
struct MwSync {
    volatile unsigned long long* prog;  // shared: one progress word per warp of the CTA
    volatile int* abort;                // shared
    int* err;                           // global status word
    unsigned long long epoch;           // the sweep's epoch, shifted left by 32
    unsigned long long limit_ns;        // bound of one wait
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned long long mw_word(const MwSync& m, int stripe, int cols) {
    return m.epoch | ((unsigned long long)stripe << 17) | (unsigned)cols;
}

// Warp-uniform: lane 0 waits until progress word `slot` reaches `target`.
__device__ __forceinline__ void mw_wait(const MwSync& m, int slot, unsigned long long target) {
    if ((threadIdx.x & 31) == 0 && m.prog[slot] < target && !*m.abort) {
        const unsigned long long t0 = global_ns();
        for (unsigned polls = 1;; ++polls) {
            if (m.prog[slot] >= target || *m.abort) break;
            if ((polls & 63) == 0 && global_ns() - t0 > m.limit_ns) {
                *m.abort = 1;
                atomicExch(m.err, kStatusTimeout);
                break;
            }
        }
    }
    __threadfence_block();  // the row entries published before the word are read after it
    __syncwarp();
}

// One lane: the row entries it wrote are visible to the CTA before the word.
__device__ __forceinline__ void mw_publish(const MwSync& m, int slot, int stripe, int cols) {
    __threadfence_block();
    m.prog[slot] = mw_word(m, stripe, cols);
}

// A stripe's place in a shared sweep: the row above comes from the predecessor
// warp's buffer and the stripe's last row goes to the own one.
struct StripeIO {
    int stripe;      // index of the stripe in the task
    int pred_slot;   // progress word of the warp with the previous stripe
    int own_slot;    // progress word of this warp
    bool publisher;  // this lane's row is the next stripe's boundary
};

// The local sweeps of one warp keep rows that only they and the path read back,
// much later: past L1, which at five CTAs per SM is small and holds the residues.
template <int MODE, bool MW>
__host__ __device__ constexpr bool rows_in_l2() {
    return MODE != MODE_GLOBAL && !MW;
}
template <bool L2>
__device__ __forceinline__ void row_store(int2* p, int2 v) {
    if constexpr (L2)
        __stcg(p, v);
    else
        *p = v;
}
template <bool L2>
__device__ __forceinline__ int2 row_load(const int2* p) {
    if constexpr (L2)
        return __ldcg(p);
    else
        return *p;
}

// E of a task's first row, given H of the row above it.
__device__ __forceinline__ int first_row_e(const Task& T, int h, int ge, int goe) {
    return max(h - T.eo - ge, h - goe);
}

// Whether the padding rows of the sweeps are sound for these penalties; the
// others (negative ones, or extensions beyond the padding score) take GEN.
constexpr int kMaxPaddedOpen = 1 << 27;
__host__ __device__ inline bool padding_sound(int go, int ge) {
    return go >= 0 && go <= kMaxPaddedOpen && ge >= 0 && ge <= -kPadScore - 1;
}

// The steps of one stripe. Lane sl processes column c = t - sl + 1 at step t.
// Lane 0 of the segment takes the row above from the chunk registers (W columns
// per lane-wide load: the previous stripe's last row, or the closed-form top
// boundary for the first stripe). The next step's residue is loaded one step
// ahead from the lane's own pointer, without clamping (the layout's guard bytes
// make the reads of fill and drain steps safe).
// The first `fill` steps (at least the used lanes less one, even, at most W),
// in which lanes wait for their first column, test each lane's column range;
// the steps after them do not: a lane past its last column computes on, from
// residues and boundary values that nothing else reads, and only its stores
// and its tracked maximum are held to the range. Those steps run two per
// iteration and a chunk (W of them) per turn of the outer loop. The sweeps are
// bound by issue slots and the ALU pipe together (40 instructions per 8 cells
// are the cells', 24 of them on that pipe), so the rest of the step counts: with
// a range test and a chunk test in every step a 1523-residue protein pair took
// 3.89 M warp instructions and 200 x 1523 89.0 ms, this way 3.16 M and 80.8 ms
// (110.4 ms before the cells' own change). Four steps per iteration overflow
// the instruction cache.
// The maximum is tracked per lane on the step's maximum over the lane's rows;
// only when it reaches the lane's own maximum is its row looked up.
// PARTIAL: gap penalties outside the range the padding rows are sound for
// (padding_sound) and a stripe that the task's last row may end inside: the rows
// past it pass the row above through, two selects per cell, so the segment's
// last used lane still emits the last real row. One copy of the step, which
// tests its range: with three the general kernels, which have most forms of it,
// wait for instructions (proteins with a negative gap opening, 100 x 400 and 60 x
// 1000: 4.60 and 6.50 ms against 4.13 and 6.83; the selects in every stripe, as
// once, 4.51 and 7.18).
// A lane with `writer` set stores its last row's (H, E) to `own`; the row above
// the stripe is read from `above`.
// MW: the stripe is one of a sweep shared by several warps (MwSync): before a
// chunk of the row above is loaded the predecessor's progress is awaited, and
// the lane with the boundary row publishes its progress between chunks (inside
// the step, with its column test, a column sweep of 1523 x 1523 took 855 k cycles instead of 760 k).
template <int R, int W, int MODE, bool PARTIAL, bool NC, bool MW = false>
__device__ __forceinline__ void run_stripe(int nsteps, int fill, bool first, const Task& T, SweepState<R>& S, int sl,
                                           int nvalid, const int2* above, int2* own, bool writer, int ge, int goe,
                                           int thresh, const uint16_t* prof_lane, const StripeIO& io = StripeIO{},
                                           const MwSync* mw = nullptr) {
    constexpr bool kL2 = rows_in_l2<MODE, MW>();
    const int8_t* cp = T.cseq - sl;                 // residue of step t: cp[t]
    int2* wp = own + 1 - sl;                        // the lane's row entry of step t: wp[t]
    const int wend = writer ? T.cols + sl : INT_MIN;  // the writer stores in steps below this
    int bnext = ldres<NC>(cp);

    auto step = [&](int t, bool test) {
        int hin = __shfl_up_sync(kFull, S.hout, 1, W);
        int ein = __shfl_up_sync(kFull, S.eout, 1, W);
        const int bh = __shfl_sync(kFull, S.ch, t, W);
        const int be = __shfl_sync(kFull, S.ce, t, W);
        if (sl == 0) {
            hin = bh;
            ein = be;
        }
        const int b = bnext;
        bnext = ldres<NC>(cp + t + 1);
        if (test && (unsigned)(t - sl) >= (unsigned)T.cols) return;
        int w[R / 2];
        load_scores<R>(prof_lane + b * (32 * R), w);
        int e = ein, d = S.diag, hup = hin, elast = ein;
        int hs[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int diag = (k & 1) ? add_score<true>(w[k / 2], d) : add_score<false>(w[k / 2], d);
            int h = MODE == MODE_LOCAL_FWD ? __vimax3_s32_relu(e, S.fp[k], diag) : __vimax3_s32(e, S.fp[k], diag);
            const int g = h - goe;
            d = S.hl[k];
            S.fp[k] = __viaddmax_s32(S.fp[k], -ge, g);
            if (PARTIAL) {
                const bool v = k < nvalid;
                const int en = __viaddmax_s32(e, -ge, g);
                elast = v ? e : elast;
                e = v ? en : e;
                h = v ? h : hup;
            } else {
                elast = e;
                e = __viaddmax_s32(e, -ge, g);
            }
            S.hl[k] = h;
            hup = h;
            hs[k] = h;
        }
        S.hout = hup;
        S.eout = e;
        S.diag = hin;
        if (MODE != MODE_GLOBAL) {
            int sm = hs[0];
#pragma unroll
            for (int k = 1; k + 1 < R; k += 2) sm = __vimax3_s32(sm, hs[k], hs[k + 1]);
            if ((R & 1) == 0) sm = max(sm, hs[R - 1]);
            if (sm >= S.thr && t - sl < T.cols) {
                // First row holding the maximum (of min(H, thresh) in the reverse sweep).
                if (MODE == MODE_LOCAL_REV) sm = min(sm, thresh);
                unsigned kk = R - 1;
#pragma unroll
                for (int k = R - 2; k >= 0; --k) kk = hs[k] >= sm ? k : kk;
                const unsigned key = (kk << 16) | (unsigned)(t - sl + 1);
                S.bk = sm > S.bv ? key : min(S.bk, key);
                S.bv = S.thr = sm;
            }
        }
        if (t < wend) row_store<kL2>(wp + t, make_int2(hup, elast));
    };
    // Between chunks (t steps done): how far the boundary row has come.
    auto publish = [&](int t) {
        if constexpr (MW) {
            if (io.publisher && t > sl) mw_publish(*mw, io.own_slot, io.stripe, min(T.cols, t - sl));
        }
    };
    // After the last step of a chunk (t: the step after it).
    auto next_chunk = [&](int t) {
        S.ch = S.nh;
        S.ce = S.ne;
        const int cfirst = t + W + 1, col = cfirst + sl;
        if (first) {
            S.nh = T.ht0 - col * T.hts;
            S.ne = first_row_e(T, S.nh, ge, goe);
        } else {
            if constexpr (MW) {
                if (cfirst <= T.cols)
                    mw_wait(*mw, io.pred_slot, mw_word(*mw, io.stripe - 1, min(T.cols, cfirst + W - 1)));
            }
            if (col <= T.cols) {
                const int2 v = row_load<kL2>(above + col);
                S.nh = v.x;
                S.ne = __viaddmax_s32(v.y, -ge, v.x - goe);
            }
        }
    };

    int t = 0;
    if (!PARTIAL)
        for (; t < fill; ++t) step(t, true);
    publish(t);  // the fill may have been all of it
    if (t == W) next_chunk(t);
    while (t < nsteps) {
        const int tend = min(nsteps, (t | (W - 1)) + 1);
        if (PARTIAL) {
            for (; t < tend; ++t) step(t, true);
        } else {
            for (; t < tend; t += 2) {  // fill and W are even: at most one step past nsteps
                step(t, false);
                step(t + 1, false);
            }
        }
        publish(t);
        if (t < nsteps) next_chunk(t);
    }
}

// Checked steps of a stripe whose segments use at most `lused` lanes.
__device__ __forceinline__ int fill_steps(int lused) { return lused & ~1; }

// A lane's share of a stripe: rows lrow0 .. lrow0 + R - 1 of the task. Rows
// outside [0, rows) are padding, with kPadScore against every residue (GEN:
// rows past the end pass the row above through instead).
// MODE_GLOBAL pads above the first row (pad < R rows, all in the first lane), so
// that the last row is always the last register of the last used lane. A
// padding row r < 0 reproduces the top boundary in every column: its F starts
// at H(-1, 1) and loses ge per column as the boundary does (hts == ge), and E
// and the diagonal term stay below it as long as gapOpen >= 0 and 0 <= ge <=
// -kPadScore. The local mode pads below the last row: such a row's H never
// exceeds one already seen above or to the left of it (gapOpen, ge >= 0), so
// it is never the first maximum. Its reverse sweep pads above too, so that its
// lanes end at the forward sweep's lane ends; those rows are at the floor, as
// the boundary is.
template <int R, int MODE, bool GEN, bool NC>
__device__ __forceinline__ void stripe_begin(const Task& T, SweepState<R>& S, int lrow0, int gbest, int ge, int goe,
                                             int track, const Env& X, int lane) {
    int a[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int r = lrow0 + k;
        a[k] = (r >= 0 && r < T.rows) ? ldres<NC>(T.rseq + r) : (GEN ? 0 : kPadRow);
    }
    __syncwarp();  // previous users of the shared region are done
    build_profile<R>(X.region(), X.smat(), a, lane, X.K);
    __syncwarp();  // previous stripe's buf writes visible to the whole segment
    constexpr int kLow = -(1 << 29);  // below every boundary value
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int r = lrow0 + k;
        S.hl[k] = T.hl0 - (r + 1) * T.hls;
        S.fp[k] = max(S.hl[k] - T.fo - ge, S.hl[k] - goe);
        if (!GEN && r < 0) {
            S.hl[k] = r == -1 ? T.corner : kLow;  // H(-1, 0), else never taken
            S.fp[k] = T.ht0 - T.hts;              // H(-1, 1)
        }
    }
    S.diag = lrow0 == 0 ? T.corner : T.hl0 - lrow0 * T.hls;
    if (!GEN && lrow0 < 0) S.diag = kLow;
    S.hout = 0;
    S.eout = 0;
    S.bv = gbest;
    S.bk = 0xffffffffu;
    S.thr = max(gbest + 1, track);
    if (lrow0 >= T.rows) S.thr = INT_MAX;  // padding only
}

// Boundary chunk registers at the start of a stripe, from the closed form or
// from the previous stripe's last row.
template <int R, int W, bool L2>
__device__ __forceinline__ void stripe_chunks(const Task& T, SweepState<R>& S, const int2* rb, bool first, int sl,
                                              int ge, int goe) {
    if (first) {
        S.ch = T.ht0 - (1 + sl) * T.hts;
        S.ce = first_row_e(T, S.ch, ge, goe);
        S.nh = T.ht0 - (W + 1 + sl) * T.hts;
        S.ne = first_row_e(T, S.nh, ge, goe);
        return;
    }
    S.ch = S.ce = S.nh = S.ne = 0;
    if (1 + sl <= T.cols) {
        const int2 v = row_load<L2>(rb + 1 + sl);
        S.ch = v.x;
        S.ce = __viaddmax_s32(v.y, -ge, v.x - goe);
    }
    if (W + 1 + sl <= T.cols) {
        const int2 v = row_load<L2>(rb + W + 1 + sl);
        S.nh = v.x;
        S.ne = __viaddmax_s32(v.y, -ge, v.x - goe);
    }
}

// Best of the stripe over the warp, folded into `best`.
template <int R>
__device__ __forceinline__ int stripe_best(const SweepState<R>& S, int lrow0, int gbest, Best& best) {
    const unsigned lk = S.bv > gbest ? S.bk + ((unsigned)lrow0 << 16) : 0xffffffffu;
    const int wv = __reduce_max_sync(kFull, S.bv);
    const unsigned wk = __reduce_min_sync(kFull, S.bv == wv ? lk : 0xffffffffu);
    if (wv > best.val) {  // later stripes hold later rows: strict keeps the first
        best.val = wv;
        best.key = wk;
    }
    return wv;
}

// Padding rows that let a task of `rows` rows end with a lane's last row.
template <int R>
__device__ __forceinline__ int lane_padding(int rows) {
    return rows > 0 ? (R - rows % R) % R : 0;
}

// Rows a local sweep keeps for the path (cwgpu_path.cuh). Node row i has the
// first i residues of the forward sequence on one side; a lane whose last row
// is the task's row r ends at i = start + dir * (r + 1) (the forward sweep: 0
// and 1; the reverse: its first row and -1). Those with 0 < i < end and
// i % every == 0 go to rows + (i / every - 1) * stride. rows == nullptr: none.
struct RowSave {
    int2* rows;
    size_t stride;
    int every;
    int start, dir, end;

    // Whether the row after the task's first `rows_done` is one of them, and
    // where it goes (`other` if it is not).
    __device__ __forceinline__ bool keeps(int rows_done) const {
        const int i = start + dir * rows_done;
        return rows && i > 0 && i < end && (i & (every - 1)) == 0;
    }
    __device__ __forceinline__ int2* row(int rows_done, int2* other) const {
        return keeps(rows_done) ? rows + (size_t)((start + dir * rows_done) / every - 1) * stride : other;
    }
};

// The wavefront sweep. W = lanes per segment (32: one task per warp, 16: two
// tasks, one per half-warp; the two tasks have the same column count).
// The local modes track the first cell of the maximum, of values from `track`
// on, and stop after the first stripe that reached thresh.
template <int R, int W, int MODE, bool GEN, bool NC = true>
__device__ __forceinline__ void sweep(const Task& T, int go, int ge, int track, int thresh, const Env& X, Best& best,
                                      const RowSave& save = RowSave{}) {
    const int lane = threadIdx.x & 31;
    const int sl = lane & (W - 1);
    const int goe = go + ge;
    constexpr int RPS = W * R;
    const int pad = T.pad;
    const int prows = T.rows + pad;
    const int nstr = prows > 0 ? (prows + RPS - 1) / RPS : 0;
    const int nstr_max = __reduce_max_sync(kFull, nstr);
    const uint16_t* prof_lane = X.region() + lane * R;
    best.val = 0;
    best.key = 0xffffffffu;
    SweepState<R> S;
    const int2* above = T.buf;

    for (int s = 0; s < nstr_max; ++s) {
        const int seg_rows = min(prows - s * RPS, RPS);
        const int lrow0 = s * RPS + sl * R - pad;
        const int nvalid = max(0, min(R, T.rows - lrow0));
        const int lused = seg_rows > 0 ? (seg_rows + R - 1) / R : 0;
        const int nsteps = (seg_rows > 0 && T.cols > 0) ? T.cols + lused - 1 : 0;
        const int nsteps_max = __reduce_max_sync(kFull, nsteps);
        const bool last = (s == nstr - 1);
        bool writer = (sl == lused - 1) && (MODE == MODE_GLOBAL || !last);
        int2* own = T.buf;
        if (R == kR && MODE != MODE_GLOBAL && !GEN && sl < lused && save.keeps(lrow0 + R)) {
            own = save.row(lrow0 + R, nullptr);
            writer = true;
        }
        const int gbest = best.val;
        stripe_begin<R, MODE, GEN, NC>(T, S, lrow0, gbest, ge, goe, track, X, lane);
        stripe_chunks<R, W, rows_in_l2<MODE, false>()>(T, S, above, s == 0, sl, ge, goe);
        const int fill = fill_steps(__reduce_max_sync(kFull, lused));
        if (GEN && (MODE == MODE_GLOBAL || !__all_sync(kFull, seg_rows == RPS)))
            run_stripe<R, W, MODE, GEN, NC>(nsteps_max, fill, s == 0, T, S, sl, nvalid, above, own, writer, ge, goe,
                                            thresh, prof_lane);
        else
            run_stripe<R, W, MODE, false, NC>(nsteps_max, fill, s == 0, T, S, sl, nvalid, above, own, writer, ge, goe,
                                              thresh, prof_lane);
        if (MODE != MODE_GLOBAL)
            above = reinterpret_cast<const int2*>(__shfl_sync(kFull, reinterpret_cast<unsigned long long>(own), W - 1));
        if (MODE != MODE_GLOBAL) {
            stripe_best<R>(S, lrow0, gbest, best);
            if (best.val >= thresh) break;
        }
    }
    __syncwarp();
}

// A sweep shared by the nw warps of a group (ranks 0..nw-1, CTA warps
// slot0 + rank): stripes of 32 x R rows are dealt round-robin, stripe s to rank
// s % nw, and each stripe's last row goes to the buffer of its warp,
// bufs + (slot0 + rank) * stride, from which the warp with the next stripe
// reads it (MwSync). Every warp tracks the best of its own stripes the way
// sweep() does (strict, so the first in row-major order); the caller reduces
// the ranks' results: maximum value, then lowest key. Local modes: *stop
// (shared, INT_MAX at the start) is lowered to every stripe that reached
// thresh; stripes above it are skipped (their progress is published as
// complete so no successor waits), which leaves the result of the lowest
// such stripe, reversePass's break cell. MODE_GLOBAL: the final row is in the
// buffer of rank (stripes - 1) % nw (see mw_last_rank); padding rows above the
// first do not change the number of stripes.
__host__ __device__ inline int mw_stripes(int rows, int R) { return rows > 0 ? (rows + 32 * R - 1) / (32 * R) : 0; }

template <int R, int MODE, bool GEN, bool NC = true>
__device__ __forceinline__ void sweep_mw(const Task& T, int go, int ge, int track, int thresh, const Env& X, Best& best,
                                         int2* bufs, size_t stride, int slot0, int rank, int nw, const MwSync& mw,
                                         volatile int* stop, const RowSave& save = RowSave{}) {
    constexpr int W = 32;
    const int lane = threadIdx.x & 31;
    const int sl = lane;
    const int goe = go + ge;
    constexpr int RPS = W * R;
    const int pad = T.pad;
    const int prows = T.rows + pad;
    const int nstr = mw_stripes(T.rows, R);
    const uint16_t* prof_lane = X.region() + lane * R;
    best.val = 0;
    best.key = 0xffffffffu;
    if (T.cols <= 0) return;  // no column: nothing to hand over (callers give columns)
    SweepState<R> S;
    StripeIO io;
    io.own_slot = slot0 + rank;

    for (int s = rank; s < nstr; s += nw) {
        io.stripe = s;
        io.pred_slot = slot0 + (s + nw - 1) % nw;
        // The row above: where the last lane of the stripe before wrote its last row.
        const int2* const above = save.row(s * RPS - pad, bufs + (size_t)io.pred_slot * stride);
        if (MODE != MODE_GLOBAL && __shfl_sync(kFull, *stop, 0) < s) {  // one decision per warp
            if (lane == 0) mw_publish(mw, io.own_slot, s, T.cols);
            continue;
        }
        const int seg_rows = min(prows - s * RPS, RPS);
        const int lrow0 = s * RPS + sl * R - pad;
        const int nvalid = max(0, min(R, T.rows - lrow0));
        const int lused = (seg_rows + R - 1) / R;
        const int nsteps = T.cols + lused - 1;
        const bool last = (s == nstr - 1);
        io.publisher = (sl == lused - 1) && (MODE == MODE_GLOBAL || !last);
        int2* const own = save.row(lrow0 + R, bufs + (size_t)(slot0 + rank) * stride);
        const bool writer = io.publisher || (sl < lused && save.keeps(lrow0 + R));
        const int gbest = best.val;
        stripe_begin<R, MODE, GEN, NC>(T, S, lrow0, gbest, ge, goe, track, X, lane);
        if (s > 0) mw_wait(mw, io.pred_slot, mw_word(mw, s - 1, min(T.cols, 2 * W)));
        stripe_chunks<R, W, rows_in_l2<MODE, true>()>(T, S, above, s == 0, sl, ge, goe);
        if (GEN && (MODE == MODE_GLOBAL || seg_rows < RPS))
            run_stripe<R, W, MODE, GEN, NC, true>(nsteps, fill_steps(lused), s == 0, T, S, sl, nvalid, above, own,
                                                  writer, ge, goe, thresh, prof_lane, io, &mw);
        else
            run_stripe<R, W, MODE, false, NC, true>(nsteps, fill_steps(lused), s == 0, T, S, sl, nvalid, above, own,
                                                    writer, ge, goe, thresh, prof_lane, io, &mw);
        if (MODE != MODE_GLOBAL) {
            const int wv = stripe_best<R>(S, lrow0, gbest, best);
            if (wv >= thresh && lane == 0) atomicMin((int*)stop, s);
        }
    }
    __syncwarp();
}

__host__ __device__ inline int mw_last_rank(int rows, int R, int nw) { return (mw_stripes(rows, R) - 1) % nw; }

// ---------------------------------------------------------------- tiny frames

// Sequential Myers-Miller (FullPairwiseAlign.cpp:418-612) on one lane for one
// frame and its whole subtree. Rows live in this lane's column of the warp's
// shared scratch (word j*32 + lane, conflict-free), the frame stack in local
// memory. Returns the frame's score; adds identities, matches and diff()
// inner-loop iterations.
template <bool NC>
static __device__ int lane_mm(const int8_t* s1, const int8_t* s2, int A0, int B0, int M0, int N0, int tbf0, int tef0, int go,
                       int ge, const Env& X, int* scratch, int& ident, int& matches, long long& cells) {
    const int lane = threadIdx.x & 31;
    int* HH = scratch + lane;
    int* DD = HH + kTinyStride * 32;
    int* RR = DD + kTinyStride * 32;
    int* SS = RR + kTinyStride * 32;
#define TI(arr, j) arr[(j) * 32]
    int4 stk[kTinyStack];
    int sp = 0;
    stk[sp++] = make_int4(A0, B0, M0, N0 | (tbf0 << 29) | (tef0 << 30));
    int root_score = 0;
    bool root = true;
    while (sp > 0) {
        const int4 fr = stk[--sp];
        const int A = fr.x, B = fr.y, M = fr.z;
        const int N = fr.w & ((1 << 29) - 1);
        const int tbf = (fr.w >> 29) & 1, tef = (fr.w >> 30) & 1;
        const int tb = tbf ? go : 0, te = tef ? go : 0;
        int midh;
        if (N <= 0) {
            midh = -(M > 0 ? tb + ge * M : 0);
        } else if (M <= 1) {
            if (M <= 0) {
                midh = -(tb + ge * N);
            } else {
                cells += N;
                midh = -(tb + ge) - (te + ge * N);
                const int hh0 = -(te + ge) - (tb + ge * N);
                if (hh0 > midh) midh = hh0;
                int midj = 0;
                const int* row = X.smat() + 32 * ldres<NC>(s1 + A);
                for (int j = 1; j <= N; ++j) {
                    const int hh = row[ldres<NC>(s2 + B + j - 1)] - (N - j > 0 ? te + ge * (N - j) : 0) -
                                   (j - 1 > 0 ? tb + ge * (j - 1) : 0);
                    if (hh > midh) {
                        midh = hh;
                        midj = j;
                    }
                }
                if (midj > 0) {
                    ++matches;
                    const int ra = ldres<NC>(s1 + A), rb = ldres<NC>(s2 + B + midj - 1);
                    if (ra != X.gp1 && rb != X.gp2 && ra == rb) ++ident;
                }
            }
        } else {
            cells += (long long)M * N;
            const int midi = M / 2;
            int t = -tb;
            TI(HH, 0) = 0;
            for (int j = 1; j <= N; ++j) {
                t -= ge;
                TI(HH, j) = t;
                TI(DD, j) = t - go;
            }
            t = -tb;
            for (int i = 1; i <= midi; ++i) {
                const int* row = X.smat() + 32 * ldres<NC>(s1 + A + i - 1);
                int s = TI(HH, 0);
                int hh = t = t - ge;
                TI(HH, 0) = hh;
                int f = t - go;
                for (int j = 1; j <= N; ++j) {
                    f = max(f - ge, hh - go - ge);
                    const int e = max(TI(DD, j) - ge, TI(HH, j) - go - ge);
                    hh = max(max(s + row[ldres<NC>(s2 + B + j - 1)], f), e);
                    s = TI(HH, j);
                    TI(HH, j) = hh;
                    TI(DD, j) = e;
                }
            }
            TI(DD, 0) = TI(HH, 0);
            TI(RR, N) = 0;
            t = -te;
            for (int j = N - 1; j >= 0; --j) {
                t -= ge;
                TI(RR, j) = t;
                TI(SS, j) = t - go;
            }
            t = -te;
            for (int i = M - 1; i >= midi; --i) {
                const int* row = X.smat() + 32 * ldres<NC>(s1 + A + i);
                int s = TI(RR, N);
                int hh = t = t - ge;
                TI(RR, N) = hh;
                int f = t - go;
                for (int j = N - 1; j >= 0; --j) {
                    f = max(f - ge, hh - go - ge);
                    const int e = max(TI(SS, j) - ge, TI(RR, j) - go - ge);
                    hh = max(max(s + row[ldres<NC>(s2 + B + j)], f), e);
                    s = TI(RR, j);
                    TI(RR, j) = hh;
                    TI(SS, j) = e;
                }
            }
            TI(SS, N) = TI(RR, N);
            midh = TI(HH, 0) + TI(RR, 0);
            int midj = 0;
            bool type2 = false;
            for (int j = 0; j <= N; ++j) {
                const int hh = TI(HH, j) + TI(RR, j);
                if (hh >= midh)
                    if (hh > midh || (TI(HH, j) != TI(DD, j) && TI(RR, j) == TI(SS, j))) {
                        midh = hh;
                        midj = j;
                    }
            }
            for (int j = N; j >= 0; --j) {
                const int hh = TI(DD, j) + TI(SS, j) + go;
                if (hh > midh) {
                    midh = hh;
                    midj = j;
                    type2 = true;
                }
            }
            if (sp + 2 > kTinyStack) {
                atomicExch(X.err, 1);
                break;
            }
            if (!type2) {
                stk[sp++] = make_int4(A + midi, B + midj, M - midi, (N - midj) | (1 << 29) | (tef << 30));
                stk[sp++] = make_int4(A, B, midi, midj | (tbf << 29) | (1 << 30));
            } else {
                stk[sp++] = make_int4(A + midi + 1, B + midj, M - midi - 1, (N - midj) | (tef << 30));
                stk[sp++] = make_int4(A, B, midi - 1, midj | (tbf << 29));
            }
        }
        if (root) root_score = midh;
        root = false;
    }
#undef TI
    return root_score;
}

// ---------------------------------------------------------------- diff()

// A CTA's shared stack of Myers-Miller frames (used by the one-CTA-per-pair
// kernel): frames (A, B, M, N | tb << 29 | te << 30) that any warp of the CTA
// may take; count and lock live in shared memory, the lock taken by one lane.
struct FrameShare {
    int4* frames;
    volatile int* count;
    int* lock;
    int cap;
    int min_rows;  // frames with fewer rows stay with the warp that made them
};

// Lane 0: pushes f if the stack has room and its lock is free within a few
// tries; returns whether it did (else the caller keeps the frame).
__device__ __forceinline__ bool share_push(const FrameShare& fs, int4 f) {
    for (int tries = 0; tries < 64; ++tries) {
        if (atomicCAS(fs.lock, 0, 1) == 0) {
            __threadfence_block();
            bool ok = false;
            const int c = *fs.count;
            if (c < fs.cap) {
                fs.frames[c] = f;
                __threadfence_block();
                *fs.count = c + 1;
                ok = true;
            }
            __threadfence_block();
            atomicExch(fs.lock, 0);
            return ok;
        }
    }
    return false;
}

// Midpoint scans of a Myers-Miller frame (FullPairwiseAlign.cpp:570-593), by
// one warp. fwd[j] holds (HH, DD) of row midi from the forward half,
// rev[N - j] holds (RR, SS) of the same row from the reverse half (j =
// 1..N and 0..N-1; the other ends are closed-form). Scan 1 keeps the first j
// reaching the maximum of HH+RR, replaced by the last tied j with HH!=DD &&
// RR==SS; scan 2 switches to a type-2 midpoint at the largest j whose
// DD+SS+gapOpen is strictly above that maximum.
__device__ __forceinline__ void midpoint_scan(const int2* fwd, const int2* rev, int M, int N, int midi, int tb, int te,
                                              int go, int ge, int& midh, int& midj, bool& type2) {
    const int lane = threadIdx.x & 31;
    const int HH0 = -tb - midi * ge;        // HH[0] = DD[0]
    const int RRN = -te - (M - midi) * ge;  // RR[N] = SS[N]
    int b1 = INT_MIN, j1 = 0x7fffffff, jc = -1, b2 = INT_MIN, j2 = -1;
    for (int j = lane; j <= N; j += 32) {
        int hh, dd, rr, ss;
        if (j == 0) {
            hh = dd = HH0;
        } else {
            const int2 v = fwd[j];
            hh = v.x;
            dd = v.y;
        }
        if (j == N) {
            rr = ss = RRN;
        } else {
            const int2 v = rev[N - j];
            rr = v.x;
            ss = v.y;
        }
        const int v1 = hh + rr;
        const bool cond = (hh != dd) && (rr == ss);
        if (v1 > b1) {
            b1 = v1;
            j1 = j;
            jc = cond ? j : -1;
        } else if (v1 == b1 && cond) {
            jc = j;
        }
        const int v2 = dd + ss + go;
        if (v2 >= b2) {
            b2 = v2;
            j2 = j;
        }
    }
    const int V = __reduce_max_sync(kFull, b1);
    const int J1 = (int)__reduce_min_sync(kFull, b1 == V ? (unsigned)j1 : 0x7fffffffu);
    const int JC = __reduce_max_sync(kFull, b1 == V ? jc : -1);
    const int W2 = __reduce_max_sync(kFull, b2);
    const int J2 = __reduce_max_sync(kFull, b2 == W2 ? j2 : -1);
    midh = V;
    midj = max(J1, JC);
    type2 = false;
    if (W2 > midh) {
        midh = W2;
        midj = J2;
        type2 = true;
    }
}

// Myers-Miller recursion (FullPairwiseAlign.cpp:418-612) for one pair. Large
// frames are divided by the warp: forward half on lanes 0-15 and reverse half
// on lanes 16-31, then the midpoint scans as warp reductions. Frames go on an
// explicit stack held in registers (lane k holds frame k); tiny frames go on a
// queue (lane k holds entry k) that is solved 32 at a time by lane_mm. Frames
// are independent once (A, B, M, N, tb, te) are known, and the identity and
// match counts are sums over the M == 1 leaves, so the traversal order is
// free; the top frame's score is diff()'s return value. tb/te are always 0 or
// gapOpen, kept as flags. s1/s2 are 0-based: the reference's 1-based residue
// seq1[A + i] is s1[A + i - 1]. s1r/s2r are the reversed copies of the n- and
// m-residue sequences (s1r[i] = s1[n - 1 - i]), which the reverse halves read.
// N0 carries the top frame's flags: tb = gapOpen if bit 29, te if bit 30 (a
// whole pair's frame has neither). list: its nlist frames (A, B, M, N and
// flags) instead of that one, and no score. SHARE: after each division the right child,
// if it has at least fs->min_rows rows, goes to the CTA's shared stack (when
// it has room) for any warp of the CTA to take, instead of this warp's own.
template <int RS, bool GEN, bool NC = true, bool SHARE = false>
static __device__ __forceinline__ void mm_align(const int8_t* s1, const int8_t* s1r, int n, const int8_t* s2, const int8_t* s2r, int m,
                                int A0, int B0, int M0, int N0, int go, int ge, int2* bufA, int2* bufB, const Env& X,
                                int& mm_score, int& n_ident, int& n_match, long long& cells,
                                const FrameShare* fs = nullptr, const int4* list = nullptr, int nlist = 0) {
    const int lane = threadIdx.x & 31;
    constexpr int NMASK = (1 << 29) - 1;
    int stA = 0, stB = 0, stM = 0, stN = 0;  // stack entry `lane`
    int qA = 0, qB = 0, qM = 0, qN = 0;      // tiny-queue entry `lane`
    if (lane == 0) {
        stA = A0;
        stB = B0;
        stM = M0;
        stN = N0;
    }
    int sp = list ? 0 : 1, nq = 0;
    int next = 0;  // of the list
    bool top = !list;
    int ident = 0, matches = 0, mm = 0;
    long long ncell = 0;
    bool q_has_top = false;  // queue entry 0 is the top frame

    while (sp > 0 || nq > 0 || next < nlist) {
        if (sp == 0 && next < nlist) {
            const int4 f = list[next++];
            if (lane == 0) {
                stA = f.x;
                stB = f.y;
                stM = f.z;
                stN = f.w;
            }
            sp = 1;
        }
        if (sp == 0 || nq == 32) {
            // Solve the queued tiny frames, one per lane.
            __syncwarp();
            int li = 0, lm = 0, score = 0;
            long long lc = 0;
            if (lane < nq) {
                score = lane_mm<NC>(s1, s2, qA, qB, qM, qN & NMASK, (qN >> 29) & 1, (qN >> 30) & 1, go, ge, X,
                                reinterpret_cast<int*>(X.region()), li, lm, lc);
            }
            __syncwarp();
            ident += __reduce_add_sync(kFull, li);
            matches += __reduce_add_sync(kFull, lm);
            ncell += (long long)__reduce_add_sync(kFull, (unsigned)lc);
            if (q_has_top) mm = __shfl_sync(kFull, score, 0);
            q_has_top = false;
            nq = 0;
            continue;
        }
        --sp;
        const int A = __shfl_sync(kFull, stA, sp);
        const int B = __shfl_sync(kFull, stB, sp);
        const int M = __shfl_sync(kFull, stM, sp);
        const int NN = __shfl_sync(kFull, stN, sp);
        const int N = NN & NMASK;
        const int tbf = (NN >> 29) & 1, tef = (NN >> 30) & 1;
        const int tb = tbf ? go : 0, te = tef ? go : 0;

        if (M <= X.tiny_m && N <= X.tiny_n) {
            if (lane == nq) {
                qA = A;
                qB = B;
                qM = M;
                qN = NN;
            }
            if (top) q_has_top = true;  // only possible as entry 0
            top = false;
            ++nq;
            continue;
        }
        if (N <= 0) {  // del(M); return -tbgap(M, tb)
            if (top) mm = -(M > 0 ? tb + ge * M : 0);
            top = false;
            continue;
        }
        if (M <= 1) {
            if (M <= 0) {  // add(N); return -tbgap(N, tb)
                if (top) mm = -(tb + ge * N);
                top = false;
                continue;
            }
            // M == 1 with a long row (:443-477): best single column, first max.
            ncell += N;
            int midh = -(tb + ge) - (te + ge * N);
            const int hh0 = -(te + ge) - (tb + ge * N);
            if (hh0 > midh) midh = hh0;
            const int ra = ldres<NC>(s1 + A);
            int bv = INT_MIN, bj = 0x7fffffff;
            for (int j = lane + 1; j <= N; j += 32) {
                const int rb = ldres<NC>(s2 + B + j - 1);
                const int v = X.smat()[ra * 32 + rb] - (N - j > 0 ? te + ge * (N - j) : 0) -
                              (j - 1 > 0 ? tb + ge * (j - 1) : 0);
                if (v > bv) {
                    bv = v;
                    bj = j;
                }
            }
            const int wv = __reduce_max_sync(kFull, bv);
            const int wj = (int)__reduce_min_sync(kFull, bv == wv ? (unsigned)bj : 0x7fffffffu);
            if (wv > midh) {
                midh = wv;
                const int rb = ldres<NC>(s2 + B + wj - 1);
                ++matches;
                if (ra != X.gp1 && rb != X.gp2 && ra == rb) ++ident;
            }
            if (top) mm = midh;
            top = false;
            continue;
        }

        // Divide (:480-593): forward half on lanes 0-15, reverse half on 16-31.
        const int midi = M / 2;
        ncell += (long long)M * N;
        Task t;
        if (lane < 16) {
            t.rseq = s1 + A;
            t.cseq = s2 + B;
            t.rows = midi;
            t.ht0 = -tb;
            t.hl0 = -tb;
            t.buf = bufA;
        } else {
            // rows A+M-1 down to A+midi and columns B+N-1 down to B, read in
            // ascending order from the reversed copies
            t.rseq = s1r + (n - A - M);
            t.cseq = s2r + (m - B - N);
            t.rows = M - midi;
            t.ht0 = -te;
            t.hl0 = -te;
            t.buf = bufB;
        }
        t.cols = N;
        t.hts = ge;
        t.eo = go;
        t.hls = ge;
        t.fo = go;
        t.corner = 0;
        t.pad = GEN ? 0 : lane_padding<RS>(t.rows);
        Best unused;
        sweep<RS, 16, MODE_GLOBAL, GEN, NC>(t, go, ge, 0, 0, X, unused);

        int midh, midj;
        bool type2;
        midpoint_scan(bufA, bufB, M, N, midi, tb, te, go, ge, midh, midj, type2);
        if (top) mm = midh;
        top = false;
        __syncwarp();  // scan reads of bufA/bufB finish before the next sweep writes

        // Push right then left so the left frame is processed first (:598-609).
        if (sp + 2 > 32) {
            if (lane == 0) atomicExch(X.err, 1);
            break;
        }
        if constexpr (SHARE) {
            const int4 right = !type2 ? make_int4(A + midi, B + midj, M - midi, (N - midj) | (1 << 29) | (tef << 30))
                                      : make_int4(A + midi + 1, B + midj, M - midi - 1, (N - midj) | (tef << 30));
            int shared = 0;
            if (lane == 0 && right.z >= fs->min_rows) shared = share_push(*fs, right) ? 1 : 0;
            if (__shfl_sync(kFull, shared, 0)) {
                if (lane == sp) {
                    stA = A;
                    stB = B;
                    stM = !type2 ? midi : midi - 1;
                    stN = !type2 ? (midj | (tbf << 29) | (1 << 30)) : (midj | (tbf << 29));
                }
                sp += 1;
                continue;
            }
        }
        if (!type2) {
            if (lane == sp) {
                stA = A + midi;
                stB = B + midj;
                stM = M - midi;
                stN = (N - midj) | (1 << 29) | (tef << 30);
            }
            if (lane == sp + 1) {
                stA = A;
                stB = B;
                stM = midi;
                stN = midj | (tbf << 29) | (1 << 30);
            }
        } else {
            if (lane == sp) {
                stA = A + midi + 1;
                stB = B + midj;
                stM = M - midi - 1;
                stN = (N - midj) | (tef << 30);
            }
            if (lane == sp + 1) {
                stA = A;
                stB = B;
                stM = midi - 1;
                stN = midj | (tbf << 29);
            }
        }
        sp += 2;
    }
    mm_score = mm;
    n_ident = ident;
    n_match = matches;
    cells = ncell;
}

// The block's shared copy of the matrix: 32x32 entries, then the padding row.
__device__ __forceinline__ void stage_matrix(int* smat, const int32_t* matrix) {
    for (int i = threadIdx.x; i < kSmatWords; i += blockDim.x) smat[i] = i < 32 * 32 ? matrix[i] : kPadScore;
}

}  // namespace cwgpu

#include "cwgpu_path.cuh"

namespace cwgpu {

struct PairArgs {
    const int8_t* codes;
    const int64_t* offs;
    const int32_t* lens;
    const int32_t* nres;
    const int32_t* pairs;
    const int32_t* order;
    const int32_t* go_table;
    const int32_t* matrix;
    float* dist;
    cwgpu_pair_stats* stats;
    int2* scratch;
    unsigned long long* counter;
    int* err;
    unsigned long long* cells;  // [3]: forward, reverse (up to its break), diff
    long long npairs;
    int lmax;
    int ge;
    int gp1, gp2;  // remapped gap codes
    int K;         // remapped alphabet size
    int tiny_m, tiny_n;
    const PathPool* path;  // on the device, for cwgpu_path.cuh; nullptr: none
    size_t path_bytes;     // of a warp's slice of it
    int general;  // host: gap penalties outside padding_sound somewhere, take the GEN kernels
};

// A sequence's reversed copy (cwgpu_layout.h).
__device__ __forceinline__ const int8_t* rev_of(const int8_t* s, int len) { return s + rev_offset(len); }

// forwardPass over all of s1 x s2.
__device__ __forceinline__ Task local_task(const int8_t* s1, int n, const int8_t* s2, int m, int go, int2* buf) {
    Task t;
    t.rseq = s1;
    t.cseq = s2;
    t.rows = n;
    t.cols = m;
    t.ht0 = t.hts = 0;
    t.eo = go;
    t.hl0 = t.hls = 0;
    t.fo = go;
    t.corner = t.pad = 0;
    t.buf = buf;
    return t;
}

// reversePass from the end cell (se1, se2): rows se1-1 .. 0 of s1, columns
// se2 .. 1. GEN: the reference's -1 boundaries; else H + 1 over the floor
// (MODE_LOCAL_FWD).
template <int RS, bool GEN>
__device__ __forceinline__ Task reverse_task(const int8_t* s1r, int n, int se1, const int8_t* s2r, int m, int se2,
                                             int go, int2* buf) {
    Task t = local_task(s1r + (n - se1), se1, s2r + (m - se2), se2, GEN ? 0 : go, buf);
    if (GEN) {
        t.ht0 = t.hl0 = -1;
    } else {
        t.corner = 1;
        t.pad = lane_padding<RS>(se1);
    }
    return t;
}

// What the local sweeps of a pair find: maxScore, its cell (1-based) and the
// start cell; whether reversePass reached maxScore (else it ran to its end).
struct PairEnds {
    int max_score, se1, se2, sb1, sb2;
    bool reached;
};

// forwardPass, then reversePass from its end cell: one copy of the sweep's code
// for both, which at this size the instruction cache rewards. fwd/rev: rows to
// keep for the path (nullptr: none).
template <int RS, bool GEN, bool NC>
__device__ __forceinline__ PairEnds pair_ends(const int8_t* s1, int n, const int8_t* s2, int m, int go, int ge,
                                              int2* buf, int2* fwd, int2* rev, size_t stride, int every,
                                              const Env& X) {
    PairEnds e{0, 0, 0, 1, 1, false};
    RowSave save{fwd, stride, every, 0, 1, n};
    Task t = local_task(s1, n, s2, m, go, buf);
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        Best b;
        if (GEN && pass == 1)
            sweep<RS, 32, GEN ? MODE_LOCAL_REV : MODE_LOCAL_FWD, GEN, NC>(t, go, ge, 1, e.max_score, X, b);
        else
            sweep<RS, 32, MODE_LOCAL_FWD, GEN, NC>(t, go, ge, pass ? e.max_score + 1 : 1,
                                                   pass ? e.max_score + 1 : INT_MAX, X, b, save);
        if (pass == 0) {
            e.max_score = b.val;
            if (b.val <= 0) break;
            e.se1 = (int)(b.key >> 16) + 1;
            e.se2 = (int)(b.key & 0xffffu);
            t = reverse_task<RS, GEN>(rev_of(s1, n), n, e.se1, rev_of(s2, m), m, e.se2, go, buf);
            save = RowSave{rev, stride, every, e.se1, -1, e.se1};
        } else {
            if (!GEN) b.val -= 1;
            if (b.val > 0) {
                e.sb1 = e.se1 - (int)(b.key >> 16);
                e.sb2 = e.se2 - (int)(b.key & 0xffffu) + 1;
            }
            e.reached = b.val >= e.max_score;
        }
    }
    return e;
}

// The inner-loop iterations the reference executes in the two local sweeps;
// reversePass stops at the first cell reaching maxScore (:404-413).
__device__ __forceinline__ unsigned long long reverse_cells(const PairEnds& e) {
    if (e.max_score <= 0) return 0;
    return e.reached ? (unsigned long long)(e.se1 - e.sb1) * e.se2 + (unsigned long long)(e.se2 - e.sb2 + 1)
                     : (unsigned long long)e.se1 * e.se2;
}

// Distance (:170-181), float arithmetic with IEEE rounding, and the statistics.
__device__ __forceinline__ float pair_result(const PairEnds& e, int mm, int ident, int matches, int len1, int len2,
                                             cwgpu_pair_stats& st) {
    float mmv = (float)(100 * ident);
    if (len1 == 0 || len2 == 0)
        mmv = 0.0f;
    else
        mmv = __fdiv_rn(mmv, (float)min(len1, len2));
    st.fwd_score = e.max_score;
    st.se1 = e.se1;
    st.se2 = e.se2;
    st.sb1 = e.sb1;
    st.sb2 = e.sb2;
    st.mm_score = mm;
    st.n_ident = ident;
    st.n_match = matches;
    return __fdiv_rn(__fsub_rn(100.0f, mmv), 100.0f);
}

// forwardPass + reversePass + diff + distance for one pair, given its 0-based
// code pointers, lengths, non-gap residue counts and gap penalties. Returns
// the distance and fills `st`; adds the algorithmic cell counts (the
// inner-loop iterations the reference executes) to acc[0..2]. RS = rows per
// lane in every sweep: any RS gives the same results; kRShort needs fewer
// warp steps when n <= 128 (one stripe, lanes of 4 rows instead of
// half-empty lanes of 8). Each sequence's reversed copy follows it at the
// next 16-byte boundary (cwgpu_layout.h), and kGuard readable bytes surround both.
template <int RS, bool GEN, bool NC = true>
static __device__ float align_one(const int8_t* s1, int n, const int8_t* s2, int m, int len1, int len2, int go, int ge,
                           int2* bufA, int2* bufB, const Env& X, cwgpu_pair_stats& st, unsigned long long (&acc)[3]) {
    st = cwgpu_pair_stats{0, 0, 0, 0, 0, 0, 0, 0};
    if (n <= 0 || m <= 0) return 1.0f;
    const PairEnds e = pair_ends<RS, GEN, NC>(s1, n, s2, m, go, ge, bufA, nullptr, nullptr, 0, 1, X);
    int mm = 0, ident = 0, matches = 0;
    long long dcells = 0;
    mm_align<RS, GEN, NC>(s1, rev_of(s1, n), n, s2, rev_of(s2, m), m, e.sb1 - 1, e.sb2 - 1, e.se1 - e.sb1 + 1,
                          e.se2 - e.sb2 + 1, go, ge, bufA, bufB, X, mm, ident, matches, dcells);
    acc[0] += (unsigned long long)n * m;
    acc[1] += reverse_cells(e);
    acc[2] += (unsigned long long)dcells;
    return pair_result(e, mm, ident, matches, len1, len2, st);
}

// Aligns pair q: FullPairwiseAlign.cpp:112-183 for one (si, sj).
template <int RS, bool GEN>
static __device__ void align_pair(const PairArgs& g, long long q, const Env& X, int2* bufA, int2* bufB,
                           unsigned long long (&acc)[3]) {
    const int lane = threadIdx.x & 31;
    const int si = g.pairs[2 * q], sj = g.pairs[2 * q + 1];
    const int n = g.lens[si], m = g.lens[sj];
    cwgpu_pair_stats st;
    const float dist = align_one<RS, GEN>(g.codes + g.offs[si], n, g.codes + g.offs[sj], m, g.nres[si], g.nres[sj],
                                 g.go_table[min(n, m)], g.ge, bufA, bufB, X, st, acc);
    if (lane == 0) {
        g.dist[q] = dist;
        if (g.stats) g.stats[q] = st;
    }
}

// The same for the long-pair kernel, with the path of cwgpu_path.cuh where the
// warp has a slice for it. In two parts: everything after the sweeps is a call
// that finds its arguments again by itself, so that the sweeps' loops have the
// registers (with it inlined the compiler computed lane numbers and addresses
// anew in every step).
struct LongPair {
    const int8_t *s1, *s2;
    int n, m, si, sj, go;
    int2* buf;
    PathMem pm;
    bool path;
};

__device__ __forceinline__ LongPair long_pair(const PairArgs& g, long long q, long long slot) {
    LongPair p;
    p.si = g.pairs[2 * q];
    p.sj = g.pairs[2 * q + 1];
    p.n = g.lens[p.si];
    p.m = g.lens[p.sj];
    p.s1 = g.codes + g.offs[p.si];
    p.s2 = g.codes + g.offs[p.sj];
    p.go = g.go_table[min(p.n, p.m)];
    p.buf = g.scratch + (size_t)slot * 2 * (g.lmax + 1);
    const PathPool pool = g.path ? *g.path : PathPool{nullptr, 0};
    p.path = (size_t)(slot + 1) * g.path_bytes <= pool.bytes && path_penalties(p.n, p.m, p.go, g.ge) &&
             path_mem(p.n, p.m, 1, pool.base + (size_t)slot * g.path_bytes, g.path_bytes, p.pm);
    return p;
}

// A pair whose path came from the kept rows, but for `rest` frames.
__device__ __forceinline__ void count_path(const PairArgs& g, int rest) {
    atomicAdd(g.cells + 4, 1ULL);
    if (rest > 0) atomicAdd(g.cells + 5, (unsigned long long)rest);
}

// Whether this pair is divided because the path would cost more: when it is weak
// and most of the launch's pairs before it were. A few weak pairs among related
// ones take the path like the others: an SM whose warps run both ways at a time
// loses more to instruction fetches (300 x 180 proteins, 6 % of the pairs weak:
// 8.6 ms by the path alone, 10.5 by divisions alone, 10.7 with the weak pairs
// divided; 300 unrelated sequences of 400: 32.1, 21.2 and 21.5).
__device__ __forceinline__ bool divide_weak(const PairArgs& g, bool weak) {
    unsigned long long seen = 0;  // weak pairs << 32 | pairs
    if ((threadIdx.x & 31) == 0 && g.cells) seen = atomicAdd(g.cells + 6, ((unsigned long long)weak << 32) + 1);
    seen = __shfl_sync(kFull, seen, 0);
    return weak && 2 * (seen >> 32) >= (seen & 0xffffffffu);
}

static __device__ __noinline__ void finish_long(const PairArgs& g, long long q, long long slot, PairEnds e,
                                                const Env& env) {
    const Env X = env;
    const LongPair p = long_pair(g, q, slot);
    int2* const bufA = p.buf;
    int2* const bufB = bufA + (g.lmax + 1);
    const int A0 = e.sb1 - 1, B0 = e.sb2 - 1;
    int mm = 0, ident = 0, matches = 0;
    long long dcells = 0;
    int rest = -1;  // frames for mm_align; -1: the pair's own
    int near;
    if (p.path && path_scores(e.max_score, p.go) &&
        path_rows(p.pm, bufB, A0, B0, e.se1, e.se2, e.max_score, p.go, 0, 1, near) &&
        !divide_weak(g, e.se1 - A0 < kMinPathRows || !path_pays<4>(near, p.pm.every, e.se1 - A0, e.se2 - B0)) &&
        path_fill<true, false>(p.s1, p.n, p.s2, p.pm, bufB, A0, B0, e.se1, e.se2, e.max_score, p.go, g.ge, X, 0, 1)) {
        rest = path_walk<true, false>(p.s1, p.n, p.s2, p.m, p.pm, bufB, A0, B0, e.se1, e.se2, p.go, g.ge, X, ident, matches,
                               dcells, 0, 1);
        mm = e.max_score;  // the box's best path is the local optimum
    }
    if (rest != 0) {
        int id = 0, mt = 0, score = 0;
        long long ce = 0;
        mm_align<kR, false, true>(p.s1, rev_of(p.s1, p.n), p.n, p.s2, rev_of(p.s2, p.m), p.m, A0, B0, e.se1 - A0,
                                  e.se2 - B0, p.go, g.ge, bufA, bufB, X, score, id, mt, ce, nullptr,
                                  rest > 0 ? p.pm.list : nullptr, max(rest, 0));
        if (rest < 0) mm = score;
        ident += id;
        matches += mt;
        dcells += ce;
    }
    if ((threadIdx.x & 31) == 0) {
        cwgpu_pair_stats st;
        g.dist[q] = pair_result(e, mm, ident, matches, g.nres[p.si], g.nres[p.sj], st);
        if (g.stats) g.stats[q] = st;
        if (g.cells) {
            atomicAdd(g.cells + 0, (unsigned long long)p.n * p.m);
            atomicAdd(g.cells + 1, reverse_cells(e));
            atomicAdd(g.cells + 2, (unsigned long long)dcells);
            if (rest >= 0) count_path(g, rest);
        }
    }
    __syncwarp();
}

__device__ __forceinline__ void align_long(const PairArgs& g, long long q, long long slot, const Env& X) {
    PairEnds e;
    {
        const LongPair p = long_pair(g, q, slot);
        if (p.n <= 0 || p.m <= 0) {
            if ((threadIdx.x & 31) == 0) {
                g.dist[q] = 1.0f;
                if (g.stats) g.stats[q] = cwgpu_pair_stats{0, 0, 0, 0, 0, 0, 0, 0};
            }
            return;
        }
        e = pair_ends<kR, false, true>(p.s1, p.n, p.s2, p.m, p.go, g.ge, p.buf, p.path ? p.pm.fwd : nullptr,
                                       p.path ? p.pm.rev : nullptr, p.pm.stride, p.pm.every, X);
    }
    finish_long(g, q, slot, e, X);
}

}  // namespace cwgpu
