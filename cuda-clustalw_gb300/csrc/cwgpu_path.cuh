// The path diff() chooses, from the rows the local sweeps saved.
//
// Myers-Miller divides a pair's box [sb1..se1] x [sb2..se2] recursively, about
// two more sweeps' worth of cells, but what it decides at a row depends only on
// the cells that lie on some optimal path: the midpoint scan takes the columns
// whose forward and reverse values add up to the frame's optimum, and its tie
// rule compares values of those columns. forwardPass and reversePass have
// already computed both values for every row. So:
//
// 1. Every G rows (G a multiple of 32) the two sweeps keep their row (H, E).
//    Adding them up gives, at such a row, exactly the columns optimal paths
//    cross it in (path_row). Local starts other than (sb1, sb2) and the -1
//    boundaries of reversePass can only add columns or values below the
//    optimum: a path from such a boundary scores at most maxScore - 1.
// 2. Between two such rows optimal paths stay inside the box of their first
//    and last columns, about G x G cells, whose forward and reverse values are
//    recomputed (path_boxes). Every row gets the first and last column of its
//    cells on an optimal path, whether through H (type 1 of the midpoint scan)
//    or inside a vertical gap (type 2).
// 3. The frames of the recursion are then walked 32 at a time, one per lane
//    (path_walk). Where a frame's middle row has a single column and type the
//    midpoint is that column. Elsewhere the lane runs diff()'s own two halves
//    over the rows' column ranges, from the nearest rows above and below where
//    every path goes through H of one cell.
// 4. A type 2 midpoint leaves children with a free gap opening at one corner
//    (tb or te 0), which diff() also grants to a horizontal gap there. Such a
//    path gains gapOpen over its true score, so it can only matter if it is
//    within gapOpen of the optimum; the rows between the corner and the next
//    saved row are computed over the columns of all paths that near, which tells
//    whether one would tie or win (path_ask). A path that uses both of a frame's
//    free corners gains twice, but parts from the optimal paths all the way
//    between: not past a saved row where every path within 2 gapOpen goes
//    through H of one cell (kPathTight). The few frames that are left, and those
//    in boxes too wide for the slice, go to mm_align.
//
// Needs gapExtend >= 1 (with a free extension a gap at the box's corner would
// tie with the local optimum) and penalties and scores that stay far from the
// placeholder for cells outside the rows' ranges (path_penalties, path_scores).
#pragma once

namespace cwgpu {

constexpr int kPathLow = -(1 << 29);  // the value of a cell that no path is taken through
constexpr int kMaxPathScore = 1 << 27;
constexpr int kMaxPathGap = 1 << 28;
// Sets in which no sequence is longer than one stripe keep no rows: their
// divisions are few, and the path's chain of rows, boxes and walk takes longer
// (proteins, divided against path: 55 x 200 0.48 against 0.62 ms, 300 x 180 8.3
// against 8.8; 300 x 300 16.2 against 14.6).
constexpr int kMinPathLength = 32 * kR + 1;
constexpr int kPathRows = 4;          // rows per lane in the boxes
constexpr int kMaxPathG = 4;          // rows between saved rows: 32 * 1, 2 or 4
constexpr int kPathRing = 4;          // steps of forward values in flight

// Whether kPathLow stands below everything it is compared with, and no sum of
// two values leaves 32 bits. The saved rows and the boxes hold whole-pair
// values, 0 to maxScore on an optimal path; the walk counts from a row where H
// is 0, so there a cell on one has -maxScore to maxScore, a midpoint at least
// -maxScore. Out of a placeholder a half gains at most maxScore + gapOpen and the
// other half holds at most as much: 3 * (maxScore + gapOpen) < -kPathLow keeps
// their sum below the midpoint's. Downwards a gap may run on from a
// placeholder for as many columns as there are.
__device__ __forceinline__ bool path_penalties(int n, int m, int go, int ge) {
    return ge >= 1 && go <= kMaxPathScore && (long long)ge * max(n, m) <= kMaxPathGap;
}
__device__ __forceinline__ bool path_scores(int best, int go) { return best > 0 && best <= kMaxPathScore - go; }

// The memory for all slices as the launches find it: nullptr, 0 if there is none.
struct PathPool {
    unsigned char* base;
    size_t bytes;
};

// A row's cells on optimal paths: through H, inside a vertical gap (no kind at
// all: the row's box was too wide).
enum { kPathH = 1, kPathD = 2, kPathTight = 4 };

// A pair's slice of the saved rows and of the working arrays below, for n x m
// residues and `warps` warps that share it, each with cells and list of
// its own (path_of_warp); fwd == nullptr when there is none.
struct PathMem {
    int every = 0;        // G
    int2* fwd = nullptr;  // row i (i % G == 0, 0 < i < n): fwd + (i / G - 1) * stride, column j at [j]
    int2* rev = nullptr;  // the same rows from reversePass, one above its values: column j at [se2 - j]
    size_t stride = 0;
    int2* cells = nullptr;  // forward values of the boxes in work
    int cell_cap = 0;
    int4* span = nullptr;  // the saved rows' columns: of optimal paths (x, y), near (z, w)
    int4* list = nullptr;  // frames left to mm_align, from the front; to ask for, from the back
    int list_cap = 0;
};

// Bytes of a slice with rows every 32 * g, and its parts. The cells hold the
// boxes a warp works on at a time, 64 columns wider than high: a wider box is
// taken alone.
__host__ __device__ inline size_t path_bytes(int n, int m, int g, int warps = 1, PathMem* p = nullptr,
                                             unsigned char* base = nullptr) {
    const int every = 32 * g;
    const size_t saved = n > 0 ? (size_t)((n - 1) / every) * (size_t)(m + 1) : 0;
    const size_t cells = (size_t)128 * ((m + 1 < every + 64 ? m + 1 : every + 64) + 8 * g);
    const size_t spans = (size_t)(n / every + 1);
    if (p) {
        p->every = every;
        p->stride = (size_t)(m + 1);
        p->cell_cap = (int)cells;
        p->cells = reinterpret_cast<int2*>(base);
        p->span = reinterpret_cast<int4*>(p->cells + warps * cells);
        p->list = p->span + spans;
        p->list_cap = n + 1;
        p->fwd = reinterpret_cast<int2*>(p->list + warps * (size_t)(n + 1));
        p->rev = p->fwd + saved;
    }
    return 8 * (warps * (cells + 2 * (size_t)(n + 1)) + 2 * spans + 2 * saved);
}

__device__ __forceinline__ PathMem path_of_warp(PathMem p, int w) {
    p.cells += (size_t)w * p.cell_cap;
    p.list += (size_t)w * p.list_cap;
    return p;
}

// The finest spacing whose slice fits `cap` bytes.
__device__ __forceinline__ bool path_mem(int n, int m, int warps, unsigned char* base, size_t cap, PathMem& p) {
    for (int g = 1; g <= kMaxPathG; g *= 2) {
        if (path_bytes(n, m, g, warps) <= cap) {
            path_bytes(n, m, g, warps, &p, base);
            return true;
        }
    }
    return false;
}

// A row's columns on optimal paths, relative to the box: first | last << 16,
// and the kinds of its cells.
__device__ __forceinline__ int2 path_entry(int lo, int hi, int kinds) { return make_int2(lo | (hi << 16), kinds); }
__device__ __forceinline__ int path_lo(int2 v) { return v.x & 0xffff; }
__device__ __forceinline__ int path_hi(int2 v) { return (int)((unsigned)v.x >> 16); }
// Every optimal path goes through H of the row's one cell.
__device__ __forceinline__ bool path_single(int2 v) {
    return (v.y & (kPathH | kPathD)) == kPathH && path_lo(v) == path_hi(v);
}

// Columns of saved row i that optimal paths cross it in (lo..hi, kinds), and
// those of paths within gapOpen of the optimum (near_lo..near_hi). kinds has
// kPathTight if that is one cell, in H, also within 2 gapOpen. jl: the first
// column any path within 2 gapOpen crosses the saved row above in, replaced by
// this row's. At the pair's edges (column 0, column se2) a path has just started
// or just ended: H 0 and, one above reversePass's -1, 0.
__device__ __forceinline__ bool path_row(const PathMem& p, int i, int& jl, int se2, int best, int go, int& lo, int& hi,
                                         int& kinds, int& near_lo, int& near_hi) {
    const int lane = threadIdx.x & 31;
    const int2* f = p.fwd + (size_t)(i / p.every - 1) * p.stride;
    const int2* r = p.rev + (size_t)(i / p.every - 1) * p.stride + se2;
    unsigned first = 0xffffffffu, nfirst = 0xffffffffu, wfirst = 0xffffffffu;
    int last = -1, nlast = -1, k = 0, within = 0;
    constexpr int U = 4;  // the rows come from DRAM: several loads in flight
    for (int j0 = jl + lane; j0 <= se2; j0 += 32 * U) {
        int2 a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = min(j0 + 32 * u, se2);
            a[u] = __ldcg(f + max(j, 1));
            b[u] = __ldcg(r - min(j, se2 - 1));
            if (j == 0) a[u] = make_int2(0, kPathLow);
            if (j == se2) b[u] = make_int2(0, kPathLow);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + 32 * u;
            const int vh = a[u].x + b[u].x - 1, vd = a[u].y + b[u].y - 1 + go;
            if (max(vh, vd) < best - 2 * go || j > se2) continue;
            within += 1 + (vd >= best - 2 * go);
            wfirst = min(wfirst, (unsigned)j);
            if (max(vh, vd) >= best - go) {
                nfirst = min(nfirst, (unsigned)j);
                nlast = j;
                const int hit = (vh == best ? kPathH : 0) | (vd == best ? kPathD : 0);
                if (hit) {
                    first = min(first, (unsigned)j);
                    last = j;
                    k |= hit;
                }
            }
        }
    }
    jl = (int)__reduce_min_sync(kFull, wfirst);
    lo = (int)__reduce_min_sync(kFull, first);
    hi = __reduce_max_sync(kFull, last);
    near_lo = (int)__reduce_min_sync(kFull, nfirst);
    near_hi = __reduce_max_sync(kFull, nlast);
    kinds = (int)__reduce_or_sync(kFull, (unsigned)k);
    if (kinds == kPathH && __reduce_add_sync(kFull, within) == 1) kinds |= kPathTight;
    return hi >= 0;
}

// Shared memory of the boxes in work: the ring, the edge rows, the residues.
constexpr int kPathRingWords = kPathRing * 64 * (int)sizeof(int4) / (int)sizeof(uint16_t);
__device__ __forceinline__ int path_code_bytes(int width, int W) { return (width + 4 * W + 7) & ~7; }
__device__ __forceinline__ int path_edge_bytes(int width, int W) { return 8 * width + path_code_bytes(width, W); }
// Whether `used` boxes of W lanes and at most `width` columns fit the slice and
// the warp's shared region.
__device__ __forceinline__ bool path_fits(const PathMem& p, int used, int width, int W, int K) {
    const int shared = kPathRingWords * (int)sizeof(uint16_t) + used * path_edge_bytes(width, W);
    return used * (width + W) <= p.cell_cap / (W * kPathRows) && shared <= warp_region_bytes(K);
}

// 16 bytes from global to shared memory without passing through registers;
// the lane that copied them reads them after the wait.
__device__ __forceinline__ void copy_async16(int4* to, const int4* from) {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from)
                 : "memory");
#else
    *to = *from;
#endif
}
__device__ __forceinline__ void copy_async_commit() {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.commit_group;" ::: "memory");
#endif
}
template <int LEFT>
__device__ __forceinline__ void copy_async_wait() {
#ifdef __CUDA_ARCH__
    asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
#endif
}

// Box b lies strictly between node rows i0 = max(A0, saved row) and i1 =
// min(se1, next saved row): rows i0 + 1 .. i1 - 1, columns jl..jh of the optimal
// paths.
struct PathBox {
    int i0, i1, jl, jh;
};

__device__ __forceinline__ PathBox path_box(const PathMem& p, int b, int nboxes, int A0, int B0, int se1, int se2) {
    PathBox x;
    const int base = A0 / p.every * p.every;
    x.i0 = b == 0 ? A0 : base + b * p.every;
    x.i1 = b == nboxes - 1 ? se1 : base + (b + 1) * p.every;
    x.jl = b == 0 ? B0 : p.span[b - 1].x;
    x.jh = b == nboxes - 1 ? se2 : p.span[b].y;
    return x;
}

// Forward and reverse values of up to 32 / (p.every / 4) boxes at once, a
// segment of p.every / 4 lanes each (box `mine`, -1: none), four rows per lane,
// columns as a wavefront like the sweeps'. The row above (below) a box comes from the saved
// forward (reverse) row, or is the box's own start (end) corner. Lane rows are
// numbered so that a box's last row ends a lane: the first `pad` ones pass the
// row above through, and a reverse lane's four rows are one forward lane's in
// reverse order, two 16-byte words. Writes the rows' entries to band[i - A0];
// false if a row has no cell on an optimal path. Bound by latency (one warp's
// chain of steps), so the residues and the edge rows are in shared memory, and
// the forward values come from L2 through a ring there, kPathRing - 1 steps
// ahead.
template <bool NC>
__device__ __noinline__ bool path_boxes(const int8_t* s1, int n, const int8_t* s2, const PathMem& mem, int2* band, int A0, int B0,
                           int se1, int se2, int mine, int width, int nboxes, int best, int go, int ge,
                           const Env& env) {
    const Env X = env;  // copies stay in registers across the stores below
    const PathMem p = mem;
    constexpr int R = kPathRows;
    const int lane = threadIdx.x & 31, W = p.every / R, seg = lane / W, sl = lane & (W - 1);
    const int goe = go + ge;
    const PathBox x = path_box(p, max(mine, 0), nboxes, A0, B0, se1, se2);
    const int ncols = mine >= 0 ? x.jh - x.jl + 1 : 1, nrows = mine >= 0 ? x.i1 - x.i0 - 1 : 0;
    const int lanes = (nrows + R - 1) / R, pad = lanes * R - nrows;
    const int nsteps = __reduce_max_sync(kFull, ncols + lanes - 1);
    const int row_quads = R * W / 2;  // int4 words of one step: rows 0, 1 of every lane, then rows 2, 3
    int4* const cells = reinterpret_cast<int4*>(p.cells) + seg * row_quads * (width + W);
    const int* const smat = X.smat();
    int4* const ring = reinterpret_cast<int4*>(X.region()) + lane;  // slot q: [64 q] and [64 q + 32]
    int8_t* const own = reinterpret_cast<int8_t*>(X.region() + kPathRingWords) +
                        (mine >= 0 ? seg : 0) * path_edge_bytes(width, W);
    int2* const edge = reinterpret_cast<int2*>(own);
    // Residues of columns jl - 1 .. jh, with 2 W more on either side.
    int8_t* const codes = own + 8 * width + 2 * W;
    const bool on = sl < lanes;
    int hl[R], fp[R], mrow[R];
    int diag = kPathLow, hout = kPathLow, eout = kPathLow;

    // Forward: lane row r is node row i0 + 1 + r - pad, which consumes residue i0 + r - pad.
    __syncwarp();
    if (nrows > 0) {
        const int2* top = p.fwd + (x.i0 == A0 ? 0 : (size_t)(x.i0 / p.every - 1) * p.stride);
        for (int c = sl; c < ncols; c += W) {
            int2 v = make_int2(x.i0 == A0 && x.jl + c == B0 ? 0 : kPathLow, kPathLow);
            if (x.i0 != A0 && x.jl + c >= 1) v = __ldcg(top + x.jl + c);
            edge[c] = v;
        }
        for (int c = sl - 2 * W; c < width + 2 * W; c += W)
            codes[c] = c >= 0 && c <= ncols && x.jl - 1 + c >= 0 ? (int8_t)ldres<NC>(s2 + x.jl - 1 + c) : (int8_t)0;
    }
    __syncwarp();
    const int own_pad = sl == 0 ? pad : 0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        mrow[k] = 32 * ldres<NC>(s1 + max(0, min(x.i0 + R * sl + k - pad, n - 1)));
        hl[k] = fp[k] = kPathLow;
    }
    int res = codes[-sl];  // of step t: codes[t - sl]
    int4* out = cells + sl;
    for (int t = 0; t < nsteps; ++t, out += row_quads) {
        int hin = __shfl_up_sync(kFull, hout, 1, W);
        int e = __shfl_up_sync(kFull, eout, 1, W);
        const int2 above = edge[min(t, ncols - 1)];
        if (sl == 0) {
            hin = above.x;
            e = __viaddmax_s32(above.y, -ge, above.x - goe);
        }
        const int b = res;
        res = codes[t + 1 - sl];
        if ((unsigned)(t - sl) < (unsigned)ncols && on) {
            int d = diag, hup = hin, v[2 * R];
#pragma unroll
            for (int k = 0; k < R; ++k) {
                int h = __vimax3_s32(e, fp[k], d + smat[mrow[k] + b]);
                const int g = h - goe;
                const bool real = k >= own_pad;
                v[2 * k + 1] = e;
                fp[k] = __viaddmax_s32(fp[k], -ge, g);
                const int en = __viaddmax_s32(e, -ge, g);
                e = real ? en : e;
                h = real ? h : hup;
                d = hl[k];
                hl[k] = hup = h;
                v[2 * k] = h;
            }
            diag = hin;
            hout = hup;
            eout = e;
            __stcg(out, make_int4(v[0], v[1], v[2], v[3]));
            __stcg(out + W, make_int4(v[4], v[5], v[6], v[7]));
        }
    }

    // Reverse: lane row r is node row i1 - 1 - r, which consumes residue i1 - 1 - r.
    __syncwarp();
    if (nrows > 0) {
        const int2* bottom = p.rev + (x.i1 == se1 ? 0 : (size_t)(x.i1 / p.every - 1) * p.stride) + se2;
        for (int c = sl; c < ncols; c += W) {
            int2 v = make_int2(x.i1 == se1 && x.jl + c == se2 ? 0 : kPathLow, kPathLow);
            if (x.i1 != se1 && x.jl + c < se2) {
                v = __ldcg(bottom - (x.jl + c));
                v.x -= 1;
                v.y -= 1;
            }
            edge[c] = v;
        }
    }
    __syncwarp();
    int span[R];  // columns with a cell on an optimal path, from jl: first | last << 16; 0xffff: none
    unsigned kinds = 0;  // four bits per row
#pragma unroll
    for (int k = 0; k < R; ++k) {
        mrow[k] = 32 * ldres<NC>(s1 + max(x.i1 - 1 - (R * sl + k), 0));
        hl[k] = fp[k] = kPathLow;
        span[k] = 0xffff;
    }
    diag = hout = eout = kPathLow;
    const int8_t* const back = codes + ncols + sl;  // residue of step t: back[-t]
    res = back[0];
    // Column jh - (t - sl) of forward lane lanes - 1 - sl: step ncols - 1 - (t - sl) + that lane's delay.
    const int4* in = cells + (size_t)(on ? ncols + lanes - 2 : 0) * row_quads + (on ? lanes - 1 - sl : 0);
    // Step t's words go to slot t % kPathRing; every step starts one copy
    // (maybe of nothing), so step t's has landed when all but the last
    // kPathRing - 1 have.
    auto fetch = [&](int t) {
        if ((unsigned)(t - sl) < (unsigned)ncols && on) {
            int4* slot = ring + 64 * (t & (kPathRing - 1));
            const int4* from = in - (ptrdiff_t)t * row_quads;
            copy_async16(slot, from);
            copy_async16(slot + 32, from + W);
        }
        copy_async_commit();
    };
#pragma unroll
    for (int t = 0; t < kPathRing - 1; ++t) fetch(t);
    for (int t = 0; t < nsteps; ++t) {
        int hin = __shfl_up_sync(kFull, hout, 1, W);
        int e = __shfl_up_sync(kFull, eout, 1, W);
        const int2 below = edge[max(ncols - 1 - t, 0)];
        if (sl == 0) {
            hin = below.x;
            e = __viaddmax_s32(below.y, -ge, below.x - goe);
        }
        const int b = res;
        res = back[-t - 1];
        const int c = t - sl;
        fetch(t + kPathRing - 1);
        copy_async_wait<kPathRing - 1>();
        if ((unsigned)c < (unsigned)ncols && on) {
            const int4 nlo = ring[64 * (t & (kPathRing - 1))], nhi = ring[64 * (t & (kPathRing - 1)) + 32];
            const int fh[R] = {nhi.z, nhi.x, nlo.z, nlo.x}, fe[R] = {nhi.w, nhi.y, nlo.w, nlo.y};
            int d = diag;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int f = fp[k];
                const int h = __vimax3_s32(e, f, d + smat[mrow[k] + b]);
                const int g = h - goe;
                d = hl[k];
                hl[k] = h;
                const int vh = fh[k] + h, vd = fe[k] + e + go;
                if (max(vh, vd) == best && R * sl + k < nrows) {
                    const int col = ncols - 1 - c;
                    span[k] = col | (span[k] == 0xffff ? col << 16 : span[k] & 0xffff0000);
                    kinds |= ((vh == best ? kPathH : 0) | (vd == best ? kPathD : 0)) << (4 * k);
                }
                fp[k] = __viaddmax_s32(f, -ge, g);
                e = __viaddmax_s32(e, -ge, g);
            }
            diag = hin;
            hout = hl[R - 1];
            eout = e;
        }
    }
    bool ok = true;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int r = R * sl + k;
        if (r >= nrows) continue;
        const int lo = span[k] & 0xffff, hi = (int)((unsigned)span[k] >> 16);
        ok = ok && lo != 0xffff;
        band[x.i1 - 1 - r - A0] =
            path_entry(lo + x.jl - B0, hi + x.jl - B0, (kinds >> (4 * k)) & 15);
    }
    __syncwarp();
    return __all_sync(kFull, ok);
}

__device__ __forceinline__ int path_box_count(const PathMem& p, int A0, int se1) {
    return (se1 - 1) / p.every - A0 / p.every + 1;
}

// The entries of the saved rows, and the box's own first and last row; warp w
// of nw. One warp follows the columns down; several start every row at the
// box's first. near: the columns near the optimum, added up over the warp's rows.
// False if a row has no cell on an optimal path.
__device__ inline bool path_rows(const PathMem& p, int2* band, int A0, int B0, int se1, int se2, int best, int go, int w,
                                 int nw, int& near) {
    near = 0;
    const int lane = threadIdx.x & 31;
    if (lane == 0 && w == 0) {
        band[0] = path_entry(0, 0, kPathH);
        band[se1 - A0] = path_entry(se2 - B0, se2 - B0, kPathH);
    }
    const int base = A0 / p.every, nboxes = path_box_count(p, A0, se1);
    for (int b = w, jl = B0; b + 1 < nboxes; b += nw) {
        const int i = (base + b + 1) * p.every;
        int lo, hi, kinds, near_lo, near_hi;
        if (nw > 1) jl = B0;
        if (!path_row(p, i, jl, se2, best, go, lo, hi, kinds, near_lo, near_hi)) return false;
        near += near_hi - near_lo + 1;
        if (lane == 0) {
            band[i - A0] = path_entry(lo - B0, hi - B0, kinds);
            p.span[b] = make_int4(lo, hi, near_lo, near_hi);
        }
    }
    __syncwarp();
    return true;
}

constexpr int kMinPathRows = 64;  // of a box

// Whether the rest of the path costs less than diff()'s divisions of the box, by
// the saved rows: the boxes and the walk's asks grow with the columns of paths
// within gapOpen, the divisions only with the box. Measured per pair (k cycles of
// a warp, path against divisions): related 1523-residue proteins, near columns
// 2 % of the box's, 2,960 against 10,200; unrelated ones of 400 residues (80 %)
// 2,150 against 1,300, of 1000 (64 %) 3,940 against 3,930, of 1500 (54 %) 9,800
// against 10,100. The line at a quarter of the columns takes the cheaper of the
// two to within 3 % of always taking it on related proteins and DNA of 300 to
// 1523 residues, 8 % on unrelated ones. Boxes of fewer than 64 rows have too
// little to divide (unrelated sequences of 30 to 2000 residues, most boxes that
// small: within 3 % of the cheaper with this line, 8 % without).
// A launch of few pairs, a CTA each, ends with its slowest pair, and there the
// walk's asks are a chain while the divisions are shared by the warps: the line
// is at a sixteenth (k cycles of 8 warps, path against divisions: 425 rows with 10
// % of the columns near 1,066 against 709, 540 rows with 14 % 1,194 against 971; of 16
// warps 2,741 rows with 20 % 5,270 against 3,900, 2,907 with 9 % 2,730 against 3,930), and
// from 1250 rows on, where the divisions outgrow the asks, at that many times
// more (one pair of unrelated sequences of 30000 193 ms against 237).
template <int SHARE>
__device__ __forceinline__ bool path_pays(int near, int every, int rows, int cols) {
    const long long columns = (long long)SHARE * every * near, box = (long long)rows * cols;
    return columns <= box || (SHARE == 16 && 1250 * columns <= box * rows);
}

// The entries of the rows between them; warp w of nw, boxes dealt in runs of
// as many as a warp takes at a time. False if some row has no cell on an
// optimal path, or (one warp) the boxes cost more than they save.
template <bool NC, bool CTA>
__device__ __noinline__ bool path_fill(const int8_t* s1, int n, const int8_t* s2, const PathMem& mem, int2* band, int A0,
                                       int B0, int se1, int se2, int best, int go, int ge, const Env& env, int w,
                                       int nw) {
    if (!CTA) w = 0, nw = 1;
    const Env X = env;  // copies stay in registers across the stores below
    const PathMem p = mem;
    const int lane = threadIdx.x & 31;
    const int nboxes = path_box_count(p, A0, se1);
    // A column of boxes costs about five steps of a sweep; mm_align's steps are
    // about a 96th of the pair's box, and a few per row for the small frames.
    // (A CTA's warps share the boxes, but not the small frames' divisions.)
    const int W = p.every / kPathRows, seg = lane / W, run = nw > 1 ? 32 / W : nboxes;
    int left = nw > 1 ? INT_MAX : (int)min((long long)(se1 - A0) * (se2 - B0) / 384 + (se1 - A0), (long long)INT_MAX);
    for (int first = w * run; first < nboxes; first += nw * run) {
        const int stop = min(first + run, nboxes);
        for (int b = first; b < stop;) {
            // As many boxes as the slice and the shared edge rows hold.
            int used = 0, width = 0, mine = -1;
            while (used * W < 32 && b + used < stop) {
                const PathBox x = path_box(p, b + used, nboxes, A0, B0, se1, se2);
                const int wide = max(width, x.jh - x.jl + 1);
                if (!path_fits(p, used + 1, wide, W, X.K)) break;
                if (seg == used) mine = b + used;
                width = wide;
                ++used;
            }
            if (nw == 1) left -= width + W;
            if (left < 0) return false;
            if (used == 0) {
                const PathBox x = path_box(p, b, nboxes, A0, B0, se1, se2);
                for (int i = x.i0 + 1 + lane; i < x.i1; i += 32) band[i - A0] = path_entry(0, 0, 0);
                ++b;
                continue;
            }
            if (!path_boxes<NC>(s1, n, s2, p, band, A0, B0, se1, se2, mine, width, nboxes, best, go, ge, X)) return false;
            b += used;
        }
    }
    __syncwarp();
    return true;
}

// The walk's rows of diff()'s halves, at the end of the warp's region: of a lane
// kPathLaneCols columns (enough if two rows in succession never span more), or
// of the whole warp kPathWarpCols; column j at j modulo that.
constexpr int kPathLaneCols = 8;
constexpr int kPathWarpCols = 32 * kPathLaneCols;
constexpr int kPathRowBytes = 2 * kPathWarpCols * (int)sizeof(int2);  // of a warp, both halves
struct PathRow {
    int2* at;  // of this lane
    __device__ __forceinline__ int2& operator[](int j) const { return at[(j & (kPathLaneCols - 1)) * 32]; }
};

// One lane: diff()'s two halves of frame (A, B, M, N) at row r = A + M / 2 over
// the rows' column ranges, and its midpoint scans (:570-593). All coordinates
// are relative to the box; s1/s2 point at its first residues. Cells outside the
// ranges are on no optimal path and only ever lose to those inside.
template <bool NC>
__device__ void path_midpoint(const int8_t* s1, const int8_t* s2, const int2* band, const PathRow F, const PathRow Rv,
                              int A, int B, int M, int N, int tb, int te, int go, int ge, const Env& X, int& midj,
                              bool& type2) {
    const int goe = go + ge, r = A + M / 2;
    // forward half, from the last single row above r
    int q = r - 1;
    while (q > A && !path_single(band[q])) --q;
    int lo, hi;
    if (q > A) {
        lo = hi = path_lo(band[q]);
        F[lo] = make_int2(0, -go);
    } else {
        q = A;
        lo = B;
        hi = min(path_hi(band[A]), B + N);
        F[B] = make_int2(0, -tb);
        for (int j = B + 1; j <= hi; ++j) F[j] = make_int2(-tb - ge * (j - B), -tb - ge * (j - B) - go);
    }
    const int first = lo;
    for (; q < r; ++q) {
        const int2 v = band[q + 1];
        const int nlo = max(path_lo(v), first), nhi = min(path_hi(v), B + N);
        const int* row = X.smat() + 32 * ldres<NC>(s1 + q);
        int diag = nlo - 1 >= lo && nlo - 1 <= hi ? F[nlo - 1].x : kPathLow;
        int f = kPathLow;
        for (int j = nlo; j <= nhi; ++j) {
            const int2 up = j >= lo && j <= hi ? F[j] : make_int2(kPathLow, kPathLow);
            const int e = __viaddmax_s32(up.y, -ge, up.x - goe);
            const int s = j > 0 ? row[ldres<NC>(s2 + j - 1)] : kPadScore;
            const int h = __vimax3_s32(e, f, diag + s);
            f = __viaddmax_s32(f, -ge, h - goe);
            diag = up.x;
            F[j] = make_int2(h, e);
        }
        lo = nlo;
        hi = nhi;
    }
    const int flo = lo, fhi = hi;
    // reverse half, from the first single row below r
    q = r + 1;
    while (q < A + M && !path_single(band[q])) ++q;
    if (q < A + M) {
        lo = hi = path_lo(band[q]);
        Rv[lo] = make_int2(0, -go);
    } else {
        q = A + M;
        hi = B + N;
        lo = max(path_lo(band[q]), B);
        Rv[hi] = make_int2(0, -te);
        for (int j = hi - 1; j >= lo; --j) Rv[j] = make_int2(-te - ge * (hi - j), -te - ge * (hi - j) - go);
    }
    const int lastc = hi;
    for (; q > r; --q) {
        const int2 v = band[q - 1];
        const int nlo = max(path_lo(v), B), nhi = min(path_hi(v), lastc);
        const int* row = X.smat() + 32 * ldres<NC>(s1 + q - 1);
        int diag = nhi + 1 >= lo && nhi + 1 <= hi ? Rv[nhi + 1].x : kPathLow;
        int f = kPathLow;
        for (int j = nhi; j >= nlo; --j) {
            const int2 dn = j >= lo && j <= hi ? Rv[j] : make_int2(kPathLow, kPathLow);
            const int e = __viaddmax_s32(dn.y, -ge, dn.x - goe);
            const int h = __vimax3_s32(e, f, diag + row[ldres<NC>(s2 + j)]);
            f = __viaddmax_s32(f, -ge, h - goe);
            diag = dn.x;
            Rv[j] = make_int2(h, e);
        }
        lo = nlo;
        hi = nhi;
    }
    lo = max(lo, flo);
    hi = min(hi, fhi);
    int midh = INT_MIN;
    midj = lo;
    type2 = false;
    for (int j = lo; j <= hi; ++j) {
        const int2 a = F[j], b = Rv[j];
        const int hh = a.x + b.x;
        if (hh >= midh && (hh > midh || (a.x != a.y && b.x == b.y))) {
            midh = hh;
            midj = j;
        }
    }
    for (int j = hi; j >= lo; --j) {
        const int hh = F[j].y + Rv[j].y + go;
        if (hh > midh) {
            midh = hh;
            midj = j;
            type2 = true;
        }
    }
    midj -= B;
}

// Whether a tight row lies strictly inside rows A .. A + M of the box.
__device__ __forceinline__ bool path_tight(const int2* band, int A, int M, int A0, int every) {
    for (int i = ((A0 + A) / every + 1) * every - A0; i < A + M; i += every)
        if (band[i].y & kPathTight) return true;
    return false;
}

// The free corner (r, c) of frame f (absolute rows and columns; end: its last,
// else its first), the saved row i (or the pair's own edge) the rows there are
// computed from, and the farthest column they are computed over.
struct PathCorner {
    int r, c, i, far;
    bool edge, loose;
};

__device__ __forceinline__ PathCorner path_corner(const PathMem& p, int4 f, bool end, int A0, int B0, int se1, int se2) {
    PathCorner x;
    x.r = end ? f.x + f.z : f.x;
    x.c = end ? f.y + (f.w & ((1 << 29) - 1)) : f.y;
    x.i = end ? max(A0, (x.r - 1) / p.every * p.every) : min(se1, (x.r / p.every + 1) * p.every);
    x.edge = end ? x.i == A0 : x.i == se1;
    const int4 span = x.edge ? make_int4(0, 0, B0, se2) : p.span[x.i / p.every - A0 / p.every - 1];
    // The frame's other corner may be the pair's own, where diff() opens gaps
    // free as well: a path may then run along the box's edge before it reaches
    // the saved row, in any column, which is no better than ending (starting)
    // where it does, at reversePass's -1 (forwardPass's 0).
    x.loose = end ? f.x == A0 && !((f.w >> 29) & 1) : f.x + f.z == se1 && !((f.w >> 30) & 1);
    x.far = x.loose ? (end ? B0 : se2) : (end ? span.z : span.w);
    return x;
}

// Whether mm_align divides frame f in fewer steps than path_ask takes to tell
// that it need not: each level takes its columns and some 40 steps, down to the
// frames one lane does; a quarter of the corner's columns, of 1.5 steps each.
// (Asked for all frames, pairs of weak alignments of 1600 residues spent 20 of
// 47 million cycles there: paths within gapOpen are a thousand columns apart.)
__device__ __forceinline__ bool path_ask_dear(const PathMem& p, int4 f, bool end, int A0, int B0, int se1, int se2) {
    const PathCorner x = path_corner(p, f, end, A0, B0, se1, se2);
    const int levels = 32 - __clz(f.z >> 5);
    return 3 * (abs(x.far - x.c) + 8) / 8 > ((f.w & ((1 << 29) - 1)) + 40) * levels + 20;
}

// Up to 32 / (p.every / 4) of the last frames asked for, a segment of lanes each
// like the boxes': those whose free corner no horizontal gap can use go to the
// stack, the others to the list. For a frame that starts at its free corner
// (r, c): the rows between the next saved row and r, over the columns from c to
// the last a path within gapOpen of the optimum crosses that row in; the gap
// can be used if the best value right of c, less its extension, reaches the
// corner's own. A frame that ends at its free corner: the same mirrored, from
// the saved row above. Lane row t is t + 1 rows from the saved row.
template <bool NC>
__device__ void path_ask(const int8_t* s1, int n, const int8_t* s2, int m, const PathMem& p, int A0, int B0, int se1,
                         int se2, int go, int ge, const Env& X, int4* stack, int& sp, int& nlist, int& nask,
                         bool keep) {
    constexpr int R = kPathRows;
    const int lane = threadIdx.x & 31, W = p.every / R, seg = lane / W, sl = lane & (W - 1);
    const int goe = go + ge;
    const int* const smat = X.smat();
    const int take = min(32 / W, nask);
    int4 f = p.list[p.list_cap - nask + min(seg, take - 1)];
    const bool end = (f.z >> 30) & 1;
    f.z &= (1 << 30) - 1;
    const int dir = end ? -1 : 1;  // from the corner to the saved row
    const PathCorner at = path_corner(p, f, end, A0, B0, se1, se2);
    const int r = at.r, c = at.c, i = at.i, far = at.far;
    const bool corner = at.edge, loose = at.loose;
    const int floor = !loose ? 2 * kPathLow : end ? 0 : -1;
    const int nrows = dir * (i - r), ncols = dir * (far - c) + 1, lanes = (nrows + R - 1) / R;
    const int nsteps = __reduce_max_sync(kFull, seg < take ? ncols + lanes - 1 : 0);
    const bool on = seg < take && sl < lanes;
    const int2* saved = corner ? p.fwd : (end ? p.fwd : p.rev + se2) + (size_t)(i / p.every - 1) * p.stride;
    int hl[R], fp[R], mrow[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        // Lane row t lies across residue i - 1 - t (below the corner's row: i + t).
        const int at = end ? i + R * sl + k : i - 1 - (R * sl + k);
        mrow[k] = 32 * ldres<NC>(s1 + max(0, min(at, n - 1)));
        hl[k] = fp[k] = kPathLow;
    }
    int diag = kPathLow, hout = kPathLow, eout = kPathLow, v = kPathLow;
    bool bad = false;
    for (int t = 0; t < nsteps; ++t) {
        int hin = __shfl_up_sync(kFull, hout, 1, W);
        int e = __shfl_up_sync(kFull, eout, 1, W);
        const int q = t - sl, j = far - dir * q;  // node column
        const bool in = (unsigned)q < (unsigned)ncols && on;
        if (in) {
            if (sl == 0) {
                int2 a = make_int2(kPathLow, kPathLow);
                if (corner) {
                    if (q == 0) a.x = 0;
                } else if (end ? j >= 1 : j < se2) {
                    a = __ldcg(end ? saved + j : saved - j);
                    if (!end) a = make_int2(a.x - 1, a.y - 1);
                }
                hin = max(a.x, floor);
                e = __viaddmax_s32(a.y, -ge, hin - goe);
            }
            const int b = ldres<NC>(s2 + max(0, min(end ? j - 1 : j, m - 1)));
            int d = diag;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int before = hl[k];
                const int h = max(__vimax3_s32(e, fp[k], d + smat[mrow[k] + b]), floor);
                const int g = h - goe;
                if (R * sl + k == nrows - 1) {
                    v = max(v, before) - ge;
                    if (q == ncols - 1) bad = v >= max(e + go, h);
                }
                d = before;
                hl[k] = h;
                fp[k] = __viaddmax_s32(fp[k], -ge, g);
                e = __viaddmax_s32(e, -ge, g);
            }
            diag = hin;
            hout = hl[R - 1];
            eout = e;
        }
    }
    const unsigned hits = __ballot_sync(kFull, bad);
    const bool head = sl == 0 && seg < take, listed = (hits >> (seg * W)) & (W == 32 ? kFull : (1u << W) - 1);
    const unsigned below = (1u << lane) - 1;
    const unsigned to_stack = __ballot_sync(kFull, head && !listed), to_list = __ballot_sync(kFull, head && listed);
    if (head && !listed) stack[sp + __popc(to_stack & below)] = make_int4(f.x - A0, f.y - B0, f.z, f.w);
    if (head && listed && keep) p.list[nlist + __popc(to_list & below)] = f;
    sp += __popc(to_stack);
    if (keep) nlist += __popc(to_list);
    nask -= take;
    __syncwarp();
}

// What one lane's halves of frame (A, M) would visit: 0 at most `most` cells,
// two rows in succession never over more than kPathLaneCols columns; 1 more; 2
// a row of a box left out.
__device__ inline int path_extent(const int2* band, int A, int M, int most) {
    const int r = A + M / 2;
    const int2 mid = band[r];
    int cells = path_hi(mid) - path_lo(mid) + 1, span = cells;
    if (mid.y == 0) return 2;
    for (int dir = -1; dir <= 1; dir += 2) {
        int2 last = mid;
        const int end = dir < 0 ? A : A + M;
        for (int q = r + dir;; q += dir) {
            const int2 v = band[q];
            if (v.y == 0) return 2;
            span = max(span, dir < 0 ? path_hi(last) - path_lo(v) + 1 : path_hi(v) - path_lo(last) + 1);
            cells += path_hi(v) - path_lo(v) + 1;
            if (cells > most || span > kPathLaneCols) return 1;
            if (q == end || path_single(v)) break;
            last = v;
        }
    }
    return 0;
}

// The same frame's midpoint by the whole warp, a row of up to 32 columns at a
// time: the gap along a row is a prefix maximum over the lanes. Returns 2 * midj
// + (type 2), or -1 if a row of a box left out is in the way, or mm_align's
// steps cost less (a row or 32 columns here about as much as three cells of the
// frame there). A lane alone spent 150 to 300 cycles per cell on frames this
// wide, the warp 250 per row. A call of its own: inlined it took registers from
// the walk (200 x 1523: 52.1 against 51.4 ms).
template <bool NC>
__device__ __noinline__ int path_midpoint_warp(const int8_t* s1, const int8_t* s2, const int2* band, int2* rows, int A,
                                               int B, int M, int N, int tb, int te, int go, int ge, int nw,
                                               const int* smat) {
    const int lane = threadIdx.x & 31, r = A + M / 2, goe = go + ge;
    const int2 mid = band[r];
    // Both ways to the nearest single row, or the frame's end.
    int start[2], cells = 0, span = path_hi(mid) - path_lo(mid) + 1, unknown = mid.y == 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int dir = h ? 1 : -1, end = h ? A + M : A;
        for (int q0 = r + dir;; q0 += 32 * dir) {
            const int q = q0 + dir * lane;
            const bool in = h ? q <= end : q >= end;
            const int2 v = in ? band[q] : make_int2(0, 0), last = in ? band[q - dir] : v;
            const unsigned stops = __ballot_sync(kFull, in && (q == end || path_single(v)));
            if (in && lane <= __ffs(stops) - 1u) {
                unknown |= v.y == 0;
                span = max(span, h ? path_hi(v) - path_lo(last) + 1 : path_hi(last) - path_lo(v) + 1);
                cells += path_hi(v) - path_lo(v) + 1;
            }
            if (stops) {
                start[h] = q0 + dir * (__ffs(stops) - 1);
                break;
            }
        }
    }
    span = __reduce_max_sync(kFull, span);
    cells = __reduce_add_sync(kFull, cells);
    if (__any_sync(kFull, unknown) || span > kPathWarpCols ||
        cells + 32ll * (start[1] - start[0]) > (long long)M * N / (3 * nw) + 2000)
        return -1;

    int lo[2], hi[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int dir = h ? -1 : 1;  // from the start row to r
        const int open = h ? te : tb;
        int2* const row = rows + h * kPathWarpCols;  // column j at [j & (kPathWarpCols - 1)]
        int q = start[h];
        const int2 v0 = band[q];
        const bool edge = q == (h ? A + M : A);
        // Columns from..to of the row so far, in the half's own direction.
        const int c0 = !edge ? path_lo(v0) : h ? B + N : B;
        int from = c0, to = c0;
        if (edge) to = h ? max(path_lo(v0), B) : min(path_hi(v0), B + N);
        __syncwarp();
        for (int k = lane; k <= dir * (to - from); k += 32) {
            const int left = edge ? -open - ge * k : 0;
            row[(from + dir * k) & (kPathWarpCols - 1)] =
                k ? make_int2(left, left - go) : make_int2(0, edge ? -open : -go);
        }
        __syncwarp();
        int2 v32 = make_int2(0, 0);
        int res32 = 0;
        for (int k = 0; q != r; ++k, q += dir) {
            if ((k & 31) == 0) {  // the next 32 rows' entries and residues
                const int qq = q + dir * lane;
                const bool in = h ? qq > r : qq < r;
                v32 = in ? band[qq + dir] : make_int2(0, 0);
                res32 = in ? (int)ldres<NC>(s1 + (h ? qq - 1 : qq)) : 0;
            }
            const int ends = __shfl_sync(kFull, v32.x, k & 31);
            const int* const sub = smat + 32 * __shfl_sync(kFull, res32, k & 31);
            const int2 v = make_int2(ends, 0);
            const int nfrom = h ? min(path_hi(v), c0) : max(path_lo(v), c0);
            const int nto = h ? max(path_lo(v), B) : min(path_hi(v), B + N);
            int carry = kPathLow, behind = kPathLow;  // the gap along the row, H above the column before
            for (int t = 0; t <= dir * (nto - nfrom); t += 32) {
                const int j = nfrom + dir * (t + lane);
                const bool in = dir * (nto - j) >= 0;
                const bool above = dir * (j - from) >= 0 && dir * (to - j) >= 0;
                const int2 up = above ? row[j & (kPathWarpCols - 1)] : make_int2(kPathLow, kPathLow);
                int diag = __shfl_up_sync(kFull, up.x, 1);
                if (lane == 0) {
                    const int jb = j - dir;
                    diag = t ? behind
                             : (dir * (jb - from) >= 0 && dir * (to - jb) >= 0 ? row[jb & (kPathWarpCols - 1)].x : kPathLow);
                }
                behind = __shfl_sync(kFull, up.x, 31);
                const int e = __viaddmax_s32(up.y, -ge, up.x - goe);
                const int jr = h ? j : j - 1;  // the column's residue
                const int sc = in && jr >= 0 ? sub[ldres<NC>(s2 + jr)] : kPadScore;
                const int he = max(e, diag + sc);
                int best = in ? he - goe : kPathLow;  // of a gap from a column up to here, at the next
                const int count = min(32, dir * (nto - nfrom) + 1 - t);
                for (int d = 1; d < count; d *= 2) {
                    const int o = __shfl_up_sync(kFull, best, d);
                    if (lane >= d) best = max(best, o - ge * d);
                }
                int f = __shfl_up_sync(kFull, best, 1);
                f = lane ? max(f, carry - ge * lane) : carry;
                carry = max(__shfl_sync(kFull, best, 31), carry - ge * 32);
                __syncwarp();  // every lane has read the row above
                if (in) row[j & (kPathWarpCols - 1)] = make_int2(max(he, f), e);
            }
            __syncwarp();
            from = nfrom;
            to = nto;
        }
        lo[h] = h ? to : from;
        hi[h] = h ? from : to;
    }
    // Type 1: the last of the best columns that has (F.x != F.y, R.x == R.y),
    // else the first; type 2, if better: the last.
    const int l = max(lo[0], lo[1]), u = min(hi[0], hi[1]);
    int h1 = INT_MIN, first = INT_MAX, tied = -1, h2 = INT_MIN, at2 = -1;
    for (int j = l + lane; j <= u; j += 32) {
        const int2 a = rows[j & (kPathWarpCols - 1)], b = rows[kPathWarpCols + (j & (kPathWarpCols - 1))];
        const int hh = a.x + b.x, vv = a.y + b.y + go;
        const bool keep = a.x != a.y && b.x == b.y;
        if (hh > h1) {
            h1 = hh;
            first = j;
            tied = keep ? j : -1;
        } else if (hh == h1 && keep) {
            tied = j;
        }
        if (vv >= h2) {
            h2 = vv;
            at2 = j;
        }
    }
    const int b1 = __reduce_max_sync(kFull, h1), b2 = __reduce_max_sync(kFull, h2);
    first = __reduce_min_sync(kFull, h1 == b1 ? first : INT_MAX);
    tied = __reduce_max_sync(kFull, h1 == b1 ? tied : -1);
    at2 = __reduce_max_sync(kFull, h2 == b2 ? at2 : -1);
    __syncwarp();
    return 2 * ((b2 > b1 ? at2 : tied >= 0 ? tied : first) - B) + (b2 > b1);
}

// Walks diff()'s frames from the box's own, 32 at a time. Adds identities,
// matches and inner-loop iterations; frames left to mm_align go to p.list
// (count returned). With nw warps (w: this one's number) all walk the first
// levels, which only warp 0 accounts for, and then a share of the frames each.
template <bool NC, bool CTA>
__device__ __noinline__ int path_walk(const int8_t* s1, int n, const int8_t* s2, int m, const PathMem& mem, const int2* band,
                                      int A0, int B0, int se1, int se2, int go, int ge, const Env& env,
                                      int& n_ident, int& n_match, long long& n_cells, int w, int nw) {
    if (!CTA) w = 0, nw = 1;
    const Env X = env;  // copies stay in registers across the stores below
    const PathMem p = mem;
    const int M0 = se1 - A0, N0 = se2 - B0;
    const int8_t* const seq1 = s1;
    const int8_t* const seq2 = s2;
    s1 += A0;
    s2 += B0;
    const int lane = threadIdx.x & 31;
    constexpr int NMASK = (1 << 29) - 1;
    int4* stack = reinterpret_cast<int4*>(X.region());
    const int cap = (warp_region_bytes(X.K) - kPathRowBytes) / (int)sizeof(int4);
    int2* const rows = reinterpret_cast<int2*>(stack + cap);
    bool dealt = nw == 1;  // this warp's frames are its own
    int ident = 0, match = 0, nlist = 0, nask = 0;
    long long cells = 0;
    __syncwarp();
    if (lane == 0) stack[0] = make_int4(0, 0, M0, N0);
    __syncwarp();
    int sp = 1;
    for (;;) {
        if (sp == 0 && nask == 0) break;
        // Not yet dealt out, stack and asks hold fewer than 4 * 16 frames: there is room for them.
        if (nask > 0 && (sp == 0 || !dealt)) {
            while (nask > 0 && sp + 32 < cap - 96)
                path_ask<NC>(seq1, n, seq2, m, p, A0, B0, se1, se2, go, ge, X, stack, sp, nlist, nask, dealt || w == 0);
            continue;
        }
        if (!dealt && sp >= 2 * nw) {  // every warp has the same frames: warp w keeps those at w, w + nw, ...
            int kept = 0;
            for (int k = w; k < sp; k += nw, ++kept) {
                const int4 f = stack[k];
                __syncwarp();
                if (lane == 0) stack[kept] = f;
                __syncwarp();
            }
            sp = kept;
            dealt = true;
            continue;
        }
        const bool mine = dealt || w == 0;
        // Taking t frames grows the stack by at most t, one at a time by at
        // most the depth of the recursion (17): near the stack's end fewer.
        const int take = max(1, min(min(32, sp), cap - 40 - sp));
        int4 fr = make_int4(0, 0, 0, 0);
        if (lane < take) fr = stack[sp - 1 - lane];
        sp -= take;
        __syncwarp();
        int4 kid[2];
        int kind[2] = {0, 0};  // 0: nothing to do, 1: to the stack, 2: to the list, 3: to ask for
        const int A = fr.x, B = fr.y, M = fr.z, N = fr.w & NMASK;
        const int tbf = (fr.w >> 29) & 1, tef = (fr.w >> 30) & 1;
        const int tb = tbf ? go : 0, te = tef ? go : 0;
        // Where the middle row leaves a choice: by 0 this lane, 1 the warp, 2 mm_align.
        const int midi = M / 2;
        int by = 3, midj = 0;
        bool type2 = false;
        if (lane < take && M > 1) {
            const int2 v = band[A + midi];
            const int kinds = v.y & (kPathH | kPathD);
            midj = path_lo(v) - B;
            type2 = kinds == kPathD;
            // The fewer frames there are, the sooner the whole warp is faster.
            if (kinds == 0 || kinds == (kPathH | kPathD) || path_lo(v) != path_hi(v))
                by = path_extent(band, A, M, 32 + 16 * take);
        }
        for (unsigned wide = __ballot_sync(kFull, by == 1); wide; wide &= wide - 1) {
            const int l = __ffs(wide) - 1;
            const int mid = path_midpoint_warp<NC>(
                s1, s2, band, rows, __shfl_sync(kFull, A, l), __shfl_sync(kFull, B, l), __shfl_sync(kFull, M, l),
                __shfl_sync(kFull, N, l), __shfl_sync(kFull, tb, l), __shfl_sync(kFull, te, l), go, ge, nw, X.smat());
            if (lane == l) {
                by = mid < 0 ? 2 : 3;
                midj = mid >> 1;
                type2 = mid & 1;
            }
        }
        if (lane < take && M == 1) {
            if (mine) cells += N;
            int midh = -(tb + ge) - (te + ge * N);
            const int hh0 = -(te + ge) - (tb + ge * N);
            midh = max(midh, hh0);
            const int2 u = band[A], v = band[A + 1];
            const int ra = ldres<NC>(s1 + A);
            const int* row = X.smat() + 32 * ra;
            int at = 0, rb = 0;
            const int j1 = min(N, min(path_hi(u) + 1, path_hi(v)) - B);
            for (int j = max(1, max(path_lo(u) + 1, path_lo(v)) - B); j <= j1; ++j) {
                const int b = ldres<NC>(s2 + B + j - 1);
                const int hh = row[b] - (N - j > 0 ? te + ge * (N - j) : 0) - (j - 1 > 0 ? tb + ge * (j - 1) : 0);
                if (hh > midh) {
                    midh = hh;
                    at = j;
                    rb = b;
                }
            }
            if (at > 0 && mine) {
                ++match;
                if (ra != X.gp1 && rb != X.gp2 && ra == rb) ++ident;
            }
        } else if (lane < take) {
            if (by == 2) {
                kid[0] = fr;
                kind[0] = 2;
            } else {
                if (mine) cells += (long long)M * N;
                if (by == 0)
                    path_midpoint<NC>(s1, s2, band, PathRow{rows + lane}, PathRow{rows + kPathWarpCols + lane}, A, B, M, N,
                                      tb, te, go, ge, X, midj, type2);
                if (!type2) {
                    kid[0] = make_int4(A + midi, B + midj, M - midi, (N - midj) | (1 << 29) | (tef << 30));
                    kid[1] = make_int4(A, B, midi, midj | (tbf << 29) | (1 << 30));
                } else {
                    kid[0] = make_int4(A + midi + 1, B + midj, M - midi - 1, (N - midj) | (tef << 30));
                    kid[1] = make_int4(A, B, midi - 1, midj | (tbf << 29));
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    if (kid[c].z > 0 && (kid[c].w & NMASK) > 0) kind[c] = 1;
                }
                if (type2) {
                    // Free openings inside the box: at kid 0's start and kid 1's end,
                    // and maybe already at their other corners.
                    if (kind[0])
                        kind[0] = tef == 0 && A + M < M0 && !path_tight(band, kid[0].x, kid[0].z, A0, p.every) ? 2 : 3;
                    if (kind[1])
                        kind[1] = tbf == 0 && A > 0 && !path_tight(band, kid[1].x, kid[1].z, A0, p.every) ? 2 : 3;
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int4 f = make_int4(kid[c].x + A0, kid[c].y + B0, kid[c].z, kid[c].w);
                        if (kind[c] == 3 && path_ask_dear(p, f, c == 1, A0, B0, se1, se2)) kind[c] = 2;
                    }
                }
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const unsigned below = (1u << lane) - 1;
            const unsigned on = __ballot_sync(kFull, kind[c] == 1), off = __ballot_sync(kFull, kind[c] == 2);
            const unsigned ask = __ballot_sync(kFull, kind[c] == 3);
            if (kind[c] == 1) stack[sp + __popc(on & below)] = kid[c];
            if (kind[c] == 2 && mine)
                p.list[nlist + __popc(off & below)] = make_int4(kid[c].x + A0, kid[c].y + B0, kid[c].z, kid[c].w);
            // Absolute rows and columns in both, the kid's number with the ones to ask for.
            if (kind[c] == 3)
                p.list[p.list_cap - 1 - nask - __popc(ask & below)] =
                    make_int4(kid[c].x + A0, kid[c].y + B0, kid[c].z | c << 30, kid[c].w);
            sp += __popc(on);
            if (mine) nlist += __popc(off);
            nask += __popc(ask);
        }
        __syncwarp();
    }
    n_ident += __reduce_add_sync(kFull, ident);
    n_match += __reduce_add_sync(kFull, match);
    for (int d = 16; d; d >>= 1) cells += __shfl_xor_sync(kFull, cells, d);
    n_cells += cells;
    return nlist;
}

}  // namespace cwgpu
