// bia_uv_walk.cuh -- the universal-variable step and the split learned step's rest pass over warp-blocks,
// shared by the single system (bia_step.cu) and the ensemble (bia_ensemble.cu).
//
// Nearly every pair of a short step is one of uv_fast_pair's.  A persistent grid of warps walks the
// warp-blocks and solves those pairs, branch-free, block by block.  The few others (a universal-variable
// Newton iteration; in the rest pass the pairs deferred to the heads too) would keep one or two lanes of
// a warp busy for several thousand cycles in every block, so a warp collects them over its blocks in a
// queue in shared memory and solves them 32 at a time, adding each onto its block's partial sums,
// which no other warp touches.  Blocks with many of them (a long step), and diagonal blocks, are finished on
// the spot.  Measured with one pass over the others at the end of every block instead: 4.31
// against 3.80 ms for the learned step of the 32768-body Plummer sphere, 8.7 against 6.2 ms for that of
// 4096 small ones.  With every pair taking uv_series and its composition in the walk: 5.70 and 8.87 ms.
//
// What bounds the walk: the register file's read ports and the FP64 pipe.  A pair takes about 77
// FP64 instructions (2 cycles each, 3 where a multiply-add reads three registers) and 75 others; at
// n = 16384 the FP64 pipe is 60 % and the issue slots 62 % busy, 263 cycles per 32 pairs and scheduler.
#pragma once
#include "bia_learned_block.cuh"
#include "bia_pair.cuh"
#include "bia_tiles.cuh"

namespace bia {

// The walk of the universal-variable and rest warp-blocks, in two passes.
//
// The first solves the short-step pairs (uv_fast_pair) at the rotation offsets in ascending k,
// the row sums in racc, the column sums in the slice (lane l adds into slot (l + k) mod 32, a
// different slot on every lane), and leaves a bit for every other pair (bit k of the returned
// mask).  Full off-diagonal blocks take two offsets a turn without a test of their particles: the
// branch-free pairs of two offsets interleave, where one pair's chain of dependent FP64 operations
// alone left the warp waiting.  A block more than a quarter of whose first kProbe offsets' pairs are
// others (a long step) leaves the rest of them to the second pass untried: 7.63 ms against 8.07 at
// a half and 7.63 at an eighth (learned, Coulomb, n = 16384, 1e-4), where half of the pairs are others.
//
// Out of line, on the dynamic shared memory of the kernel (the warp's slice begins `slice` doubles
// into it), so that the loop has the whole register budget whatever the kernel around it keeps:
// inlined in the ensemble's rest kernel it spilled, 8.1 against 5.6 ms on the 4096 Plummer systems.
constexpr int kProbe = 2;

struct UvRow {
    double s[6], cdt2;  // the lane's row; its coupling times dt^2 (and its charge)
    double dt;
};

// The relative state of a row and column slot src as uv_fast_pair takes it, velocities times dt: their difference
// first, so that a velocity common to the particles leaves no rounding.
__device__ __forceinline__ void walk_diff(const double *ws, int src, const UvRow &row, double r[3], double w[3])
{
    slice_diff(ws, src, row.s, r, w);
#pragma unroll
    for (int d = 0; d < 3; d++) w[d] = __dmul_rn(w[d], row.dt);
}

template <bool kQ>
static __device__ __noinline__ unsigned uv_walk_full(int slice, const UvRow row, int lane, double *racc_out)
{
    double *ws = warp_slices + slice;
    double racc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    unsigned left = 0u;
#pragma unroll 1
    for (int k = 0; k < 32; k += 2) {
        int src[2];
        double h[2][6];
        bool ok[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            src[u] = (lane + k + u) & 31;
            double r[3], w[3];
            walk_diff(ws, src[u], row, r, w);
            ok[u] = uv_fast_pair(kQ ? row.cdt2 * ws[6 * 32 + src[u]] : row.cdt2, r, w, h[u]);
        }
        if (!(ok[0] && ok[1])) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                left |= (ok[u] ? 0u : 1u) << (k + u);
#pragma unroll
                for (int c = 0; c < 6; c++) h[u][c] = ok[u] ? h[u][c] : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            slice_add(ws, src[u], h[u], racc);
            __syncwarp();  // slot src is the next offset's slot of lane - 1
        }
        if (k + 2 == kProbe && __reduce_add_sync(0xffffffffu, (unsigned)__popc(left)) > 32u * kProbe / 4u) {
            left |= 0xffffffffu << kProbe;
            break;
        }
    }
#pragma unroll
    for (int c = 0; c < 6; c++) racc_out[c] = racc[c];
    return left;
}

// the same over a diagonal or ragged block, one offset a turn
template <bool kQ>
static __device__ __noinline__ unsigned uv_walk_part(int slice, const UvRow row, int lane, bool diag, bool row_live,
                                                     int ncols, double *racc_out)
{
    double *ws = warp_slices + slice;
    double racc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    unsigned left = 0u;
    const int k0 = diag ? 1 : 0, k1 = diag ? 16 : 31;
#pragma unroll 1
    for (int k = k0; k <= k1; k++) {
        const int src = (lane + k) & 31;
        const bool active = (!diag || k < 16 || lane < 16) && row_live && src < ncols;
        double r[3], w[3], h[6];
        walk_diff(ws, src, row, r, w);
        const bool ok = uv_fast_pair(kQ ? row.cdt2 * ws[6 * 32 + src] : row.cdt2, r, w, h);
        left |= (active && !ok ? 1u : 0u) << k;
#pragma unroll
        for (int c = 0; c < 6; c++) h[c] = active && ok ? h[c] : 0.0;
        slice_add(ws, src, h, racc);
        __syncwarp();
    }
#pragma unroll
    for (int c = 0; c < 6; c++) racc_out[c] = racc[c];
    return left;
}

// The second pass: slow(src, k, h) gives h of the pairs in `left`, in ascending k on each lane.  Few
// of them: every lane takes its own next one each turn, so a turn solves a pair on as many lanes
// as have one left, and lanes that meet in a column add in lane order.  Many: the lanes walk the
// offsets together (distinct columns).  Which, depends on the block's pairs alone.  The line at half
// of the block's pairs: Plummer, n = 16384, a universal-variable step of 1e-3, 3.46 ms at a quarter,
// 3.40 at half, 3.56 at three quarters; the Coulomb cubes there differ by 1 %.  The universal-variable
// solve is in line in both loops: 2.80 against 3.56 ms out of line (Coulomb, 1e-4), 1.5 % slower
// where the walk leaves few pairs; the rest pass's pair, longer, is faster out of line (13.05
// against 13.65 ms for the learned step of 1e-3).
template <class Slow>
__device__ __forceinline__ void uv_walk_rest(unsigned left, double *ws, int lane, const double si[7], double racc[6],
                                             Slow &slow)
{
    const unsigned full = 0xffffffffu;
    const unsigned count = __reduce_add_sync(full, (unsigned)__popc(left));
    if (count <= 512u) {
        const unsigned lt = (1u << lane) - 1u;
        for (;;) {
            const bool busy = left != 0u;
            const unsigned bm = __ballot_sync(full, busy);
            if (bm == 0u) break;
            if (busy) {
                const int k = __ffs(left) - 1;
                left &= left - 1u;
                const int src = (lane + k) & 31;
                double h[6];
                slow(src, k, si, h);
                const unsigned grp = __match_any_sync(bm, src);
                const int rank = __popc(grp & lt);
                const int turns = (int)__reduce_max_sync(bm, (unsigned)__popc(grp));
                for (int t = 0; t < turns; t++) {
                    if (rank == t) slice_add(ws, src, h, racc);
                    __syncwarp(bm);
                }
            }
        }
    } else {
        for (unsigned any = __reduce_or_sync(full, left); any; any &= any - 1u) {
            const int k = __ffs(any) - 1;
            const int src = (lane + k) & 31;
            if ((left >> k) & 1u) {
                double h[6];
                slow(src, k, si, h);
                slice_add(ws, src, h, racc);
            }
            __syncwarp();
        }
    }
    __syncwarp();
}

// pairs of the lane in a block (the walk's offsets whose particles exist)
__device__ __forceinline__ int block_lane_pairs(int lane, int bi, int bj, int n)
{
    if (bi * 32 + lane >= n) return 0;
    const int ncols = n - bj * 32;
    if (bi != bj) return ncols >= 32 ? 32 : ncols;
    int c = 0;
    for (int k = 1; k <= 16; k++) c += ((k < 16 || lane < 16) && ((lane + k) & 31) < ncols) ? 1 : 0;
    return c;
}

// A system as the walk sees it: particles x..w[0, n) (charges q), coupling eps_th, and where its
// partial sums go (deterministic: part[m][6][plane]; atomic: one accumulator plane).
struct WalkSystem {
    const double *x, *y, *z, *u, *v, *w, *q;
    int n;
    double eps_th;
    double *part;
    size_t plane;
};

// A warp-block: its block row and column, its system, and its index for the finish kernel.
struct WalkBlock {
    int bi, bj, sys;
    unsigned int item;
};

// The queue of a warp: at most 32 pairs (block slot << 10 | k << 5 | lane of the pair) of at most 32
// blocks, behind the warp's column slice.
constexpr int kQueuePairs = 32;
constexpr int kQueueDoubles = kQueuePairs * (int)(sizeof(WalkBlock) + sizeof(unsigned int)) / (int)sizeof(double);
constexpr int kWalkSliceDoubles = kTileSmemDoubles + kQueueDoubles;
// the rest pass adds 1024 row slots for the head inputs of a block finished on the spot
template <bool kRest>
__host__ __device__ constexpr int walk_warp_doubles() { return kWalkSliceDoubles + (kRest ? 1024 * 4 / 8 : 0); }
template <bool kRest>
__host__ __device__ constexpr size_t walk_smem_bytes(int warps) { return (size_t)warps * walk_warp_doubles<kRest>() * sizeof(double); }

struct WalkCounts {
    int pairs, iters, over, nonfinite;  // universal-variable pairs, Newton iterations, not converged
};

// The warp's counts onto the context's counters.
__device__ __forceinline__ void walk_flush_counts(const WalkCounts &c, unsigned long long *stats, int lane)
{
    PairCounters p;
    counters_zero(p);
    p.cls[kUniversal] = c.pairs;
    p.it_uv = c.iters;
    p.nonconverged = c.over;
    p.nonfinite = c.nonfinite;
    flush_counters(p, stats, lane);
}

// A walk flushes its counts every this many blocks: 1024 pairs each, of at most kUvItMax + 1 iterations, stay
// below 2^31 summed over a warp.
constexpr int kWalkFlushBlocks = 8192;
static_assert(1024LL * (kUvItMax + 1) * kWalkFlushBlocks < 1LL << 31, "");

// One pair of the second kind: its displacement in h (uv: returns kLearnedPlain always), or its head and
// head input x01.  Counted in c unless deferred.
template <bool kRest>
__device__ __forceinline__ int walk_other_pair(double eps_ij, double dt, const double r[3], const double g[3],
                                               double h[6], uint32_t &x01, WalkCounts &c)
{
    double hs[6];
    int it = 0;
    if (kRest) {
        uint32_t x = 0u;
        const int kind = rest_pair(eps_ij, dt, r[0], r[1], r[2], g[0], g[1], g[2], hs, &x, &it);
        x01 = x;
        if (kind != kLearnedPlain) {
            c.pairs--;
#pragma unroll
            for (int k = 0; k < 6; k++) h[k] = 0.0;
            return kind;
        }
    } else {
        it = uv_halfdisp_fast(eps_ij, dt, r, g, hs);  // in line: see uv_walk_rest
    }
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 6; k++) {
        h[k] = hs[k];
        finite = finite && isfinite(hs[k]);
    }
    c.iters += it;
    c.over += it > kUvItMax ? 1 : 0;
    c.nonfinite += finite ? 0 : 1;
    return kLearnedPlain;
}

// Block sums onto the partials or accumulators: racc of row 32 bi + lane, -cacc of column 32 bj + lane.
template <bool kDeterministic>
__device__ __forceinline__ void walk_write(const WalkSystem &S, int bi, int bj, int lane, const double racc[6],
                                           const double cacc[6])
{
    if (kDeterministic) {
        write_partials(S.part, S.plane, bi, bj, lane, racc, cacc);
        return;
    }
    const int i = bi * 32 + lane, j = bj * 32 + lane;
#pragma unroll
    for (int c = 0; c < 6; c++) {
        if (bi == bj) {
            if (i < S.n) atomicAdd(&S.part[c * S.plane + i], racc[c] - cacc[c]);
        } else {
            if (i < S.n) atomicAdd(&S.part[c * S.plane + i], racc[c]);
            if (j < S.n) atomicAdd(&S.part[c * S.plane + j], -cacc[c]);
        }
    }
}

// The queue's pairs, one per lane (qn of them), onto their blocks' sums; the deferred ones (rest) into
// the heads' rows and the list, an entry for each of their blocks.  A block's pairs are all in one
// queue, in lane and then k order, and are added in that order whatever blocks share the queue, so the
// sums do not depend on how the blocks were dealt to the warps.
template <bool kDeterministic, bool kRest, class Items>
__device__ __forceinline__ void walk_queue(const Items &I, const LearnedRows &R, double dt, const unsigned int *queue,
                                           const WalkBlock *blocks, int qn, int lane, WalkCounts &c)
{
    const unsigned full = 0xffffffffu, lt = (1u << lane) - 1u;
    const bool act = lane < qn;
    int kind = -1, slot = 0, l = 0, k = 0, j = 0;
    uint32_t x01 = 0u;
    double h[6] = {0, 0, 0, 0, 0, 0};
    WalkBlock B{};
    WalkSystem S{};
    if (act) {
        const unsigned int e = queue[lane];
        slot = (int)(e >> 10);
        k = (int)((e >> 5) & 31u);
        l = (int)(e & 31u);
        j = (l + k) & 31;
        B = blocks[slot];
        S = I.system(B.sys);
        double si[7], sj[7], r[3], g[3];
        load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, B.bi * 32 + l, si);
        load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, B.bj * 32 + j, sj);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            r[d] = si[d] - sj[d];
            g[d] = si[3 + d] - sj[3 + d];
        }
        const double eps_ij = S.q ? S.eps_th * si[6] * sj[6] : S.eps_th;
        kind = walk_other_pair<kRest>(eps_ij, dt, r, g, h, x01, c);
    }
    const unsigned am = __ballot_sync(full, kind == kLearnedPlain);
    if (kind == kLearnedPlain) {
#pragma unroll
        for (int pass = 0; pass < 2; pass++) {  // the rows, then the columns
            const unsigned grp = __match_any_sync(am, (slot << 6) | (pass == 0 ? l : 32 | j));
            double sum[6] = {0, 0, 0, 0, 0, 0};
            for (unsigned m = grp; m; m &= m - 1u) {  // members in lane order (grp-uniform)
                const int src = __ffs(m) - 1;
#pragma unroll
                for (int d = 0; d < 6; d++) sum[d] += __shfl_sync(grp, h[d], src);
            }
            if (lane == 31 - __clz(grp)) {  // the group's last lane adds the sum once
                const int p = pass == 0 ? B.bi * 32 + l : B.bj * 32 + j;
                const size_t m0 = kDeterministic ? (size_t)(pass == 0 ? B.bj : B.bi) * 6 * S.plane : 0;
#pragma unroll
                for (int d = 0; d < 6; d++) {
                    double *dst = S.part + m0 + (size_t)d * S.plane + p;
                    const double v = pass == 0 ? sum[d] : -sum[d];
                    if (kDeterministic) *dst += v;
                    else atomicAdd(dst, v);
                }
            }
        }
    }
    if (kRest) {
        const unsigned he = __ballot_sync(full, kind == kLearnedEll), hh = __ballot_sync(full, kind == kLearnedHyp);
        const unsigned dm = he | hh;
        if (dm != 0u) {  // warp-uniform
            const bool mine = (dm >> lane) & 1u;
            const unsigned grp = mine ? __match_any_sync(dm, slot) : 0u;
            const bool lead = mine && (grp & lt) == 0u;
            const unsigned lm = __ballot_sync(full, lead);
            // rows of each head and list entries for the whole queue: one atomic each
            unsigned long long base = 0ull;
            if (lane == kHeadEll && he) base = atomicAdd(&R.counts[kHeadEll], (unsigned long long)__popc(he));
            if (lane == kHeadHyp && hh) base = atomicAdd(&R.counts[kHeadHyp], (unsigned long long)__popc(hh));
            if (lane == 2) base = atomicAdd(R.nlist, (unsigned int)__popc(lm));
            const unsigned long long be = __shfl_sync(full, base, kHeadEll), bh = __shfl_sync(full, base, kHeadHyp);
            const unsigned int e0 = (unsigned int)__shfl_sync(full, base, 2);
            const bool fits = (he == 0u || be + __popc(he) <= R.rows_cap) && (hh == 0u || bh + __popc(hh) <= R.rows_cap);
            if (mine) {
                const int hd = kind == kLearnedHyp ? kHeadHyp : kHeadEll;
                const unsigned int row = (unsigned int)(hd == kHeadHyp ? bh : be) + __popc((hd == kHeadHyp ? hh : he) & lt);
                if (fits) R.rows[hd][row] = x01;
                const unsigned int e = e0 + __popc(lm & ((1u << (__ffs(grp) - 1)) - 1u));
                R.pairs[(size_t)e * kBatchPairs + __popc(grp & lt)] =
                    make_uint2(fits ? row : kNoRows, (unsigned)l | ((unsigned)k << 5) | ((unsigned)hd << 10));
                if (lead) R.entries[e] = make_uint4(B.item, kNoRows, kNoRows, (unsigned)__popc(grp));
            }
        }
    }
    __syncwarp();
}

// Whether the short step may take a block's pairs: eps_ij dt^2 of every coupling that is not zero has to be a normal
// number (below, uv_fast_pair would lose bits of the interaction or all of it; an infinite one gives NaN, which it
// refuses), and so have its factors in that order.  cdt2: eps dt^2 times the lane's row charge qi; qj: the charge of
// its column.  The same on every lane.
__device__ __forceinline__ bool walk_coupling_normal(const WalkSystem &S, double dt2, double cdt2, double qi, double qj)
{
    constexpr int kOne = 1023 << 20, kLeast = (1023 - 960) << 20;  // 1 and 2^-960 as high words
    if (S.eps_th == 0.0) return true;
    const int e = __double2hiint(fabs(S.eps_th * dt2));
    if (!S.q || e < kLeast) return e >= kLeast;
    int a = qi != 0.0 ? __double2hiint(fabs(cdt2)) : kOne;
    int b = qj != 0.0 ? __double2hiint(fabs(qj)) : kOne;
    a = __reduce_min_sync(0xffffffffu, a);
    b = __reduce_min_sync(0xffffffffu, b);
    return a >= kLeast && a >= kLeast + (kOne - b);  // the high words of a product add up, but for kOne
}

// What a block's sums lack after its first pass: the half-displacement's constant factors, and
// velocities over dt (uv_fast_pair).
__device__ __forceinline__ void walk_scale(const UvFastStep &T, double *ws, int lane, double racc[6])
{
    const double sv = 0.5 / T.dt;
    double2 *acc = slice_sums(ws);
    double2 a = acc[lane];
    acc[lane] = make_double2(0.25 * a.x, 0.25 * a.y);
    a = acc[32 + lane];
    acc[32 + lane] = make_double2(0.25 * a.x, sv * a.y);
    a = acc[64 + lane];
    acc[64 + lane] = make_double2(sv * a.x, sv * a.y);
#pragma unroll
    for (int d = 0; d < 6; d++) racc[d] *= d < 3 ? 0.25 : sv;
    __syncwarp();
}

// A block after its first pass (sums racc and the slice's, the pairs in `left` unsolved): many others, or a
// diagonal block, finished on the spot; its sums written.  Returns how many are left for the queue.
template <bool kDeterministic, bool kRest>
__device__ __forceinline__ unsigned walk_block_finish(const WalkSystem &S, const WalkBlock &B, unsigned left, double racc[6],
                                                      double *ws, uint32_t *wslots, const LearnedRows &R, double dt,
                                                      int lane, WalkCounts &c)
{
    const bool diag = B.bi == B.bj;
    const int i = B.bi * 32 + lane, j = B.bj * 32 + lane;
    c.pairs += block_lane_pairs(lane, B.bi, B.bj, S.n);
    unsigned others = __reduce_add_sync(0xffffffffu, (unsigned)__popc(left));
    if (others != 0u && (diag || others > (unsigned)kQueuePairs)) {  // finished on the spot
        double si[7], sj[7];
        load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, i, si);
        // the slice has the columns' states already; without these three lines the registers around the walk come out
        // such that it is slower (plummer_32768, learned: 3.82 against 3.86 ms)
        load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, j, sj);
        slice_states(ws, lane, sj);
        __syncwarp();
        uint32_t mask[kMlpHeads] = {0u, 0u};
        auto other = [&](int src, int k, const double *row, double *h) {
            double r[3], g[3];
            const double eps_ij = slice_pair(ws, src, row, S.q != nullptr, S.eps_th, r, g);
            uint32_t x01 = 0u;
            const int kind = walk_other_pair<kRest>(eps_ij, dt, r, g, h, x01, c);
            if (kRest && kind != kLearnedPlain) {
                mask[kHeadHyp] |= (kind == kLearnedHyp ? 1u : 0u) << k;
                mask[kHeadEll] |= (kind == kLearnedHyp ? 0u : 1u) << k;
                wslots[lane * 32 + k] = x01;
            }
        };
        uv_walk_rest(left, ws, lane, si, racc, other);
        if (kRest) rest_block_defer(R, B.item, mask, wslots, lane);
        others = 0u;
    }
    double cacc[6];
    slice_sums_of(ws, lane, cacc);
    walk_write<kDeterministic>(S, B.bi, B.bj, lane, racc, cacc);
    __syncwarp();  // the slice is reused by the next block; the sums are there for the queue
    return others;
}

// the pairs in `left` of block B, the queue's nblocks-th, behind the qn pairs there
__device__ __forceinline__ void walk_queue_push(unsigned int *queue, WalkBlock *blocks, const WalkBlock &B, unsigned left,
                                                int qn, int nblocks, int lane)
{
    unsigned incl = (unsigned)__popc(left);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    int at = qn + (int)incl - __popc(left);
    for (unsigned m = left; m; m &= m - 1u)
        queue[at++] = ((unsigned)nblocks << 10) | ((unsigned)(__ffs(m) - 1) << 5) | (unsigned)lane;
    if (lane == 0) blocks[nblocks] = B;
    __syncwarp();
}

// lane's pairs of a block, bit k (no short step)
__device__ __forceinline__ unsigned walk_all_pairs(bool diag, int lane, bool row_live, int ncols)
{
    unsigned left = 0u;
    const int k0 = diag ? 1 : 0, k1 = diag ? 16 : 31;
    for (int k = k0; k <= k1; k++)
        if ((!diag || k < 16 || lane < 16) && row_live && ((lane + k) & 31) < ncols) left |= 1u << k;
    return left;
}

// One block by a CTA of kWalkBlockWarps warps (small systems, where a warp's 32 offsets in a row are most of
// a step): the warps solve the first pass's pairs of four offsets each, every h waits in shared memory, and a
// warp per component adds the rows and the columns in offset order; warp 0 does the rest of the
// block as the walk does.  The same sums, bitwise.  Dynamic shared memory, in doubles: warp 0's slice and
// queue as the walk's, the row sums, the masks of pairs left, the h.
constexpr int kWalkBlockWarps = 8;
template <bool kRest>
__host__ __device__ constexpr size_t walk_block_smem_bytes()
{
    return (size_t)(walk_warp_doubles<kRest>() + 6 * 32 + 16 + 6 * 1024) * sizeof(double);
}

template <bool kDeterministic, bool kRest, class Items>
__device__ __forceinline__ void uv_block_solve(const Items &I, long long t, double dt, const LearnedRows &R, WalkCounts &c)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *ws = warp_slices;
    WalkBlock *blocks = reinterpret_cast<WalkBlock *>(ws + kTileSmemDoubles);
    unsigned int *queue = reinterpret_cast<unsigned int *>(blocks + kQueuePairs);
    uint32_t *wslots = reinterpret_cast<uint32_t *>(ws + kWalkSliceDoubles);
    double *rsums = ws + walk_warp_doubles<kRest>();
    unsigned *lefts = reinterpret_cast<unsigned *>(rsums + 6 * 32);
    double *hs = rsums + 6 * 32 + 16;
    const UvFastStep T = uv_fast_step(dt);
    const WalkBlock B = I.block(t);
    const WalkSystem S = I.system(B.sys);
    const bool diag = B.bi == B.bj;
    const int i = B.bi * 32 + lane, ncols = S.n - B.bj * 32;
    const bool full_block = !diag && ncols >= 32;
    const int k0 = diag ? 1 : 0, k1 = diag ? 16 : 31;
    UvRow row;
    bool fast = T.on;  // the same for the CTA
    {
        double si[7];
        load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, i, si);
        row.cdt2 = S.q ? S.eps_th * T.dt2 * si[6] : S.eps_th * T.dt2;
#pragma unroll
        for (int d = 0; d < 6; d++) row.s[d] = si[d];
        row.dt = T.dt;
        if (warp == 0) {
            double sj[7];
            load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, B.bj * 32 + lane, sj);
            fast = fast && walk_coupling_normal(S, T.dt2, row.cdt2, si[6], sj[6]);
            slice_fill(ws, lane, sj);
            lefts[lane] = 0u;
        }
    }
    fast = __syncthreads_and(fast);
    if (fast) {
        unsigned mine = 0u;
        for (int k = k0 + warp; k <= k1; k += kWalkBlockWarps) {
            const int src = (lane + k) & 31;
            const bool active = full_block || ((!diag || k < 16 || lane < 16) && i < S.n && src < ncols);
            double r[3], w[3], h[6];
            walk_diff(ws, src, row, r, w);
            const bool ok = uv_fast_pair(S.q ? row.cdt2 * ws[6 * 32 + src] : row.cdt2, r, w, h);
            mine |= (active && !ok ? 1u : 0u) << k;
#pragma unroll
            for (int d = 0; d < 6; d++) hs[1024 * d + 32 * k + lane] = active && ok ? h[d] : 0.0;
        }
        if (mine) atomicOr(&lefts[lane], mine);
        __syncthreads();
        if (warp < 6) {
            unsigned left = lefts[lane];
            int last = k1;  // the walk stops after kProbe offsets of a long step's block
            if (full_block && __reduce_add_sync(0xffffffffu, (unsigned)__popc(left & ((1u << kProbe) - 1u))) > 32u * kProbe / 4u)
                last = kProbe - 1;
            const double *h = hs + 1024 * warp;
            double rsum = 0.0, csum = 0.0;
#pragma unroll 8
            for (int k = k0; k <= last; k++) {
                rsum += h[32 * k + lane];
                csum += h[32 * k + ((lane - k) & 31)];
            }
            rsums[32 * warp + lane] = rsum;
            double2 *acc = slice_sums(ws) + (warp >> 1) * 32 + lane;
            if (warp & 1) acc->y = csum;
            else acc->x = csum;
        }
        __syncthreads();
    }
    if (warp != 0) return;
    unsigned left;
    double racc[6];
    if (fast) {
        left = lefts[lane];
        if (full_block && __reduce_add_sync(0xffffffffu, (unsigned)__popc(left & ((1u << kProbe) - 1u))) > 32u * kProbe / 4u)
            left |= 0xffffffffu << kProbe;
#pragma unroll
        for (int d = 0; d < 6; d++) racc[d] = rsums[32 * d + lane];
        walk_scale(T, ws, lane, racc);
    } else {
#pragma unroll
        for (int d = 0; d < 6; d++) racc[d] = 0.0;
        left = walk_all_pairs(diag, lane, i < S.n, ncols);
    }
    const unsigned others = walk_block_finish<kDeterministic, kRest>(S, B, left, racc, ws, wslots, R, dt, lane, c);
    if (others != 0u) {
        walk_queue_push(queue, blocks, B, left, 0, 0, lane);
        walk_queue<kDeterministic, kRest>(I, R, dt, queue, blocks, (int)others, lane, c);
    }
}

// The walk of a persistent grid: warp `first` of `stride` warps takes blocks first, first + stride, ... of
// `count`.  I.block(t) gives block t, I.system(s) a system; `slice` is where the warp's doubles
// (walk_warp_doubles) begin in the dynamic shared memory.  The counts go to stats.
template <bool kDeterministic, bool kRest, class Items>
__device__ __forceinline__ void uv_walk_blocks(const Items &I, long long first, long long stride, long long count,
                                               double dt, int slice, const LearnedRows &R, unsigned long long *stats)
{
    const int lane = threadIdx.x & 31;
    WalkCounts c = {0, 0, 0, 0};
    double *ws = warp_slices + slice;
    WalkBlock *blocks = reinterpret_cast<WalkBlock *>(ws + kTileSmemDoubles);
    unsigned int *queue = reinterpret_cast<unsigned int *>(blocks + kQueuePairs);
    uint32_t *wslots = reinterpret_cast<uint32_t *>(ws + kWalkSliceDoubles);
    const UvFastStep T = uv_fast_step(dt);
    int qn = 0, nblocks = 0;  // pairs and blocks in the queue
    int uncounted = 0;        // blocks since the counts were flushed
    for (long long t = first;; t += stride) {  // warp-uniform
        const bool have = t < count;
        unsigned left = 0u, others = 0u;
        WalkBlock B{};
        if (have) {
            B = I.block(t);
            const WalkSystem S = I.system(B.sys);
            const bool diag = B.bi == B.bj;
            const int i = B.bi * 32 + lane, j = B.bj * 32 + lane;
            const int ncols = S.n - B.bj * 32;  // bi <= bj: the rows of an off-diagonal block are all there
            double racc[6] = {0, 0, 0, 0, 0, 0};
            {
                double si[7], sj[7];
                load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, i, si);
                load_particle(S.x, S.y, S.z, S.u, S.v, S.w, S.q, S.n, j, sj);
                UvRow row;
                row.cdt2 = S.q ? S.eps_th * T.dt2 * si[6] : S.eps_th * T.dt2;
#pragma unroll
                for (int d = 0; d < 6; d++) row.s[d] = si[d];
                row.dt = T.dt;
                slice_fill(ws, lane, sj);
                __syncwarp();
                if (T.on && walk_coupling_normal(S, T.dt2, row.cdt2, si[6], sj[6])) {
                    if (!diag && ncols >= 32) {
                        left = S.q ? uv_walk_full<true>(slice, row, lane, racc) : uv_walk_full<false>(slice, row, lane, racc);
                    } else {
                        left = S.q ? uv_walk_part<true>(slice, row, lane, diag, i < S.n, ncols, racc)
                                   : uv_walk_part<false>(slice, row, lane, diag, i < S.n, ncols, racc);
                    }
                    walk_scale(T, ws, lane, racc);
                } else {
                    left = walk_all_pairs(diag, lane, i < S.n, ncols);
                }
            }
            others = walk_block_finish<kDeterministic, kRest>(S, B, left, racc, ws, wslots, R, dt, lane, c);
        }
        if (qn != 0 && (!have || qn + (int)others > kQueuePairs)) {
            walk_queue<kDeterministic, kRest>(I, R, dt, queue, blocks, qn, lane, c);
            qn = nblocks = 0;
        }
        if (!have || ++uncounted == kWalkFlushBlocks) {
            walk_flush_counts(c, stats, lane);
            if (!have) return;
            c = {0, 0, 0, 0};
            uncounted = 0;
        }
        if (others != 0u) {
            walk_queue_push(queue, blocks, B, left, qn, nblocks, lane);
            nblocks++;
            qn += (int)others;
        }
    }
}

}  // namespace bia
