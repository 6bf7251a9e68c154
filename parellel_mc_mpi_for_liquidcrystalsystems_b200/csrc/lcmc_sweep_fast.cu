// lcmc_sweep_fast.cu - FP32 checkerboard phase (production path).
//
// One CTA per active cell (grid-stride over all active cells of all replicas).
// Within a colour phase the 26 neighbour cells of an active cell do not move
// (they have other colours), and each particle of the active cell is attempted
// exactly once, from its phase-start state, with a trial state that depends
// only on its own Philox draws (precomputed for the whole sweep by the rebin
// gather, k_gather).  So for every particle k the energy against the 26 static
// cells, old and new, is independent of the other attempts:
//
//   dE_k = [S_new(k) - S_old(k)]                               static cells
//        + sum_{m > k} [phi(n_k, o_m) - phi(o_k, o_m)]          later in-cell partners
//        + sum_{m < k} [phi(n_k, n_m) - phi(o_k, n_m)]  if m was accepted,
//                      [phi(n_k, o_m) - phi(o_k, o_m)]  if not  earlier partners
//        + U_coll(n_k) - U_coll(o_k)
//
// Each earlier partner contributes exactly one of its two terms, never one and
// then a correction: a near-overlap term of 1e20 or more that would cancel must
// not pass through the FP64 sum, whose rounding at that size (1e4 and up) would
// swamp dE_k.  This is exactly E_new - E_old of attempt_monte_carlo_move
// (MCnptColloid.c:2491-2563) for the sequential in-cell order (ascending id);
// only the decisions depend on each other, through a triangular system.
//
// What bounds it: one cell's attempt is a chain of short stages (staging, reach
// tests, pair terms, decisions, write-back) with a block barrier between them,
// so an SM needs several cells in flight, and how many is set by the shared
// memory of one (36-74 KB, 21 KB for the cells of a gas); with six blocks of four warps the schedulers issue
// in 58 % of the cycles (the pair terms take 37 % of the instructions, the
// MUFU pipe is at 29 %, DRAM at 3 %).  Stages of a cell:
//   1 copies   the 26 static cells' FP32 states (float4 x,y,z,ux and float2
//              uy,uz, relative to each particle's own cell origin) come into
//              shared memory as bulk copies that ran under the previous cell's
//              decisions; the stencil offset is added, and each candidate gets
//              a half-precision test vector
//   2 tests    which candidates lie within reach (cutoff plus displacement) of
//              a particle's old position, eight particles and sixteen
//              candidates per matrix instruction (mma m16n8k8); the sign bits
//              become the particle's candidate list.  The same tests on the
//              FP32 pipes, 16 instructions per 32 pairs with ballots and prefix
//              counts, were half of the old kernel's task time
//   3 tasks    warps take tasks from a shared queue:
//              particle task (two particles): Gay-Berne terms of the old and
//                the trial state over both lists, packed FP32 operations (both
//                states in one instruction), lane sums of new - old in FP64
//              pair task: 32 unordered in-cell pairs, 4 terms each
//              (old/new x old/new)
//   4 base     four threads per particle: static + colloid + later in-cell
//              partners
//   5 decide   warp 0: Metropolis decisions in id order; warp 1 looks up the
//              next cell's stencil and starts its copies, threads 32 + k fetch
//              the next cell's records and this cell's FP64 trial states
//   6 write    accepted trial states to the FP64 master arrays
// The list order, and so every sum, depends neither on the block size nor on
// the capacity class: a system's moves do not depend on how it is batched.
// One B200, 1,048,576 rods at rho* = 0.32 (5832 cells per phase), all eight
// phases: 1.97 ms before the tests went to matrix instructions and the terms to
// packed operations, 1.49 ms now; 262,144 rods at 0.28: 0.57 -> 0.46 ms; a grid
// of at most one cell per SM (wide blocks): 0.32 -> 0.19 ms (32,768 rods NPT).
//
// FP64 for overlaps: FP32 rounding of a pair term is relative to the term,
// and near an overlap (R^12 up to 1e36 just above the 1e9 clamp) it exceeds
// any energy scale, so a decision or a running energy built from such terms
// is meaningless.  A static pair whose FP32 term (old or new state) exceeds
// f_big in magnitude, hits the overlap clamp or is not finite is evaluated
// again in FP64 from the master arrays, both states, on the one-fold minimum image; the lane
// sums are FP64, so such terms carry FP64 rounding only.  A cell with such an
// in-cell term (whose pair differences are kept in FP32) makes no move here and
// is handed over to k_phase_rescue, which attempts it from the same phase-start
// state in FP64; a cell above this kernel's capacity (particles, staged
// candidates or list entries) is run again there in FP32 with the largest
// capacity, and in FP64 when its class does not hold it.  Below f_big the FP32 terms carry an absolute
// error of at most about 2e-4 f_big / 100 (1.9e-4 relative, stated per pair),
// so decisions differ from FP64 only at near-ties.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "lcmc_gb.cuh"
#include "lcmc_internal.h"
#include "lcmc_rng.cuh"
#include "lcmc_tc.cuh"
#include "lcmc_trial.cuh"

namespace lcmc {

// FP64 pair term for a pair the FP32 term cannot carry: pair_energy64's
// form for mu = 2, nu = 1, sigma0 = 1, else the reference-order pair_exact.
template <bool SPEC21>
__device__ __forceinline__ double pair64_t(const GBConsts &k, double r2, const double d[3], const double ei[3],
                                           const double ej[3])
{
    return SPEC21 ? pair_energy64_21(k, r2, d, ei, ej) : pair_exact(k, r2, d, ei, ej);
}

struct BigPair {
    double e0, e1; // FP64 terms of the old and the new state (0 beyond the cutoff)
    int n;         // in-cutoff states (0, 1 or 2)
};

// Both states of one static pair (active particle at slot gk, its trial
// state, candidate at slot gj) in FP64 from the master arrays, on the one-fold
// minimum image, the cutoff decided in FP64.  (For fixup_big, which is not
// inlined: the rare path keeps its registers out of the hot loop's allocation.)
template <bool SPEC21>
__device__ __forceinline__ BigPair big_pair64(const double *__restrict__ px, const double *__restrict__ py,
                                           const double *__restrict__ pz, const double *__restrict__ ox,
                                           const double *__restrict__ oy, const double *__restrict__ oz,
                                           const double *__restrict__ tnx, const double *__restrict__ tny,
                                           const double *__restrict__ tnz, const double *__restrict__ tux,
                                           const double *__restrict__ tuy, const double *__restrict__ tuz,
                                           const Replica *__restrict__ rp, int gk, int gj)
{
    const Replica &p = *rp;
    const double rj[3] = {px[gj], py[gj], pz[gj]};
    const double ej[3] = {ox[gj], oy[gj], oz[gj]};
    const double ro[3] = {px[gk], py[gk], pz[gk]};
    const double eo[3] = {ox[gk], oy[gk], oz[gk]};
    const double rn[3] = {tnx[gk], tny[gk], tnz[gk]};
    const double en[3] = {tux[gk], tuy[gk], tuz[gk]};
    BigPair b;
    double d[3];
    double q2 = dist_fold(ro[0], ro[1], ro[2], rj[0], rj[1], rj[2], p.L, d);
    const bool i0 = q2 < p.k.rc2;
    b.e0 = i0 ? pair64_t<SPEC21>(p.k, q2, d, eo, ej) : 0.0;
    q2 = dist_fold(rn[0], rn[1], rn[2], rj[0], rj[1], rj[2], p.L, d);
    const bool i1 = q2 < p.k.rc2;
    b.e1 = i1 ? pair64_t<SPEC21>(p.k, q2, d, en, ej) : 0.0;
    b.n = (int)i0 + (int)i1;
    return b;
}

template <int AMAX, int CCAP, int LCAP>
struct FastSmem {
    static constexpr int NPAIR = AMAX * (AMAX - 1) / 2;
    float4 cpos[CCAP]; // x, y, z, ux of the static cells' particles, cell by cell
    float2 cori[CCAP]; // uy, uz
    union {
        // half-precision test vectors (x, y, z, |c|^2 rounded down) of the
        // candidates, relative to the cell centre, scaled; dead once the lists stand
        uint2 ch[CCAP + 16];
        // in-cell pair terms rounded to FP32: C - A, and (B - A, D - C) (for a later particle the decisions
        // add D - C if the earlier partner moved, B - A if it stayed)
        struct {
            float2 pBD[NPAIR];
            float pCA[NPAIR];
        };
    };
    // old (a) and trial (b) state of each active particle, relative to the cell origin, in pairs:
    // [0] = (ax, bx, ay, by), [1] = (az, bz, aux, bux), [2] = (auy, buy, auz, buz)
    float4 pst[AMAX][3];
    union {
        struct {
            uint2 qh[AMAX]; // (-2x, -2y, -2z, 1) of a particle (the reach tests)
            float qc[AMAX]; // |q|^2 - reach^2 of a particle (1e30: nothing in reach)
        };
        struct {
            // static part of dE (the task queue), then all of it that does not depend on a decision
            double Sdif[AMAX];
        };
    };
    double tdU[AMAX], tlu[AMAX]; // colloid dU of the trial, log of the Metropolis draw
    unsigned long long pairs;
    uint64_t full; // mbarrier: the static cells' copies have landed
    unsigned short lst[AMAX], lcnt[AMAX]; // a particle's part of the list
    union {
        unsigned short list[LCAP]; // candidates in reach, particle by particle
        // from the end of the task queue to the next cell's reach tests, thread 32 + k's own fetches:
        // the next cell's particle k, and the FP64 trial state of this cell's
        struct {
            ActRec next[AMAX];
            double wn[AMAX][6];
        };
    };
    unsigned char hard[AMAX];
    unsigned char acc[AMAX];
    // pairs whose FP32 term is above f_big (overlaps), evaluated in FP64 by the
    // fix-up pass after the task queue: static pairs (particle k << 16 | staged
    // candidate) and in-cell pairs (pair index)
    static constexpr int BIGCAP = 32;
    unsigned int bigs[BIGCAP];
    unsigned short bigp[BIGCAP];
    int nbigs, nbigp;
    struct Stencil {
        int start[27], cnt[27], pos[28]; // stencil cells: first slot, particles, place of the copy
        int skip;                        // 0 runs here, 1 not an FP32 cell, 2 above a capacity
    } st[2]; // the cell that runs and the next
    int nlist, task;
    int overflow;
    int big; // a pair term above f_big (or clamped, or non-finite): attempt the cell in FP64
};

// Hand a cell over to the FP64 phase kernel (k_phase_rescue, launched after
// this one in the same colour phase); it writes the cell's results.
__device__ __forceinline__ void hand_over(const DevView &v, int ci, int cell, int mode)
{
    const int i = atomicAdd(&v.resc_count[ci], 1);
    v.resc_list[(size_t)ci * v.ctot + i] = cell * 4 + mode;
}



// FP64 pair term of particles at ri (orientation ei) and rj (ej), one-fold
// minimum image, 0 beyond the cutoff.
template <bool SPEC21>
__device__ __forceinline__ double term64(const Replica &p, const double ri[3], const double ei[3], const double rj[3],
                                         const double ej[3])
{
    double d[3];
    const double r2 = dist_fold(ri[0], ri[1], ri[2], rj[0], rj[1], rj[2], p.L, d);
    return r2 < p.k.rc2 ? pair64_t<SPEC21>(p.k, r2, d, ei, ej) : 0.0;
}

// FP64 fix-up of the pairs whose FP32 term is above f_big (overlaps), after
// the task queue, with every thread of the block:
//   in-cell pairs (thread per listed pair): the four terms phi(o/n_q, o/n_p)
//     in FP64 from the master arrays; the differences C - A, B - A, D - C
//     replace the FP32 ones (rounded to FP32 once: below 1e5 eps0 that keeps
//     them within 0.01 eps0); a larger term (the overlap clamp and its
//     neighbourhood) sends the cell to the FP64 hand-over kernel;
//   static pairs (thread per particle): the particle's listed pairs in
//     ascending staged order, both states in FP64, added to its static sums
//     (a fixed order: the bits do not depend on scheduling).
template <int NT, typename SM, bool SPEC21>
__device__ __noinline__ void fixup_big(const DevView *__restrict__ vp, int r, int g0, int na, int which, SM &sm)
{
    const DevView &v = *vp;
    const Replica &p = v.rep[r];
    const int t = threadIdx.x;
    const int nbp = min(sm.nbigp, SM::BIGCAP), nbs = min(sm.nbigs, SM::BIGCAP);
    for (int e = t; e < nbp; e += NT) {
        const int idx = sm.bigp[e];
        int q = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)idx)) * 0.5f);
        while (q * (q - 1) / 2 > idx) q--;
        while ((q + 1) * q / 2 <= idx) q++;
        const int pp = idx - q * (q - 1) / 2;
        const int gq = g0 + q, gp = g0 + pp;
        const double oq[3] = {v.px[gq], v.py[gq], v.pz[gq]}, uq[3] = {v.ox[gq], v.oy[gq], v.oz[gq]};
        const double nq[3] = {v.tnx[gq], v.tny[gq], v.tnz[gq]}, wq[3] = {v.tux[gq], v.tuy[gq], v.tuz[gq]};
        const double op[3] = {v.px[gp], v.py[gp], v.pz[gp]}, up[3] = {v.ox[gp], v.oy[gp], v.oz[gp]};
        const double np_[3] = {v.tnx[gp], v.tny[gp], v.tnz[gp]}, wp[3] = {v.tux[gp], v.tuy[gp], v.tuz[gp]};
        // A = (o_q, o_p), B = (n_q, o_p), C = (o_q, n_p), D = (n_q, n_p)
        double term[4] = {term64<SPEC21>(p, op, up, oq, uq), term64<SPEC21>(p, op, up, nq, wq),
                          term64<SPEC21>(p, np_, wp, oq, uq), term64<SPEC21>(p, np_, wp, nq, wq)};
        // terms with the trial state of a particle that cannot move are never used
        const bool hp = sm.hard[pp] != 0, hq = sm.hard[q] != 0;
        if (hq) term[1] = term[3] = 0.0;
        if (hp) term[2] = term[3] = 0.0;
        if (hp && hq) term[0] = 0.0;
        if (!(fabs(term[0]) <= 1e5 && fabs(term[1]) <= 1e5 && fabs(term[2]) <= 1e5 && fabs(term[3]) <= 1e5)) {
            sm.big = 1;
        } else {
            sm.pCA[idx] = (float)(term[2] - term[0]);
            sm.pBD[idx] = make_float2((float)(term[1] - term[0]), (float)(term[3] - term[2]));
        }
    }
    unsigned long long extra = 0ull;
    for (int k = t; k < na; k += NT) {
        double so = 0.0, sn = 0.0;
        bool any = false;
        int last = -1;
        for (;;) { // this particle's listed candidates in ascending staged order
            int best = 1 << 30;
            for (int e = 0; e < nbs; e++) {
                const unsigned u = sm.bigs[e];
                const int j = (int)(u & 0xFFFFu);
                if ((int)(u >> 16) == k && j > last && j < best) best = j;
            }
            if (best == (1 << 30)) break;
            last = best;
            int sl = 0, hi = 27; // the candidate's cell: the last that begins at or before it
            // (a cell without particles shares the place of the next one, or lies before a gap: never picked)
            while (hi - sl > 1) {
                const int mid = (sl + hi) >> 1;
                if (sm.st[which].pos[mid] <= best) sl = mid;
                else hi = mid;
            }
            const BigPair b = big_pair64<SPEC21>(v.px, v.py, v.pz, v.ox, v.oy, v.oz, v.tnx, v.tny, v.tnz, v.tux,
                                                 v.tuy, v.tuz, v.rep + r, g0 + k,
                                                 sm.st[which].start[sl] + best - sm.st[which].pos[sl]);
            so += b.e0;
            sn += b.e1;
            extra += (unsigned long long)b.n;
            any = true;
        }
        if (any) {
            sm.Sdif[k] += sn - so;
        }
    }
    if (extra) atomicAdd(&sm.pairs, extra);
}

// Sums over the warp of two values per lane: lanes 0-15 get the sum of a, 16-31
// of b (one exchange halves the values a lane carries).
__device__ __forceinline__ double warp_sum2(double a, double b, int lane)
{
    const bool up = lane & 16;
    const double s = up ? a : b;
    double x = (up ? b : a) + __shfl_xor_sync(0xffffffffu, s, 16);
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// One warp: the stencil of active cell `rec`, and the places of its 26 static
// cells' copies in shared memory.  Cells that cannot run here are marked.
template <typename ST, int AMAX, int CCAP>
__device__ __forceinline__ void prepare_stencil(const DevView &v, ST &st, const int4 rec, int lane)
{
    const Replica &p = v.rep[rec.y];
    const int nc0 = p.nc[0], nc1 = p.nc[1], nc2 = p.nc[2];
    int start = 0, cnt = 0;
    if (lane < 27) {
        int x = (rec.z & 255) + lane % 3 - 1, y = ((rec.z >> 8) & 255) + (lane / 3) % 3 - 1,
            z = ((rec.z >> 16) & 255) + lane / 9 - 1;
        x += x < 0 ? nc0 : (x >= nc0 ? -nc0 : 0);
        y += y < 0 ? nc1 : (y >= nc1 ? -nc1 : 0);
        z += z < 0 ? nc2 : (z >= nc2 ? -nc2 : 0);
        const int c = p.cell_off + (z * nc1 + y) * nc0 + x;
        start = v.cell_start[c];
        cnt = v.cell_start[c + 1] - start;
    }
    const int na = __shfl_sync(0xffffffffu, cnt, 13);
    // a cell's copy keeps the parity of its slots (granules of two entries); cells that follow one another in
    // memory (a row's, usually) follow one another here, others begin a granule of their own
    int end = lane < 27 ? start + cnt : 0;
    const int e12 = __shfl_sync(0xffffffffu, end, 12);
    const int s13 = lane == 13 ? e12 : start;
    if (lane == 13) end = e12; // the cell itself has no copy
    int prev = __shfl_up_sync(0xffffffffu, end, 1);
    if (lane == 0) prev = -1;
    const int pad = lane >= 27 || s13 == prev ? 0 : (lane > 0 ? prev & 1 : 0) + (s13 & 1);
    const int own = lane < 27 ? end - s13 : 0;
    int pos = pad + own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, pos, o);
        if (lane >= o) pos += y;
    }
    const int all = __shfl_sync(0xffffffffu, pos, 31);
    if (lane < 27) {
        st.start[lane] = start;
        st.cnt[lane] = cnt;
        st.pos[lane] = pos - own;
    }
    if (lane == 27) st.pos[27] = all;
    if (lane == 0) st.skip = !p.use_fast ? 1 : (na > AMAX || na > p.cap || all + 1 > CCAP ? 2 : 0);
}

// One warp: the copies of a prepared cell's static cells (one bulk copy per
// cell and array, in granules of 16 bytes), completing on sm.full.
template <typename SM>
__device__ __forceinline__ void copy_static(const DevView &v, SM &sm, int which, int lane)
{
    const auto &st = sm.st[which];
    if (st.skip) return; // (uniform)
    const int start = lane < 27 ? st.start[lane] : 0, cnt = lane < 27 && lane != 13 ? st.cnt[lane] : 0;
    const int n = cnt == 0 ? 0 : ((start + cnt + 1) & ~1) - (start & ~1); // entries copied
    const unsigned bytes = 24u * __reduce_add_sync(0xffffffffu, (unsigned)n);
    tc::fence_proxy_async_smem(); // the block's reads and writes of the last cell's copies came before its barrier
    if (lane == 0) tc::mbar_arrive_expect_tx(&sm.full, bytes);
    __syncwarp();
    if (n > 0) {
        const int pos = st.pos[lane] & ~1, from = start & ~1;
        tc::bulk_load(&sm.cpos[pos], v.cl4 + from, (unsigned)n * 16u, &sm.full);
        tc::bulk_load(&sm.cori[pos], v.cl2 + from, (unsigned)n * 8u, &sm.full);
    }
}

template <int BYTES>
__device__ __forceinline__ void fetch_async(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The fetch of one particle's attempt record.
__device__ __forceinline__ void fetch_rec(ActRec *dst, const ActRec *src)
{
#pragma unroll
    for (int i = 0; i < (int)sizeof(ActRec); i += 16) fetch_async<16>((char *)dst + i, (const char *)src + i);
}

constexpr unsigned FAST_WAIT_TRIES = 1u << 24; // mbarrier tries for the copies of a block that leaves

// Cells a retry left to the FP64 attempts of its block.
struct RetryFailed {
    int n, ticket;
    int cell[32]; // cell * 4 + mode
};

// The FP32 attempts of a block: active cells a, a + step, ... below `total` of
// phase ci (RETRY: of the phase's retry list).  ONE_K: the pair constants are
// the launch's, ku, else each cell's replica's.
template <int NT, int AMAX, int CCAP, int LCAP, bool SPEC21, bool ONE_K, bool RETRY>
__device__ __forceinline__ void phase_fast_body(const DevView &v, const FastK &ku, int ci, unsigned char *smem_raw, int a,
                                                const int total, const int step, RetryFailed *failed)
{
    using SM = FastSmem<AMAX, CCAP, LCAP>;
    constexpr int NW = NT / 32;
    static_assert(AMAX <= 64, "the decision warp holds two particles per lane");
    static_assert(AMAX + 32 <= NT, "threads 32 .. 32 + AMAX - 1 hold a particle each");
    static_assert(AMAX % 8 == 0 && CCAP % 2 == 0, "test tiles of eight particles; copies of 16 bytes");
    SM &sm = *reinterpret_cast<SM *>(smem_raw);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int4 *tab = v.act_tab + (size_t)ci * v.act_max;
    const int *list = v.retry_list + (size_t)ci * v.act_max;
    auto entry = [&](int i) { return tab[RETRY ? list[i] : i]; };
    // cells without particles are passed by: from entry i, its record e, to the next that has some (i >= total: none)
    auto pass_empty = [&](int &i, int4 &e) {
        while (!RETRY && i < total && !((unsigned)e.z >> 24)) { // (32 entries at a time)
            const int q = i + step * (1 + lane);
            const unsigned some = __ballot_sync(0xffffffffu, q < total && ((unsigned)tab[q].z >> 24));
            i += step * (some ? __ffs(some) : 32);
            if (some || i < total) e = tab[i];
        }
    };
    if (a >= total) return;
    int4 rec = entry(a); // cell, replica, coordinates (8 bits each) and count of the particles (capped), first slot
    pass_empty(a, rec);
    if (a >= total) return; // (the whole block)
    if (t == 0) {
        tc::mbar_init(&sm.full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    int an = a + step; // the next cell
    int4 nxt = an < total ? entry(an) : make_int4(0, 0, 0, 0);
    const int kw = t - 32; // thread 32 + k: particle k
    if (w == 1) {
        prepare_stencil<typename SM::Stencil, AMAX, CCAP>(v, sm.st[0], rec, lane);
        __syncwarp();
        copy_static(v, sm, 0, lane);
    }
    if (kw >= 0 && kw < AMAX && kw < (int)((unsigned)rec.z >> 24)) fetch_rec(&sm.next[kw], v.act_rec + rec.w + kw);
    unsigned phase = 0;
    int which = 0, id = 0; // id: of particle kw of the cell that runs
    fetch_wait();          // (a first cell that does not run here reads no record)
    __syncthreads();

    for (;;) {
        const int cell = rec.x, r = rec.y, g0 = rec.w;
        const Replica &p = v.rep[r];
        const FastK K = ONE_K ? ku : fast_consts(p.k);
        int mode = sm.st[which].skip; // 0 runs here, 1 not an FP32 cell, 2 handed over (capacity), 3 handed over (terms)
        const int na = sm.st[which].cnt[13];
        int s26 = 0;
        unsigned long long npairs = 0ull;
        if (mode == 0) {
            // ---- 1 the prepared cell's copies: offsets and test vectors ----
            const float wx = (float)p.w[0], wy = (float)p.w[1], wz = (float)p.w[2];
            const float wmax = fmaxf(wx, fmaxf(wy, wz));
            const float mc = 2.0f * wmax; // above any candidate's coordinate from the cell centre (1.5 cells)
            // power of two that brings mc into [4, 8): half precision then rounds a coordinate by at most 2^-11 of it
            const float sc = __int_as_float((129 + 127 - ((__float_as_int(mc) >> 23) & 0xff)) << 23);
            // sqrt(3) axes, a candidate's and a particle's rounding, and the FP32 sums' own
            const float slack = 1.75f / 2048.0f * (mc + 0.5f * wmax) + 1e-3f;
            if (t == 0) {
                sm.overflow = 0;
                sm.big = 0;
                sm.nbigs = 0;
                sm.nbigp = 0;
                sm.pairs = 0ull;
                sm.nlist = 0;
                sm.task = 0;
            }
            if (kw >= 0 && kw < ((na + 7) & ~7)) { // particle kw: states, trial, test vector
                uint2 qh = make_uint2(0u, 0x3c000000u); // (0, 0, 0, 1)
                float qc = 1e30f;
                if (kw < na) {
                    const ActRec ar = sm.next[kw];
                    sm.pst[kw][0] = ar.p0;
                    sm.pst[kw][1] = ar.p1;
                    sm.pst[kw][2] = ar.p2;
                    sm.hard[kw] = (unsigned char)ar.code;
                    sm.tdU[kw] = ar.tdU;
                    sm.tlu[kw] = ar.tlu;
                    id = ar.id;
                    if (!ar.code) {
                        const float rr = ((float)p.k.rc + ar.reach + 1e-3f + slack) * sc;
                        const __half2 xy = __floats2half2_rn((ar.p0.x - 0.5f * wx) * sc, (ar.p0.z - 0.5f * wy) * sc);
                        const __half2 z1 = __floats2half2_rn((ar.p1.x - 0.5f * wz) * sc, -0.5f);
                        const float fx = __low2float(xy), fy = __high2float(xy), fz = __low2float(z1);
                        qc = fx * fx + fy * fy + fz * fz - rr * rr;
                        const __half2 m2 = __floats2half2_rn(-2.0f, -2.0f);
                        qh = make_uint2(tc::h2_bits(__hmul2(xy, m2)), tc::h2_bits(__hmul2(z1, m2)));
                    }
                }
                sm.qh[kw] = qh;
                sm.qc[kw] = qc;
            }
            const auto &st = sm.st[which];
            const int ncand = st.pos[27]; // places of the copies
            if (w == 0) s26 = __reduce_add_sync(0xffffffffu, lane < 27 && lane != 13 ? st.cnt[lane] : 0);
            bool ok = tc::mbar_wait_bounded(&sm.full, phase, v.wait_tries);
            phase ^= 1u;
#pragma unroll 2
            for (int s = w; s < 27; s += NW) {
                const int pos = st.pos[s], cnt = s == 13 ? 0 : st.cnt[s];
                // places between two copies: far from everything
                const int gap = s == 0 ? 0 : st.pos[s - 1] + (s == 14 ? 0 : st.cnt[s - 1]);
                if (gap + lane < pos) sm.ch[gap + lane] = make_uint2(0u, 0x7b000000u);
                const float ox = (float)(s % 3 - 1) * wx, oy = (float)((s / 3) % 3 - 1) * wy, oz = (float)(s / 9 - 1) * wz;
                for (int i = lane; i < cnt; i += 32) {
                    float4 c = sm.cpos[pos + i]; // relative to its own cell's origin
                    c.x += ox;
                    c.y += oy;
                    c.z += oz;
                    sm.cpos[pos + i] = c;
                    const __half2 xy = __floats2half2_rn((c.x - 0.5f * wx) * sc, (c.y - 0.5f * wy) * sc);
                    const __half hz = __float2half_rn((c.z - 0.5f * wz) * sc);
                    const float fx = __low2float(xy), fy = __high2float(xy), fz = __half2float(hz);
                    const __half hs = __float2half_rd(fx * fx + fy * fy + fz * fz);
                    sm.ch[pos + i] = make_uint2(tc::h2_bits(xy), tc::h2_bits(__halves2half2(hz, hs)));
                }
            }
            if (t < 16) sm.ch[ncand + t] = make_uint2(0u, 0x7b000000u); // beyond the last: likewise
            if (__syncthreads_or(!ok)) { // (uniform) the copies did not land within the limit: flag it and leave,
                if (t == 0) atomicOr(&v.stats[r].flags, F_TIMEOUT); // the copies waited for (no others are on their way)
                tc::mbar_wait_bounded(&sm.full, phase ^ 1u, FAST_WAIT_TRIES);
                break;
            }
        // ---- 2 reach tests of eight particles against every candidate ----
        for (int task = w; task < (na + 7) >> 3; task += NW) {
            {
                // test_tile: which candidates lie within reach of eight particles' old positions (cutoff plus the
                // trial's displacement, so both states are covered), by matrix instructions: a candidate's row
                // (x, y, z, |c|^2) times a particle's column (-2x, -2y, -2z, 1) plus |q|^2 - reach^2 is negative
                // when it is in reach.  The operands are in half precision; `slack` covers their rounding (2^-11
                // of a coordinate each) and |c|^2 is rounded down, so every pair inside the cutoff is in the
                // list, and the few beyond it add nothing (the pair evaluation tests the FP32 distance).
                // Lanes q >= 2 carry the unused half of the inner dimension: their column entries are zero.
                // A sign bit is shifted into the lane's mask for each row: lane 4 g + q holds the candidates
                // 8 z + g of particles 2 q and 2 q + 1, the first in the highest bit.
                constexpr int NB = (CCAP + 255) / 256;
                const int g = lane >> 2, q = lane & 3, k0 = 8 * task;
                const uint2 bq = sm.qh[k0 + g];
                const unsigned b0 = q == 0 ? bq.x : (q == 1 ? bq.y : 0u);
                const float c0 = sm.qc[k0 + 2 * q], c1 = sm.qc[k0 + 2 * q + 1];
                const unsigned *ah = reinterpret_cast<const unsigned *>(sm.ch) + 2 * g + (q & 1);
                unsigned m0[NB], m1[NB];
                const int nmt = (ncand + 15) >> 4;
                int n0 = 0, n1 = 0;
#pragma unroll
                for (int b = 0; b < NB; b++) {
                    unsigned x0 = 0u, x1 = 0u;
                    const int e = min(16, nmt - 16 * b);
#pragma unroll 4
                    for (int i = 0; i < e; i++) {
                        const unsigned a0 = ah[32 * (16 * b + i)], a1 = ah[32 * (16 * b + i) + 16];
                        float d[4];
                        tc::mma_16x8x8(d, a0, a1, b0, c0, c1);
                        x0 = __funnelshift_l(__float_as_uint(d[0]), x0, 1);
                        x1 = __funnelshift_l(__float_as_uint(d[1]), x1, 1);
                        x0 = __funnelshift_l(__float_as_uint(d[2]), x0, 1);
                        x1 = __funnelshift_l(__float_as_uint(d[3]), x1, 1);
                    }
                    if (e <= 0) x0 = x1 = 0u;
                    else if (e < 16) {
                        x0 <<= 32 - 2 * e;
                        x1 <<= 32 - 2 * e;
                    }
                    m0[b] = x0;
                    m1[b] = x1;
                    n0 += __popc(x0);
                    n1 += __popc(x1);
                }
                // offsets: lanes of a particle (stride 4) in order, then the particles
                int i0 = n0, i1 = n1;
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    const int y0 = __shfl_up_sync(0xffffffffu, i0, o), y1 = __shfl_up_sync(0xffffffffu, i1, o);
                    if (lane >= o) {
                        i0 += y0;
                        i1 += y1;
                    }
                }
                const int t0 = __shfl_sync(0xffffffffu, i0, 28 + q), t1 = __shfl_sync(0xffffffffu, i1, 28 + q);
                int s = t0 + t1;
                {
                    int y = __shfl_up_sync(0xffffffffu, s, 1, 4);
                    if (q >= 1) s += y;
                    y = __shfl_up_sync(0xffffffffu, s, 2, 4);
                    if (q >= 2) s += y;
                }
                const int all = __shfl_sync(0xffffffffu, s, 3);
                int base = 0;
                if (lane == 0) base = atomicAdd(&sm.nlist, all);
                base = __shfl_sync(0xffffffffu, base, 0);
                const bool fits = base + all <= LCAP;
                base += s - t0 - t1;
                if (g == 0) {
                    sm.lst[k0 + 2 * q] = (unsigned short)base;
                    sm.lst[k0 + 2 * q + 1] = (unsigned short)(base + t0);
                    sm.lcnt[k0 + 2 * q] = (unsigned short)(fits ? t0 : 0);
                    sm.lcnt[k0 + 2 * q + 1] = (unsigned short)(fits ? t1 : 0);
                }
                if (!fits) {
                    if (lane == 0) sm.overflow = 1;
                } else {
                    unsigned short *l0 = sm.list + base + i0 - n0, *l1 = sm.list + base + t0 + i1 - n1;
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        const int c = 256 * b + g;
                        unsigned x0 = m0[b], x1 = m1[b];
                        while (x0 | x1) { // both particles' next candidates (two independent chains)
                            const int z0 = __clz(x0), z1 = __clz(x1); // 32 when exhausted
                            if (x0) *l0++ = (unsigned short)(c + 8 * z0);
                            if (x1) *l1++ = (unsigned short)(c + 8 * z1);
                            x0 &= 0x7fffffffu >> z0;
                            x1 &= 0x7fffffffu >> z1;
                        }
                    }
                }
            }
        }
        __syncthreads();
        // ---- 3 task queue: Gay-Berne terms of two particles' lists, old and trial state; in-cell pairs ----
        const int nptask = (na + 1) >> 1, npair = na * (na - 1) / 2;
        const int ntask2 = nptask + (npair + 31) / 32;
        for (;;) {
            int task = 0;
            if (lane == 0) task = sm.overflow ? ntask2 : atomicAdd(&sm.task, 1);
            task = __shfl_sync(0xffffffffu, task, 0);
            if (task >= ntask2) break;
            if (task >= nptask) { // 32 in-cell pairs, four terms each
            const int idx = (task - nptask) * 32 + lane;
            int npin = 0;
            if (idx < npair) {
                int q = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)idx)) * 0.5f);
                while (q * (q - 1) / 2 > idx) q--;
                while ((q + 1) * q / 2 <= idx) q++;
                const int pp = idx - q * (q - 1) / 2;
                float A, B, Cc, D;
                {
                    // q's states in pairs against p's old (A, B) and trial state (C, D)
                    const float4 Q0 = sm.pst[q][0], Q1 = sm.pst[q][1], Q2 = sm.pst[q][2];
                    const float4 R0 = sm.pst[pp][0], R1 = sm.pst[pp][1], R2 = sm.pst[pp][2];
                    const f32x2 qx = pack2(Q0.x, Q0.y), qy = pack2(Q0.z, Q0.w), qz = pack2(Q1.x, Q1.y);
                    const f32x2 ux = pack2(Q1.z, Q1.w), uy = pack2(Q2.x, Q2.y), uz = pack2(Q2.z, Q2.w);
                    const f32x2 neg = dup2(-1.0f);
                    bool in0, in1;
                    pair_fast_x2<SPEC21>(K, fma2(dup2(R0.x), neg, qx), fma2(dup2(R0.z), neg, qy), fma2(dup2(R1.x), neg, qz),
                                         dup2(R1.z), dup2(R2.x), dup2(R2.z), ux, uy, uz, A, B, in0, in1);
                    A = in0 ? A : 0.0f;
                    B = in1 ? B : 0.0f;
                    npin += 2 * (int)in0 + (int)in1;
                    pair_fast_x2<SPEC21>(K, fma2(dup2(R0.y), neg, qx), fma2(dup2(R0.w), neg, qy), fma2(dup2(R1.y), neg, qz),
                                         dup2(R1.w), dup2(R2.y), dup2(R2.w), ux, uy, uz, Cc, D, in0, in1);
                    Cc = in0 ? Cc : 0.0f;
                    D = in1 ? D : 0.0f;
                    npin += (int)in0;
                }
                // a particle that cannot move (colloid hard core, or a trial out of the cell) keeps
                // its old state: terms with its trial state are never used, so they are dropped
                // before the size test (p hard: C and D unused; q hard: B and D unused)
                const bool hp = sm.hard[pp] != 0, hq = sm.hard[q] != 0;
                if (hq) B = D = 0.0f;
                if (hp) Cc = D = 0.0f;
                if (hp && hq) A = 0.0f;
                if (!(fabsf(A) <= K.big && fabsf(B) <= K.big && fabsf(Cc) <= K.big && fabsf(D) <= K.big)) {
                    const int slot = atomicAdd(&sm.nbigp, 1); // the fix-up pass rewrites this pair
                    if (slot < SM::BIGCAP) sm.bigp[slot] = (unsigned short)idx;
                    else sm.overflow = 1;
                }
                // differences in FP64, then rounded (each term is at most f_big here)
                const double a = A, b = B, c = Cc, d = D;
                sm.pCA[idx] = (float)(c - a);
                sm.pBD[idx] = make_float2((float)(b - a), (float)(d - c));
            }
                npairs += (unsigned long long)__reduce_add_sync(0xffffffffu, npin);
                continue;
            }
            const int ka = 2 * task, kb = ka + 1; // kb = na has an empty list (its tile's padding)
            const int ca = sm.lcnt[ka], cb = kb < na ? sm.lcnt[kb] : 0;
            const int la = sm.lst[ka], lb = (kb < na ? sm.lst[kb] : 0) - ca;
            double sa = 0.0, sb = 0.0; // new minus old of either particle
            int np = 0;
            // FP64 lane sums of the FP32 terms.  Entries [0, ca) belong to
            // particle a, [ca, ca + cb) to particle b.  An entry with a term
            // FP32 cannot carry is listed for the FP64 fix-up pass.
            const int n = ca + cb;
            const f32x2 neg = dup2(-1.0f);
            for (int q = lane; q < n; q += 32) {
                const bool isa = q < ca;
                const int j = sm.list[(isa ? la : lb) + q], k = isa ? ka : kb;
                const float4 P0 = sm.pst[k][0], P1 = sm.pst[k][1], P2 = sm.pst[k][2];
                const float4 c = sm.cpos[j];
                const float2 u = sm.cori[j];
                float e0, e1;
                bool in0, in1;
                pair_fast_x2<SPEC21>(K, fma2(pack2(P0.x, P0.y), neg, dup2(c.x)), fma2(pack2(P0.z, P0.w), neg, dup2(c.y)),
                                     fma2(pack2(P1.x, P1.y), neg, dup2(c.z)), pack2(P1.z, P1.w), pack2(P2.x, P2.y),
                                     pack2(P2.z, P2.w), dup2(c.w), dup2(u.x), dup2(u.y), e0, e1, in0, in1);
                e0 = in0 ? e0 : 0.0f; // beyond the cutoff
                e1 = in1 ? e1 : 0.0f;
                if (!(fmaxf(fabsf(e0), fabsf(e1)) <= K.big) || e0 != e0 || e1 != e1) {
                    const int slot = atomicAdd(&sm.nbigs, 1);
                    if (slot < SM::BIGCAP) sm.bigs[slot] = ((unsigned)k << 16) | (unsigned)j;
                    else sm.overflow = 1;
                    e0 = e1 = 0.0f; // the fix-up counts its pairs
                } else {
                    np += (int)in0 + (int)in1;
                }
                const double d = (double)e1 - (double)e0;
                if (isa) sa += d;
                else sb += d;
            }
            __syncwarp();
            const double sum = warp_sum2(sa, sb, lane);
            if (lane == 0) sm.Sdif[ka] = sum;
            if (lane == 16 && kb < na) sm.Sdif[kb] = sum;
            npairs += (unsigned long long)__reduce_add_sync(0xffffffffu, np);
        }
        if (lane == 0 && npairs) atomicAdd(&sm.pairs, npairs);
        tc::fence_proxy_async_smem(); // the next cell's copies overwrite what this cell read and wrote
        __syncthreads();
        if (!sm.overflow && (sm.nbigs | sm.nbigp)) { // (uniform) FP64 fix-up of the listed pairs
            fixup_big<NT, SM, SPEC21>(&v, r, g0, na, which, sm);
            __syncthreads();
        }
        // a capacity exceeded, or an in-cell term too large to keep in FP32
        if (sm.overflow || sm.big) mode = sm.overflow ? 2 : 3;
        // ---- 4 the part of dE that no decision changes: static cells, colloid, and the in-cell partners after k
        //      (still at their old state when k is tried); four threads per particle ----
        if (mode == 0) {
            for (int k0 = 0; k0 < na; k0 += NT / 4) {
                const int k = k0 + (t >> 2);
                double s0 = 0.0, s1 = 0.0;
                if (k < na) {
                    for (int m = k + 1 + (t & 3); m < na; m += 8) {
                        const int m1 = m + 4;
                        s0 += (double)sm.pCA[m * (m - 1) / 2 + k];
                        s1 += (double)(m1 < na ? sm.pCA[m1 * (m1 - 1) / 2 + k] : 0.0f);
                    }
                }
                s0 += s1;
                s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
                s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
                if ((t & 3) == 0 && k < na) sm.Sdif[k] = sm.Sdif[k] + s0 + sm.tdU[k];
            }
            __syncthreads();
        }
        } // mode == 0

        // ---- 5 warp 0: the Metropolis decisions in id order; meanwhile warp 1 prepares the next cell (its copies run under the decisions), thread
        //      32 + k loads the next cell's particle k and the FP64 trial state of this cell's ----
        // dE_k = base_k + sum over earlier m of (D - C if m was accepted, else
        // B - A): lane k carries dE_k (and lane k - 32 the particles from 32 on);
        // step m decides particle m, whose sum is then complete, and adds m's
        // term to every later particle's.  Both terms are converted ahead of the
        // step, so its chain is the test, the vote and one addition.
        unsigned acc0 = 0u, acc1 = 0u, hc0 = 0u, hc1 = 0u;
        double x0 = 0.0, x1 = 0.0;
        if (w == 0 && mode == 0) {
            const double beta = p.k.beta;
            const bool v0 = lane < na, v1 = lane + 32 < na;
            const bool go0 = v0 && !sm.hard[lane], go1 = v1 && !sm.hard[lane + 32];
            const double lu0 = v0 ? sm.tlu[lane] : 0.0, lu1 = v1 ? sm.tlu[lane + 32] : 0.0;
            x0 = v0 ? sm.Sdif[lane] : 0.0;
            x1 = v1 ? sm.Sdif[lane + 32] : 0.0;
            const float2 *row0 = sm.pBD + (lane * (lane - 1)) / 2, *row1 = sm.pBD + ((lane + 32) * (lane + 31)) / 2;
            if (na <= 32) { // (uniform)
                for (int m0 = 0; m0 < na; m0 += 4) {
                    double ba[4], dc[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float2 q = v0 && m0 + i < lane ? row0[m0 + i] : make_float2(0.0f, 0.0f);
                        ba[i] = (double)q.x;
                        dc[i] = (double)q.y;
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const bool a0 = go0 && ((x0 <= 0.0) || (lu0 <= -beta * x0));
                        const unsigned bit = __ballot_sync(0xffffffffu, a0) & (1u << (m0 + i));
                        acc0 |= bit;
                        x0 += bit ? dc[i] : ba[i];
                    }
                }
            } else {
                for (int m = 0; m < na; m++) {
                    const float2 q0 = m < lane ? row0[m] : make_float2(0.0f, 0.0f);
                    const float2 q1 = v1 && m < lane + 32 ? row1[m] : make_float2(0.0f, 0.0f);
                    const double ba0 = (double)q0.x, dc0 = (double)q0.y, ba1 = (double)q1.x, dc1 = (double)q1.y;
                    const double xm = m < 32 ? x0 : x1;
                    const bool am = (m < 32 ? go0 : go1) && ((xm <= 0.0) || ((m < 32 ? lu0 : lu1) <= -beta * xm));
                    const unsigned bit = __ballot_sync(0xffffffffu, am) & (1u << (m & 31));
                    if (m < 32) acc0 |= bit;
                    else acc1 |= bit;
                    x0 += bit ? dc0 : ba0;
                    x1 += bit ? dc1 : ba1;
                }
            }
            if (v0) sm.acc[lane] = (acc0 >> lane) & 1u;
            if (v1) sm.acc[lane + 32] = (acc1 >> lane) & 1u;
            // colloid hard-core rejects (code 1) counted apart from moves that leave their cell (code 3)
            hc0 = __ballot_sync(0xffffffffu, v0 && sm.hard[lane] == 1);
            hc1 = __ballot_sync(0xffffffffu, v1 && sm.hard[lane + 32] == 1);
            if (v.rec_dE) {
                if (v0) {
                    v.rec_dE[p.p_off + v.id[g0 + lane]] = sm.hard[lane] ? 0.0 : x0;
                    v.rec_lu[p.p_off + v.id[g0 + lane]] = lu0;
                }
                if (v1) {
                    v.rec_dE[p.p_off + v.id[g0 + lane + 32]] = sm.hard[lane + 32] ? 0.0 : x1;
                    v.rec_lu[p.p_off + v.id[g0 + lane + 32]] = lu1;
                }
            }
        }
        pass_empty(an, nxt); // (here its record has long been loaded)
        const bool more = an < total;
        // (the list is read no more: every thread has passed the barrier after the task queue)
        if (w != 0) {
            if (w == 1 && more) {
                prepare_stencil<typename SM::Stencil, AMAX, CCAP>(v, sm.st[which ^ 1], nxt, lane);
                __syncwarp();
                copy_static(v, sm, which ^ 1, lane);
            }
            if (mode == 0 && kw < na) {
                const int g = g0 + kw;
                fetch_async<8>(&sm.wn[kw][0], v.tnx + g);
                fetch_async<8>(&sm.wn[kw][1], v.tny + g);
                fetch_async<8>(&sm.wn[kw][2], v.tnz + g);
                fetch_async<8>(&sm.wn[kw][3], v.tux + g);
                fetch_async<8>(&sm.wn[kw][4], v.tuy + g);
                fetch_async<8>(&sm.wn[kw][5], v.tuz + g);
            }
            if (more && kw < AMAX && kw < (int)((unsigned)nxt.z >> 24)) fetch_rec(&sm.next[kw], v.act_rec + nxt.w + kw);
        }
        if (mode >= 2 && t == 0) {
            if (RETRY) failed->cell[failed->n++] = cell * 4 + (mode == 2 ? 2 : 1);
            else if (mode == 2 && na <= p.cap) // above this kernel's capacity, not the class's
                v.retry_list[(size_t)ci * v.act_max + atomicAdd(&v.retry_count[ci], 1)] = a;
            else hand_over(v, ci, cell, mode == 2 ? 2 : 1);
        }
        __syncthreads();

        // ---- 6 write-back ----
        // Every thread's own fetches have landed before its cell ends, read or not: the next cell's list (and, after a
        // retry, the staged FP64 states) take the place of this cell's trial states, and the fetches of the cell after a
        // skipped one that of its records.
        fetch_wait();
        if (mode == 0 && kw >= 0 && kw < na) {
            const int k = kw, g = g0 + k;
            const int acc = sm.acc[k];
            if (acc) {
                v.px[g] = sm.wn[k][0];
                v.py[g] = sm.wn[k][1];
                v.pz[g] = sm.wn[k][2];
                v.ox[g] = sm.wn[k][3];
                v.oy[g] = sm.wn[k][4];
                v.oz[g] = sm.wn[k][5];
                const float4 P0 = sm.pst[k][0], P1 = sm.pst[k][1], P2 = sm.pst[k][2];
                v.cl4[g] = make_float4(P0.y, P0.w, P1.y, P1.w);
                v.cl2[g] = make_float2(P2.y, P2.w);
            }
            v.outcome[p.p_off + id] = sm.hard[k] == 1 ? 2 : acc;
        }
        // warp 0, while the others go on: the cell's results
        if (w == 0 && mode == 0) {
            // accepted dE summed in a fixed (butterfly) order
            double dsum = ((acc0 >> lane) & 1u ? x0 : 0.0) + ((acc1 >> lane) & 1u ? x1 : 0.0);
            double dabs = ((acc0 >> lane) & 1u ? fabs(x0) : 0.0) + ((acc1 >> lane) & 1u ? fabs(x1) : 0.0);
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                dsum += __shfl_xor_sync(0xffffffffu, dsum, o);
                dabs += __shfl_xor_sync(0xffffffffu, dabs, o);
            }
            const int nacc = __popc(acc0) + __popc(acc1), nhard = __popc(hc0) + __popc(hc1);
            if (lane == 0) {
                if (!(dsum - dsum == 0.0)) atomicOr(&v.stats[r].flags, F_NONFINITE);
                v.cell_e0[cell] = dsum;
                v.cell_abs[cell] = dabs;
                v.cell_fp64[cell] = 0;
                v.cell_n0[cell] = nacc;
                v.cell_n1[cell] = nhard;
                v.cell_pairs[cell] = sm.pairs;
                v.cell_cands[cell] = (unsigned long long)na * (unsigned long long)(s26 + na - 1);
            }
        }
        if (!more) break;
        rec = nxt;
        a = an;
        an += step;
        if (an < total) nxt = entry(an);
        which ^= 1;
    }
    if (RETRY) { // the block comes back with the barrier's memory
        __syncthreads();
        if (t == 0) asm volatile("mbarrier.inval.shared.b64 [%0];" ::"r"(tc::smem_u32(&sm.full)) : "memory");
    }
}

template <int NT, int MINB, int AMAX, int CCAP, int LCAP, bool SPEC21, bool ONE_K>
__global__ void __launch_bounds__(NT, MINB)
    k_phase_fast(const __grid_constant__ DevView v, const __grid_constant__ FastK ku, int ci)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int *off = v.act_off + ci * (v.R + 1); // this launch's replicas: active cells [off[r_lo], off[r_hi])
    phase_fast_body<NT, AMAX, CCAP, LCAP, SPEC21, ONE_K, false>(v, ku, ci, smem_raw, off[v.r_lo] + (int)blockIdx.x,
                                                                off[v.r_hi], (int)gridDim.x, nullptr);
}

// FP64 attempts of the cells the FP32 phase kernel handed over in colour phase
// ci (a pair term above f_big: an overlap, where FP32 rounding of R^12
// exceeds every energy scale; or a cell above the kernel's capacity), block
// per cell, sequentially in the in-cell order (ascending id) from the
// phase-start state, with the trial moves the gather drew (tn*, tu*, tdU, tlu,
// thard): E_old and E_new of each attempt are sums of the FP64 pair term
// (pair_exact; its lighter form for mu = 2, nu = 1, sigma0 = 1) over the 27
// stencil cells' particles read from the FP64 master arrays (earlier accepted
// in-cell moves already written), one-fold minimum image, every thread of the
// block over the candidates, then a fixed-order block sum.
// dE = (E_new - E_old) + dU_colloid, accepted if dE <= 0 or ln u <= -beta dE
// (MCnptColloid.c:2491-2574).  The FP32 state copy of an accepted particle is
// written exactly as the FP32 kernel writes it.  The stencil's FP64 states
// are staged in shared memory once per cell (the own cell's entries updated
// as moves are accepted) when they fit in RESCUE_CAP particles, what the retry's
// shared memory holds; a larger stencil is read from global memory, so any cell
// count works.  A block takes its next cell from a counter: one that ran a
// retry, and the cell's FP64 attempts after it, takes fewer of the others
// (100,000 rods, displacements up to 1.0, 330 cells handed over in a phase and
// 28 run again: phases 5.45 ms a sweep with 1024 staged particles and every
// 148th cell, 3.98 now; 30,000 rods on a lattice, turned at random, 3.39 -> 2.19).  The other
// cells of the colour do not interact with these, so running them after the
// FP32 kernel changes nothing in the chain.
#define FAST_RETRY 64, 1664, 7168 // active particles, places of the static cells' particles, list entries
constexpr int RESCUE_CAP = (int)(sizeof(FastSmem<FAST_RETRY>) / (6 * sizeof(double))); // particles of a staged stencil

template <int NT, bool SPEC21>
__global__ void __launch_bounds__(NT) k_phase_rescue(const __grid_constant__ DevView v, int ci)
{
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *sx = reinterpret_cast<double *>(smem_raw); // [6][RESCUE_CAP]: x, y, z, ux, uy, uz of the staged stencil
    __shared__ int st_start[27], st_cnt[27], pre[28];
    __shared__ double spo[NW], spn[NW];
    __shared__ int snp[NW];
    __shared__ RetryFailed failed;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int nretry = v.retry_count[ci], count = v.resc_count[ci];
    if (nretry == 0 && count == 0) return;
    if (t == 0) failed.n = 0;
    __syncthreads();
    // Rounds of at most 32 retries of this block, each followed by the FP64 attempts of those that failed; then the
    // cells the phase kernel handed over.
    for (int a0 = blockIdx.x, f = 0;;) {
        if (f == failed.n && a0 < nretry) { // (uniform, as all choices here)
            __syncthreads();
            if (t == 0) failed.n = 0;
            f = 0;
            tc::fence_proxy_async_smem(); // the staged states of the last round's cells come before this round's copies
            __syncthreads();
            phase_fast_body<NT, FAST_RETRY, SPEC21, false, true>(v, FastK(), ci, smem_raw, a0,
                                                                 min(nretry, a0 + 32 * (int)gridDim.x), (int)gridDim.x, &failed);
            a0 += 32 * gridDim.x;
            __syncthreads();
            continue;
        }
        {
            int code;
            if (f < failed.n) {
                code = failed.cell[f++];
            } else {
                if (t == 0) failed.ticket = atomicAdd(&v.resc_next[ci], 1);
                __syncthreads();
                if (failed.ticket >= count) break;
                code = v.resc_list[(size_t)ci * v.ctot + failed.ticket];
            }
            const int cell = code >> 2, mode = code & 3;
            const int r = v.p2c[cell];
            const Replica &p = v.rep[r];
            const int nc0 = p.nc[0], nc1 = p.nc[1], nc2 = p.nc[2];
            const int loc = cell - p.cell_off;
            const int cx = loc % nc0, cy = (loc / nc0) % nc1, cz = loc / (nc0 * nc1);
            if (t < 27) {
                int x = cx + t % 3 - 1, y = cy + (t / 3) % 3 - 1, z = cz + t / 9 - 1;
                x += x < 0 ? nc0 : (x >= nc0 ? -nc0 : 0);
                y += y < 0 ? nc1 : (y >= nc1 ? -nc1 : 0);
                z += z < 0 ? nc2 : (z >= nc2 ? -nc2 : 0);
                const int c = p.cell_off + (z * nc1 + y) * nc0 + x;
                st_start[t] = v.cell_start[c];
                st_cnt[t] = v.cell_start[c + 1] - v.cell_start[c];
            }
            __syncthreads();
            if (t < 32) {
                const int c = t < 27 ? st_cnt[t] : 0;
                int inc = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += y;
                }
                if (t < 27) pre[t] = inc - c;
                if (t == 26) pre[27] = inc;
            }
            __syncthreads();
            const int total = pre[27];
            const int g0 = st_start[13], na = st_cnt[13];
            const bool staged = total <= RESCUE_CAP;
            if (staged) {
                for (int f = t; f < total; f += NT) {
                    int sl = 0, hi = 27;
                    while (hi - sl > 1) {
                        const int mid = (sl + hi) >> 1;
                        if (pre[mid] <= f) sl = mid;
                        else hi = mid;
                    }
                    const int j = st_start[sl] + (f - pre[sl]);
                    sx[f] = v.px[j];
                    sx[RESCUE_CAP + f] = v.py[j];
                    sx[2 * RESCUE_CAP + f] = v.pz[j];
                    sx[3 * RESCUE_CAP + f] = v.ox[j];
                    sx[4 * RESCUE_CAP + f] = v.oy[j];
                    sx[5 * RESCUE_CAP + f] = v.oz[j];
                }
                __syncthreads();
            }
            double dsum = 0.0, dabs = 0.0;
            int nacc = 0, nhard = 0;
            unsigned long long npairs = 0ull;
            for (int k = 0; k < na; k++) {
                const int g = g0 + k;
                const int id = v.id[g];
                const unsigned char code = v.thard[g];
                if (code) { // colloid hard-core reject (1) or a move out of the cell (3): no energy evaluation
                    if (t == 0) {
                        v.outcome[p.p_off + id] = code == 1 ? 2 : 0;
                        if (v.rec_dE) {
                            v.rec_dE[p.p_off + id] = 0.0;
                            v.rec_lu[p.p_off + id] = v.tlu[g];
                        }
                    }
                    nhard += code == 1;
                    continue;
                }
                const double ro[3] = {v.px[g], v.py[g], v.pz[g]};
                const double eo[3] = {v.ox[g], v.oy[g], v.oz[g]};
                const double rn[3] = {v.tnx[g], v.tny[g], v.tnz[g]};
                const double en[3] = {v.tux[g], v.tuy[g], v.tuz[g]};
                double po = 0.0, pn = 0.0;
                int np = 0;
                const int fk = pre[13] + k; // this particle's own entry
                for (int f = t; f < total; f += NT) {
                    if (f == fk) continue;
                    double rj[3], ej[3];
                    if (staged) {
                        rj[0] = sx[f], rj[1] = sx[RESCUE_CAP + f], rj[2] = sx[2 * RESCUE_CAP + f];
                        ej[0] = sx[3 * RESCUE_CAP + f], ej[1] = sx[4 * RESCUE_CAP + f], ej[2] = sx[5 * RESCUE_CAP + f];
                    } else {
                        int sl = 0, hi = 27;
                        while (hi - sl > 1) {
                            const int mid = (sl + hi) >> 1;
                            if (pre[mid] <= f) sl = mid;
                            else hi = mid;
                        }
                        const int j = st_start[sl] + (f - pre[sl]);
                        rj[0] = v.px[j], rj[1] = v.py[j], rj[2] = v.pz[j];
                        ej[0] = v.ox[j], ej[1] = v.oy[j], ej[2] = v.oz[j];
                    }
                    double d[3];
                    double r2 = dist_fold(ro[0], ro[1], ro[2], rj[0], rj[1], rj[2], p.L, d);
                    if (r2 < p.k.rc2) {
                        po += SPEC21 ? pair_energy64_21(p.k, r2, d, eo, ej) : pair_exact(p.k, r2, d, eo, ej);
                        np++;
                    }
                    r2 = dist_fold(rn[0], rn[1], rn[2], rj[0], rj[1], rj[2], p.L, d);
                    if (r2 < p.k.rc2) {
                        pn += SPEC21 ? pair_energy64_21(p.k, r2, d, en, ej) : pair_exact(p.k, r2, d, en, ej);
                        np++;
                    }
                }
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) {
                    po += __shfl_xor_sync(0xffffffffu, po, o);
                    pn += __shfl_xor_sync(0xffffffffu, pn, o);
                    np += __shfl_xor_sync(0xffffffffu, np, o);
                }
                if (lane == 0) {
                    spo[w] = po;
                    spn[w] = pn;
                    snp[w] = np;
                }
                __syncthreads();
                if (t == 0) {
                    double so = spo[0], sn = spn[0];
                    int sp = snp[0];
                    for (int q = 1; q < NW; q++) {
                        so += spo[q];
                        sn += spn[q];
                        sp += snp[q];
                    }
                    const double dE = (sn - so) + v.act_rec[g].tdU;
                    const double lu = v.tlu[g];
                    const bool acc = (dE <= 0.0) || (lu <= -p.k.beta * dE);
                    if (acc) {
                        v.px[g] = rn[0];
                        v.py[g] = rn[1];
                        v.pz[g] = rn[2];
                        v.ox[g] = en[0];
                        v.oy[g] = en[1];
                        v.oz[g] = en[2];
                        if (staged) {
                            const int fk = pre[13] + k;
                            sx[fk] = rn[0], sx[RESCUE_CAP + fk] = rn[1], sx[2 * RESCUE_CAP + fk] = rn[2];
                            sx[3 * RESCUE_CAP + fk] = en[0], sx[4 * RESCUE_CAP + fk] = en[1], sx[5 * RESCUE_CAP + fk] = en[2];
                        }
                        const ActRec &ar = v.act_rec[g];
                        v.cl4[g] = make_float4(ar.p0.y, ar.p0.w, ar.p1.y, ar.p1.w);
                        v.cl2[g] = make_float2(ar.p2.y, ar.p2.w);
                        dsum += dE;
                        dabs += fabs(dE);
                        nacc++;
                    }
                    v.outcome[p.p_off + id] = acc ? 1 : 0;
                    if (v.rec_dE) {
                        v.rec_dE[p.p_off + id] = dE;
                        v.rec_lu[p.p_off + id] = lu;
                    }
                    npairs += (unsigned long long)sp;
                }
                __syncthreads(); // the accepted state is visible to the next attempt
            }
            if (t == 0) {
                if (!(dsum - dsum == 0.0)) atomicOr(&v.stats[r].flags, F_NONFINITE);
                v.cell_e0[cell] = dsum;
                v.cell_abs[cell] = dabs;
                v.cell_n0[cell] = nacc;
                v.cell_n1[cell] = nhard;
                v.cell_pairs[cell] = npairs;
                v.cell_cands[cell] = (unsigned long long)na * (unsigned long long)(total > 0 ? total - 1 : 0);
                v.cell_fp64[cell] = mode;
            }
            __syncthreads();
        }
    }
}

} // namespace lcmc

#include "lcmc_launch.h"

namespace lcmc {

// Capacity classes: (active particles, places of the static cells' particles, list entries).
// "Light" is the 48-particle class for systems whose capacity rule asks for at most 40, "sparse" for gases.
#define FAST32 32, 336, 2048
#define FAST40 40, 780, 2688
#define FAST48 48, 832, 3456
#define FAST56 56, 1040, 4096
#define FAST64 64, 1440, 5376
static_assert(sizeof(FastSmem<FAST32>) + 1024 <= 233472 / 10, "sparse: ten blocks per SM");
static_assert(sizeof(FastSmem<FAST40>) + 1024 <= 233472 / 6, "light: six blocks per SM");
static_assert(sizeof(FastSmem<FAST48>) + 1024 <= 233472 / 5, "48-class: five blocks per SM");
static_assert(sizeof(FastSmem<FAST56>) + 1024 <= 233472 / 4, "56-class: four blocks per SM");
static_assert(sizeof(FastSmem<FAST64>) + 1024 <= 233472 / 3, "64-class: three blocks per SM");
static const FastVariant kVariants[] = {{48}, {56}, {64}};

int fast_variant_count() { return (int)(sizeof(kVariants) / sizeof(kVariants[0])); }
FastVariant fast_variant(int i) { return kVariants[i]; }

static constexpr int shape_candidates(int, int ccap, int) { return ccap; }
int fast_shape_candidates(int shape)
{
    constexpr int n[FAST_SHAPES] = {shape_candidates(FAST32), shape_candidates(FAST40), shape_candidates(FAST48), shape_candidates(FAST56),
                                    shape_candidates(FAST64)};
    return n[shape];
}

template <int NT, int MINB, int AMAX, int CCAP, int LCAP, bool S21, bool K1>
struct FastLaunch {
    static constexpr int bytes = (int)sizeof(FastSmem<AMAX, CCAP, LCAP>);
    static void launch(const DevView &v, const FastK &k, cudaStream_t s, int ci, int grid)
    {
        k_phase_fast<NT, MINB, AMAX, CCAP, LCAP, S21, K1><<<grid, NT, bytes, s>>>(v, k, ci);
    }
    static int blocks()
    {
        auto k = k_phase_fast<NT, MINB, AMAX, CCAP, LCAP, S21, K1>;
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, NT, bytes);
        return n > 0 ? n : 1;
    }
};

// Threads: four warps per cell where a phase has more cells than SMs (1,048,576
// rods, all phases: 1.48 ms; three warps 1.60, five 1.53, six at five blocks
// 1.66), sixteen where it has not and a phase takes one cell's latency (32,768
// rods NPT: 0.19 ms against 0.30 with four).  The light shape holds six blocks
// per SM where the class's own 48-particle arrays leave five (1.48 against 1.60).
// The sparse one takes two warps per cell: the cells of a gas have a few particles
// with some hundred neighbours, and what counts is how many are in flight.
// The kernel of a variant: shape, wide (a block per SM), specialisation (mu = 2,
// nu = 1, sigma0 = 1; of that, whether all replicas have the same pair constants,
// which then come as a kernel argument).  Twelve systems of 30,000 rods of three
// kappas, all phases and the rest of a sweep: 1.26 ms with the general terms, 1.04
// with these and each replica's constants; 1.05 when all have one kappa.
template <typename F>
static auto with_variant(const FastChoice &c, F f)
{
#define FAST_SPEC(NT, MINB, ...)                                                                                       \
    (!c.spec21 ? f(FastLaunch<NT, MINB, __VA_ARGS__, false, false>())                                                  \
               : c.one_k ? f(FastLaunch<NT, MINB, __VA_ARGS__, true, true>()) : f(FastLaunch<NT, MINB, __VA_ARGS__, true, false>()))
#define FAST_PICK(MINB, ...) (c.wide ? FAST_SPEC(512, 1, __VA_ARGS__) : FAST_SPEC(128, MINB, __VA_ARGS__))
    if (c.shape == 0) return FAST_SPEC(64, 10, FAST32);
    if (c.shape == 1) return FAST_PICK(6, FAST40);
    if (c.shape == 2) return FAST_PICK(5, FAST48);
    if (c.shape == 3) return FAST_PICK(4, FAST56);
    return FAST_PICK(3, FAST64);
#undef FAST_PICK
#undef FAST_SPEC
}

void launch_phase_fast(const FastChoice &c, const GBConsts &k, const DevView &v, cudaStream_t s, int ci, int grid)
{
    const FastK K = fast_consts(k);
    with_variant(c, [&](auto l) {
        decltype(l)::launch(v, K, s, ci, grid);
        return 0;
    });
}

static constexpr int rescue_bytes()
{
    return std::max(6 * RESCUE_CAP * (int)sizeof(double), (int)sizeof(FastSmem<FAST_RETRY>));
}

void launch_phase_rescue(bool spec21, const DevView &v, cudaStream_t s, int ci, int grid)
{
    if (spec21) k_phase_rescue<256, true><<<grid, 256, rescue_bytes(), s>>>(v, ci);
    else k_phase_rescue<256, false><<<grid, 256, rescue_bytes(), s>>>(v, ci);
}

// Opts the hand-over kernel in to its dynamic shared memory (call once).
void rescue_init()
{
    const int bytes = rescue_bytes();
    cudaFuncSetAttribute(k_phase_rescue<256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    cudaFuncSetAttribute(k_phase_rescue<256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Also opts the kernel in to its dynamic shared memory size: call once
// before the first launch of a choice.
int fast_blocks_per_sm(const FastChoice &c)
{
    return with_variant(c, [](auto l) { return decltype(l)::blocks(); });
}

} // namespace lcmc
