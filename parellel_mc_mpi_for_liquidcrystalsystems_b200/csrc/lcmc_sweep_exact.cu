// lcmc_sweep_exact.cu - FP64 checkerboard phase, bit-identical to the CPU oracle.
//
// Compiled with -fmad=false: every double operation is a single IEEE-rounded
// +, -, *, / or sqrt, in the order of the reference's pij_GB / GBCollRod
// (MCnptColloid.c:2607-2681, 1758-1854), so the accept/reject sequence equals
// the oracle's canonical sweep.
//
// The particles of a cell are attempted one after another in ascending id (the
// reference picks a random particle per cycle, MCnptColloid.c:2475; its MPI path
// loops over an active subcell's particles, 683-700).  For each attempt the 32
// lanes of a warp split the stencil slots q (q mod 32), sum the old and new pair
// energies lane-locally in q order and combine them with a xor butterfly: the
// canonical order the oracle reproduces.
#include <cuda_runtime.h>

#include <algorithm>

#include "lcmc_gb.cuh"
#include "lcmc_internal.h"
#include "lcmc_launch.h"
#include "lcmc_rng.cuh"
#include "lcmc_tc.cuh"
#include "lcmc_trial.cuh"
#include "lcmc_volume_cells.cuh"

namespace lcmc {

__device__ __forceinline__ int find_replica(const int *off, int R, int a)
{
    int lo = 0, hi = R;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (off[mid] <= a) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ double warp_sum_butterfly(double x)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) x = x + __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// An active cell and its stencil, as one warp holds it: kept cells and the
// prefix of their counts in shared memory, canonical order (dz, dy, dx =
// -1..1, duplicates of small grids dropped at their first occurrence).
struct CellView {
    int r, cell, cx, cy, cz;
    int ncell; // kept stencil cells
    int total; // particles in them (the cell's own included)
    int own;   // kept slot of the cell itself
    int cs, na; // first slot and count of its particles
};

// Active cell a (of the colour-phase enumeration) -> replica and coordinates.
__device__ __forceinline__ void active_cell(const DevView &v, const int *off, int ci, int a, CellView &c)
{
    c.r = find_replica(off, v.R, a);
    const Replica &p = v.rep[c.r];
    const int col = p.perm[ci];
    const int bx = col % p.kc[0], by = (col / p.kc[0]) % p.kc[1], bz = col / (p.kc[0] * p.kc[1]);
    const int nc0 = p.nc[0], nc1 = p.nc[1], nc2 = p.nc[2];
    const int nax = axis_colour_count(nc0, p.kc[0], bx), nay = axis_colour_count(nc1, p.kc[1], by);
    int loc = a - off[c.r];
    c.cx = axis_colour_cell(nc0, p.kc[0], bx, loc % nax);
    loc /= nax;
    c.cy = axis_colour_cell(nc1, p.kc[1], by, loc % nay);
    c.cz = axis_colour_cell(nc2, p.kc[2], bz, loc / nay);
    c.cell = p.cell_off + (c.cz * nc1 + c.cy) * nc0 + c.cx;
    c.cs = v.cell_start[c.cell];
    c.na = v.cell_start[c.cell + 1] - c.cs;
}

// The stencil of c (every lane of the warp): s_first[k] = first particle slot
// of kept cell k, s_base[k] = its prefix (s_base[ncell] = total).
__device__ __forceinline__ void cell_stencil(const DevView &v, CellView &c, int lane, int *s_first, int *s_base)
{
    const Replica &p = v.rep[c.r];
    const int nc0 = p.nc[0], nc1 = p.nc[1], nc2 = p.nc[2];
    int cc = -1;
    if (lane < 27) {
        const int dz = lane / 9 - 1, dy = (lane / 3) % 3 - 1, dx = lane % 3 - 1;
        const int x = (c.cx + dx + nc0) % nc0, y = (c.cy + dy + nc1) % nc1, z = (c.cz + dz + nc2) % nc2;
        cc = p.cell_off + (z * nc1 + y) * nc0 + x;
    }
    const unsigned same = __match_any_sync(0xffffffffu, cc);
    const bool keep = lane < 27 && (__ffs(same) - 1) == lane;
    const unsigned kb = __ballot_sync(0xffffffffu, keep);
    const unsigned ob = __ballot_sync(0xffffffffu, keep && cc == c.cell);
    c.ncell = __popc(kb);
    c.own = __popc(kb & ((ob & (0u - ob)) - 1u));
    const int slot = __popc(kb & ((1u << lane) - 1u));
    int first = 0, cnt = 0;
    if (keep) {
        first = v.cell_start[cc];
        cnt = v.cell_start[cc + 1] - first;
    }
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    __syncwarp();
    if (keep) {
        s_first[slot] = first;
        s_base[slot] = inc - cnt;
    }
    c.total = __shfl_sync(0xffffffffu, inc, 31);
    if (lane == 0) s_base[c.ncell] = c.total;
    __syncwarp();
}

// ---------------------------------------------------------------------------
// FP64 colour phase in two kernels.
//
// What bounds it: the attempts of a cell follow one another, so a warp that
// walks the stencil for each attempt in turn spends its time in the latency of
// FP64 distances, divisions and square roots with most of the GPU idle (one
// warp per active cell: a 1000-rod box has one active cell in a phase).  But
// only the choice between terms depends on the earlier attempts, not the terms:
// particle k sees static cells, and each in-cell partner m in its old state or,
// if m < k was accepted, in its trial state, which is known before the phase
// (the gather drew every trial move).  So
//   k_exact_terms   block per active particle, all cells at once: distances to
//                   every stencil slot, the in-cutoff terms of the old and the
//                   trial state through a compacted list with all lanes busy,
//                   then the lane sums of the canonical order as far as they do
//                   not depend on a decision;
//   k_exact_decide  block per cell: for each attempt in ascending id, the lane
//                   sums completed with the chosen in-cell terms and the static
//                   terms after them, the xor butterfly, the Metropolis test.
// Phases per sweep: 1000 rods 38 -> 0.48 ms, 8192 rods 16.7 -> 0.35 ms.
// The order of every FP64 addition is the canonical one (lane q mod 32 adds the
// stencil slots q in increasing q; a term beyond the cutoff adds +0.0, which
// changes no bit), so outcomes and energies equal the CPU oracle's bit for bit.
//
// Record of particle k, rows of 32 double2 (lane = q mod 32, x = old state of k,
// y = its trial state):
//   0            ExactHead
//   1            sums over the static slots before the own cell
//   2 .. 1+J     own-cell slots, partner in its old state (J chunks of 32 slots)
//   2+J .. 1+2J  own-cell slots, partner in its trial state
//   2+2J ..      the lane's static terms after the own cell, in order (nsuf rows, a
//                multiple of four; zeros at the end)
// The records of a phase lie in a scratch of ex_cap rows; a phase with more is
// run in ex_nb batches of cells.  A cell above a capacity (particles, stencil,
// in-cutoff terms, terms after the own cell in one lane) is attempted by
// k_exact_decide the sequential way (exact_cell_sequential).
// The stencil's and the terms' capacity reach to cutoffs of 5 and 6 in a liquid: 8000
// rods at 0.30 and a cutoff of 5, 125 in a cell, 101 -> 0.97 ms of phases a sweep
// (96 chunks and 640 terms before; one warp per cell without records 88); the
// arrays cost the terms kernel no resident block.
// ---------------------------------------------------------------------------
constexpr int EX_NA = 256;   // particles of a cell
constexpr int EX_CH = 128;   // chunks of 32 stencil slots
constexpr int EX_ENT = 1024; // in-cutoff terms of a particle
constexpr int EX_SUF = 12;   // static terms after the own cell, per lane
constexpr int EX_J = 9;      // most chunks an own cell touches

// chunks of 32 slots that na consecutive slots can touch, rounded up to a class
// (2, 3, 5, 9) the decisions are unrolled for (chunks beyond the cell's are empty)
__host__ __device__ __forceinline__ int ex_chunks(int na) { return na <= 33 ? 2 : (na <= 65 ? 3 : (na <= 129 ? 5 : EX_J)); }
__host__ __device__ __forceinline__ int ex_rows_per_particle(int na) { return 2 + 2 * ex_chunks(na) + EX_SUF; }

struct ExactHead {
    double uo, un, lu;          // colloid term of the old and the trial state, log of the Metropolis draw
    int code, nsuf, nstat, pad; // trial code (thard), suffix rows, in-cutoff static terms
    unsigned mask[4][EX_J];     // in-cutoff own-cell slots per chunk: (old, old), (trial, old), (old, trial), (trial, trial)
};
static_assert(sizeof(ExactHead) <= 512, "one row");

// Per phase: exclusive prefix of the particles and of the record rows over the
// active cells of replicas on the FP64 kernel.  Block per phase.
__global__ void __launch_bounds__(1024) k_exact_offsets(DevView v)
{
    const int ci = blockIdx.x, t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int *off = v.act_off + ci * (v.R + 1);
    const int total = off[v.R];
    int *ep = v.ex_p + (size_t)ci * (v.ex_act + 1);
    long long *er = v.ex_r + (size_t)ci * (v.ex_act + 1);
    unsigned char *fl = v.ex_flag + (size_t)ci * v.ex_act;
    __shared__ long long sp[32], sr[32];
    long long bp = 0, br = 0;
    for (int b = 0; b < total; b += 1024) {
        const int a = b + t;
        long long np = 0, nr = 0;
        if (a < total) {
            CellView c;
            active_cell(v, off, ci, a, c);
            const bool mine = !v.rep[c.r].use_fast;
            const bool fits = c.na <= EX_NA;
            if (mine && fits) {
                np = c.na;
                nr = (long long)c.na * ex_rows_per_particle(c.na);
            }
            fl[a] = mine && !fits;
        }
        long long ip = np, ir = nr;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, ip, o), z = __shfl_up_sync(0xffffffffu, ir, o);
            if (lane >= o) {
                ip += y;
                ir += z;
            }
        }
        if (lane == 31) {
            sp[w] = ip;
            sr[w] = ir;
        }
        __syncthreads();
        long long op = bp, orr = br;
        for (int q = 0; q < 32; q++) {
            if (q < w) {
                op += sp[q];
                orr += sr[q];
            }
            bp += sp[q];
            br += sr[q];
        }
        if (a < total) {
            ep[a] = (int)(op + ip - np);
            er[a] = orr + ir - nr;
        }
        __syncthreads();
    }
    if (t == 0) {
        ep[total] = (int)bp;
        er[total] = br;
    }
}

// first a in [lo, hi) with x[a] >= key, else hi
template <typename T, typename K>
__device__ __forceinline__ int lower_bound_dev(const T *x, int lo, int hi, K key)
{
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((K)x[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

struct ExactBatch {
    int lo, hi;     // active cells of this batch
    long long row0; // row prefix that is scratch row 0
};

__device__ __forceinline__ ExactBatch exact_batch(const DevView &v, const int *off, const long long *er, int b)
{
    ExactBatch e;
    const int a0 = off[v.r_lo], a1 = off[v.r_hi];
    const long long r0 = er[a0];
    e.row0 = r0 + (long long)b * v.ex_cap;
    e.lo = b == 0 ? a0 : lower_bound_dev(er, a0, a1, e.row0);
    e.hi = lower_bound_dev(er, a0, a1, e.row0 + (long long)v.ex_cap);
    return e;
}

__global__ void __launch_bounds__(128) k_exact_terms(const __grid_constant__ DevView v, int ci, int b)
{
    phase_begin();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    __shared__ int s_first[27], s_base[28];
    __shared__ unsigned s_mask[4][EX_CH];
    __shared__ unsigned short s_off[EX_CH];
    __shared__ int s_ent[EX_ENT];
    __shared__ double s_val[EX_ENT];
    __shared__ int s_ne, s_nstat;
    __shared__ CellView s_c;
    const int *off = v.act_off + ci * (v.R + 1);
    const int *ep = v.ex_p + (size_t)ci * (v.ex_act + 1);
    const long long *er = v.ex_r + (size_t)ci * (v.ex_act + 1);
    const ExactBatch eb = exact_batch(v, off, er, b);
    const int p_hi = ep[eb.hi];
    for (int idx = ep[eb.lo] + blockIdx.x; idx < p_hi; idx += gridDim.x) {
        // the last active cell whose prefix is <= idx (cells without particles share their successor's prefix)
        const int a = lower_bound_dev(ep, eb.lo, eb.hi, idx + 1) - 1;
        if (w == 0) {
            CellView c;
            active_cell(v, off, ci, a, c);
            cell_stencil(v, c, lane, s_first, s_base);
            if (lane == 0) {
                s_c = c;
                s_ne = 0;
                s_nstat = 0;
            }
        }
        __syncthreads();
        const CellView c = s_c;
        const Replica &p = v.rep[c.r];
        const int k = idx - ep[a], g = c.cs + k;
        double2 *rec = v.ex_rows + ((size_t)(er[a] - eb.row0) + (size_t)k * ex_rows_per_particle(c.na)) * 32;
        ExactHead *hd = reinterpret_cast<ExactHead *>(rec);
        const int code = v.thard[g];
        if (t == 0) {
            hd->code = code;
            hd->lu = v.tlu[g];
        }
        const int nch = (c.total + 31) >> 5;
        // a trial in the colloid or out of its cell is never evaluated
        if (code || nch > EX_CH) { // (uniform)
            if (t == 0 && !code) v.ex_flag[(size_t)ci * v.ex_act + a] = 1;
            __syncthreads();
            continue;
        }
        const double ro[3] = {v.px[g], v.py[g], v.pz[g]};
        const double rn[3] = {v.tnx[g], v.tny[g], v.tnz[g]};
        const double rc2 = p.k.rc2;
        const int q13 = s_base[c.own];
        // 1 distances, a chunk of 32 slots per warp: in-cutoff terms appended to the list, masks per chunk
        int sc = 0, nstat = 0;
        for (int h = w; h < nch; h += 4) {
            const int q = 32 * h + lane;
            bool f0 = false, f1 = false, f2 = false, f3 = false;
            int j = 0;
            if (q < c.total) {
                while (s_base[sc + 1] <= q) sc++;
                j = s_first[sc] + (q - s_base[sc]);
                if (j != g) {
                    double d[3];
                    const double xj = v.px[j], yj = v.py[j], zj = v.pz[j];
                    f0 = dist_fold(ro[0], ro[1], ro[2], xj, yj, zj, p.L, d) < rc2;
                    f1 = dist_fold(rn[0], rn[1], rn[2], xj, yj, zj, p.L, d) < rc2;
                    if (sc == c.own && j < g && v.thard[j] == 0) { // partner's trial state
                        const double xt = v.tnx[j], yt = v.tny[j], zt = v.tnz[j];
                        f2 = dist_fold(ro[0], ro[1], ro[2], xt, yt, zt, p.L, d) < rc2;
                        f3 = dist_fold(rn[0], rn[1], rn[2], xt, yt, zt, p.L, d) < rc2;
                    }
                    if (sc != c.own) nstat += (int)f0 + (int)f1;
                }
            }
            const unsigned b0 = __ballot_sync(0xffffffffu, f0), b1 = __ballot_sync(0xffffffffu, f1);
            const unsigned b2 = __ballot_sync(0xffffffffu, f2), b3 = __ballot_sync(0xffffffffu, f3);
            const int n0 = __popc(b0), n1 = __popc(b1), n2 = __popc(b2), n3 = __popc(b3);
            int ne = 0;
            if (lane == 0) ne = atomicAdd(&s_ne, n0 + n1 + n2 + n3);
            ne = __shfl_sync(0xffffffffu, ne, 0);
            if (ne + n0 + n1 + n2 + n3 <= EX_ENT) {
                if (f0) s_ent[ne + __popc(b0 & lt)] = j;
                if (f1) s_ent[ne + n0 + __popc(b1 & lt)] = j | (1 << 30);
                if (f2) s_ent[ne + n0 + n1 + __popc(b2 & lt)] = j | (int)(2u << 30);
                if (f3) s_ent[ne + n0 + n1 + n2 + __popc(b3 & lt)] = j | (int)(3u << 30);
            }
            if (lane == 0) {
                s_mask[0][h] = b0;
                s_mask[1][h] = b1;
                s_mask[2][h] = b2;
                s_mask[3][h] = b3;
                s_off[h] = (unsigned short)ne;
            }
        }
        nstat = __reduce_add_sync(0xffffffffu, nstat);
        if (lane == 0 && nstat) atomicAdd(&s_nstat, nstat);
        __syncthreads();
        const int ne = s_ne;
        if (ne > EX_ENT) { // (uniform)
            if (t == 0) v.ex_flag[(size_t)ci * v.ex_act + a] = 1;
            __syncthreads();
            continue;
        }
        // 2 the listed terms, every lane busy
        for (int e = t; e < ne; e += 128) {
            const unsigned u = (unsigned)s_ent[e];
            const int j = (int)(u & 0x3fffffffu);
            const bool nk = u & (1u << 30), nj = u & (2u << 30);
            const double ri[3] = {nk ? rn[0] : ro[0], nk ? rn[1] : ro[1], nk ? rn[2] : ro[2]};
            const double ei[3] = {nk ? v.tux[g] : v.ox[g], nk ? v.tuy[g] : v.oy[g], nk ? v.tuz[g] : v.oz[g]};
            const double rj[3] = {nj ? v.tnx[j] : v.px[j], nj ? v.tny[j] : v.py[j], nj ? v.tnz[j] : v.pz[j]};
            const double ej[3] = {nj ? v.tux[j] : v.ox[j], nj ? v.tuy[j] : v.oy[j], nj ? v.tuz[j] : v.oz[j]};
            double d[3];
            const double r2 = dist_fold(ri[0], ri[1], ri[2], rj[0], rj[1], rj[2], p.L, d);
            s_val[e] = pair_exact(p.k, r2, d, ei, ej);
        }
        // colloid terms: the old state and the trial state
        if (t >= 126 && p.k.coll_on) {
            const bool nk = t & 1;
            const double r3[3] = {nk ? rn[0] : ro[0], nk ? rn[1] : ro[1], nk ? rn[2] : ro[2]};
            const double e3[3] = {nk ? v.tux[g] : v.ox[g], nk ? v.tuy[g] : v.oy[g], nk ? v.tuz[g] : v.oz[g]};
            const double u = colloid_rod(p.k, r3, e3, p.L);
            if (nk) hd->un = u;
            else hd->uo = u;
        }
        __syncthreads();
        // 3 the lane sums, in slot order: warp 0 the slots before the own cell, warp 1 the own cell's, warp 2 those after
        const int J = ex_chunks(c.na);
        const int c0 = q13 >> 5, q14 = q13 + c.na, c1 = (q14 - 1) >> 5;
        auto term = [&](unsigned m, int o) { return (m >> lane) & 1u ? s_val[o + __popc(m & lt)] : 0.0; };
        if (w == 0) {
            double po = 0.0, pn = 0.0;
            for (int h = 0; h <= c0; h++) {
                unsigned b0 = s_mask[0][h], b1 = s_mask[1][h];
                const int o = s_off[h];
                const double t0 = term(b0, o), t1 = term(b1, o + __popc(b0));
                if (32 * h + lane < q13) {
                    po += t0;
                    pn += t1;
                }
            }
            rec[32 + lane] = make_double2(po, pn);
        } else if (w == 1) {
            for (int h = c0; h < c0 + J; h++) { // chunks beyond the last one the cell touches are written as empty
                const int q = 32 * h + lane;
                const bool mine = q >= q13 && q < q14;
                const unsigned own = __ballot_sync(0xffffffffu, mine);
                unsigned m[4] = {0u, 0u, 0u, 0u};
                double x[4] = {0.0, 0.0, 0.0, 0.0};
                if (h <= c1) {
                    int o = s_off[h];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        m[i] = s_mask[i][h];
                        x[i] = mine ? term(m[i], o) : 0.0;
                        o += __popc(m[i]);
                    }
                }
                rec[(size_t)(2 + h - c0) * 32 + lane] = make_double2(x[0], x[1]);
                rec[(size_t)(2 + J + h - c0) * 32 + lane] = make_double2(x[2], x[3]);
                if (lane < 4) {
                    const unsigned mm = lane == 0 ? m[0] : (lane == 1 ? m[1] : (lane == 2 ? m[2] : m[3]));
                    hd->mask[lane][h - c0] = mm & own;
                }
            }
        } else if (w == 2) {
            int ns = 0;
            double2 *suf = rec + (size_t)(2 + 2 * J) * 32;
            for (int h = c1; h < nch; h++) {
                const unsigned b0 = s_mask[0][h], b1 = s_mask[1][h];
                const int o = s_off[h];
                if (32 * h + lane >= q14 && (((b0 | b1) >> lane) & 1u)) {
                    if (ns < EX_SUF) suf[(size_t)ns * 32 + lane] = make_double2(term(b0, o), term(b1, o + __popc(b0)));
                    ns++;
                }
            }
            const int nsuf = __reduce_max_sync(0xffffffffu, ns);
            if (nsuf > EX_SUF) {
                if (lane == 0) v.ex_flag[(size_t)ci * v.ex_act + a] = 1;
            } else {
                const int nsuf4 = (nsuf + 3) & ~3; // the decisions take them four at a time
                for (int s = ns; s < nsuf4; s++) suf[(size_t)s * 32 + lane] = make_double2(0.0, 0.0);
                if (lane == 0) {
                    hd->nsuf = nsuf4;
                    hd->nstat = s_nstat;
                }
            }
        }
        __syncthreads();
    }
}

// One cell attempted by one warp, attempt after attempt: for every particle
// the lanes split the stencil slots, evaluate the terms where they are found
// and combine the lane sums (the canonical order again).  For cells above a
// capacity of the two-kernel path.
__device__ __forceinline__ void exact_cell_sequential(const DevView *__restrict__ vp, const CellView &c, int lane,
                                                      const int *s_first, const int *s_base)
{
    const DevView &v = *vp;
    const Replica &p = v.rep[c.r];
    // (held in registers: the stores of the accepted states might change them, for all the compiler knows)
    double *const px = v.px, *const py = v.py, *const pz = v.pz, *const ox = v.ox, *const oy = v.oy, *const oz = v.oz;
    const double L[3] = {p.L[0], p.L[1], p.L[2]};
    const GBConsts k = p.k;
    const int cell = c.cell, ncell = c.ncell;
    const int cs = c.cs, ce = c.cs + c.na;
    double dE_sum = 0.0, dE_abs = 0.0;
    int nacc = 0, nhard = 0;
    unsigned long long npairs = 0ull;
    const unsigned long long cands = (unsigned long long)(c.total - 1) * (unsigned long long)(ce - cs);
    for (int g = cs; g < ce; g++) {
        const uint32_t id = (uint32_t)v.id[g];
        const int code = v.thard[g];
        const double lu = v.tlu[g];
        if (code) { // colloid hard core (1), out of its cell (3): rejected, no energy evaluation
            if (lane == 0) {
                v.outcome[p.p_off + id] = code == 1 ? 2 : 0;
                if (v.rec_dE) {
                    v.rec_dE[p.p_off + id] = 0.0;
                    v.rec_lu[p.p_off + id] = lu;
                }
            }
            nhard += code == 1;
            continue;
        }
        const double ro[3] = {px[g], py[g], pz[g]}, eo[3] = {ox[g], oy[g], oz[g]};
        const double rn[3] = {v.tnx[g], v.tny[g], v.tnz[g]}, en[3] = {v.tux[g], v.tuy[g], v.tuz[g]};
        double po = 0.0, pn = 0.0;
        int np = 0;
        for (int s = 0; s < ncell; s++) {
            const int B = s_base[s], n_s = s_base[s + 1] - B;
            const int g0 = s_first[s];
            for (int q = B + ((lane - B) & 31); q < B + n_s; q += 32) {
                const int j = g0 + (q - B);
                if (j == g) continue;
                const double rj[3] = {px[j], py[j], pz[j]}, ej[3] = {ox[j], oy[j], oz[j]};
                double d[3];
                double r2 = dist_fold(ro[0], ro[1], ro[2], rj[0], rj[1], rj[2], L, d);
                if (r2 < k.rc2) {
                    po += pair_exact(k, r2, d, eo, ej);
                    np++;
                }
                r2 = dist_fold(rn[0], rn[1], rn[2], rj[0], rj[1], rj[2], L, d);
                if (r2 < k.rc2) {
                    pn += pair_exact(k, r2, d, en, ej);
                    np++;
                }
            }
        }
        double Eo = warp_sum_butterfly(po);
        double En = warp_sum_butterfly(pn);
        if (k.coll_on) {
            Eo = Eo + colloid_rod(k, ro, eo, L);
            En = En + colloid_rod(k, rn, en, L);
        }
        const double dE = En - Eo;
        const bool acc = (dE <= 0.0) || (lu <= -k.beta * dE);
        npairs += (unsigned long long)np;
        if (acc) {
            if (lane == 0) {
                px[g] = rn[0];
                py[g] = rn[1];
                pz[g] = rn[2];
                ox[g] = en[0];
                oy[g] = en[1];
                oz[g] = en[2];
            }
            dE_sum += dE;
            dE_abs += fabs(dE);
            nacc++;
        }
        if (lane == 0) {
            v.outcome[p.p_off + id] = acc ? 1 : 0;
            if (v.rec_dE) {
                v.rec_dE[p.p_off + id] = dE;
                v.rec_lu[p.p_off + id] = lu;
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) npairs += __shfl_xor_sync(0xffffffffu, npairs, o);
    if (lane == 0) {
        v.cell_e0[cell] = dE_sum;
        v.cell_abs[cell] = dE_abs;
        v.cell_fp64[cell] = 0;
        v.cell_n0[cell] = nacc;
        v.cell_n1[cell] = nhard;
        v.cell_pairs[cell] = npairs;
        v.cell_cands[cell] = cands;
    }
    __syncwarp();
}

// The cells of a block that were left to the sequential attempts, after its others
// (called among them, its registers were spilled from the decisions: a gas of 20,000
// rods 0.60 -> 0.64 ms of phases a sweep).  Warp 0.
__device__ __noinline__ void exact_cells_left(const DevView *__restrict__ vp, const ExactBatch eb, int ci, int a1, int *s_first,
                                              int *s_base)
{
    const DevView &v = *vp;
    const int *off = v.act_off + ci * (v.R + 1);
    const int lane = threadIdx.x & 31;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    for (int a = eb.lo + blockIdx.x; a < a1; a += gridDim.x) {
        if (a < eb.hi && !v.ex_flag[(size_t)ci * v.ex_act + a]) continue;
        CellView c;
        active_cell(v, off, ci, a, c);
        if (v.rep[c.r].use_fast || c.na == 0) continue;
        cell_stencil(v, c, lane, s_first, s_base);
        exact_cell_sequential(vp, c, lane, s_first, s_base);
        __syncwarp();
    }
}

// The attempts of one cell (J chunks of own-cell slots), D = 3 at a time: attempt
// k + d depends on the outcomes of k .. k + d - 1, so a warp evaluates it for
// each of their 2^d patterns (2^D - 1 warps), and every warp then follows the
// outcomes through the decisions.  What a warp does is what one alone would do
// per attempt: a dozen additions, the butterfly, the test, all of it latency, so
// three attempts take the time of one plus a barrier.  The records come from L2
// by bulk copies, a round ahead.  A cell of 125 particles: 58 us with one warp,
// 31 us; 15 warps for four attempts 33 us, three warps with 1, 2 and 4 chains
// each 46 us (the instructions of a warp count, not its waits).
constexpr int EX_SMS = 148;
constexpr int EX_DEPTH = 3, EX_WARPS = 8; // attempts of a round and the warps of a block (the eighth is a double)
template <int J> struct ExactStage {
    static constexpr int PF = 2 + 2 * J + EX_SUF;      // rows copied per attempt
    static constexpr int D = J <= 5 ? EX_DEPTH : 2;    // attempts of a round
    static constexpr int BYTES = 2 * D * PF * 32 * 16; // this round's records and the next one's
};
constexpr int ex_max(int a, int b) { return a > b ? a : b; }
constexpr int EX_BYTES = ex_max(ex_max(ExactStage<2>::BYTES, ExactStage<3>::BYTES),
                                ex_max(ExactStage<5>::BYTES, ExactStage<EX_J>::BYTES));

constexpr unsigned EX_WAIT_TRIES = 1u << 24; // mbarrier tries for the copies of a block that leaves

struct ExactShared {
    uint64_t full[2];       // mbarriers: a half's records have landed
    double dE[EX_NA];       // energy change of an accepted attempt, else 0
    int failed[2];          // a half's records did not land
    unsigned pairs[EX_WARPS], hard[EX_WARPS];
    CellView c;
    int first[27], base[28];
};

// false: a copy did not land (the flag is set)
template <int J>
__device__ __forceinline__ bool exact_decide_cell(const DevView &v, const CellView &c, int q13, const double2 *rows,
                                                  double2 *buf, ExactShared &sh, unsigned &phase)
{
    constexpr int PF = ExactStage<J>::PF, RPP = 2 + 2 * J + EX_SUF, D = ExactStage<J>::D, W = (1 << D) - 1;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const Replica &p = v.rep[c.r];
    const int na = c.na, c0 = q13 >> 5;
    const double beta = p.k.beta;
    const bool coll = p.k.coll_on;
    // warp w: the attempt at depth wd of a round, for the pattern wh of outcomes before it (the eighth as the seventh)
    const int wi = min(w, W - 1), wd = 31 - __clz(wi + 1), wh = wi + 1 - (1 << wd);
    // lanes of this warp that report its decision: the block's count is then the decisions' bits, 1 << w for warp w
    const bool report = w < W - (W == 7) ? lane < (1 << w) : W == 7;
    auto fetch = [&](int k0, int half) { // attempts k0 .. k0 + D - 1
        const int n = min(D, na - k0);
        if (t != EX_WARPS * 32 - 32 || n <= 0) return;
        tc::fence_proxy_async_smem(); // the block's reads of the records there came before its barrier
        tc::mbar_arrive_expect_tx(&sh.full[half], (uint32_t)n * (PF * 512));
        for (int d = 0; d < n; d++)
            tc::bulk_load(buf + (half * D + d) * (PF * 32), rows + (size_t)(k0 + d) * RPP * 32, PF * 512, &sh.full[half]);
    };
    fetch(0, 0);
    fetch(D, 1);
    if (na > 0) { // (uniform; an empty cell copies nothing)
        if (!tc::mbar_wait_bounded(&sh.full[0], phase & 1u, v.wait_tries)) sh.failed[0] = 1;
        phase ^= 1u;
    }
    __syncthreads();
    bool ok = !sh.failed[0];
    unsigned accm = 0u; // bit j: the particle at slot 32 (c0 + j) + lane was accepted
    int half = 0, k0 = 0;
    for (; k0 < na && ok; k0 += D, half ^= 1) {
        const int k = k0 + wd, q0 = q13 + k0;
        const int mine = (lane - q0) & 31, jm = ((q0 + mine) >> 5) - c0; // this lane's slot is the round's mine-th
        double dE = 0.0, lu = 0.0;
        bool acc = false;
        if (w < EX_WARPS && k < na) {
            const unsigned am = accm | ((unsigned)((wh >> mine) & 1) << jm); // with the pattern
            const double2 *rw = buf + (half * D + wd) * (PF * 32) + lane;
            const ExactHead *hd = reinterpret_cast<const ExactHead *>(rw - lane);
            struct { double lu; int code, nsuf; } h; // one load
            static_assert(offsetof(ExactHead, lu) == 16 && offsetof(ExactHead, code) == 24 && offsetof(ExactHead, nsuf) == 28, "layout");
            *reinterpret_cast<int4 *>(&h) = *reinterpret_cast<const int4 *>(&hd->lu);
            lu = h.lu;
            if (!h.code) {
                double2 x[J], y[4];
                double po = rw[32].x, pn = rw[32].y;
#pragma unroll
                for (int j = 0; j < J; j++) x[j] = rw[(2 + j) * 32 + ((am >> j) & 1u) * (J * 32)];
#pragma unroll
                for (int j = 0; j < J; j++) {
                    po += x[j].x;
                    pn += x[j].y;
                }
#pragma unroll
                for (int s0 = 0; s0 < EX_SUF; s0 += 4) {
                    if (s0 >= h.nsuf) break; // (uniform)
#pragma unroll
                    for (int s = 0; s < 4; s++) y[s] = rw[(2 + 2 * J + s0 + s) * 32];
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        po += y[s].x;
                        pn += y[s].y;
                    }
                }
                // the butterfly of both sums: the first level leaves the old state's to the lower lanes and the trial
                // state's to the upper ones (the additions are those of two butterflies)
                const bool up = lane & 16;
                double e = (up ? pn : po) + __shfl_xor_sync(0xffffffffu, up ? po : pn, 16);
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) e = e + __shfl_xor_sync(0xffffffffu, e, o);
                if (coll) e = e + (up ? hd->un : hd->uo);
                const double other = __shfl_xor_sync(0xffffffffu, e, 16);
                dE = up ? e - other : other - e;
                acc = (dE <= 0.0) || (lu <= -beta * dE);
            }
        }
        if (w == EX_WARPS - 1 && k0 + D < na) { // the next round's records
            if (!tc::mbar_wait_bounded(&sh.full[half ^ 1], (phase >> (half ^ 1)) & 1u, v.wait_tries)) sh.failed[half ^ 1] = 1;
        }
        if (k0 + D < na) phase ^= 1u << (half ^ 1);
        const int m = __syncthreads_count(acc && report); // bit w: warp w's attempt was accepted
        fetch(k0 + 2 * D, half);                          // over this round's
        const int a0 = m & 1, a1 = (m >> (1 + a0)) & 1, h2 = a0 | (a1 << 1);
        const int hist = D == 2 ? h2 : h2 | (((m >> (3 + h2)) & 1) << 2); // bit d: attempt k0 + d was accepted
        accm |= (unsigned)((hist >> mine) & 1) << jm;
        if (w < W && k < na && wh == (hist & ((1 << wd) - 1)) && lane == 0) { // this warp's pattern came about
            sh.dE[k] = (hist >> wd) & 1 ? dE : 0.0;
            if (v.rec_dE) {
                const int id = v.id[c.cs + k];
                v.rec_dE[p.p_off + id] = dE;
                v.rec_lu[p.p_off + id] = lu;
            }
        }
        // written before this round's barrier; the next round writes the other half's, the one after that comes past
        // the next barrier: every thread reads the same
        ok = !sh.failed[half ^ 1];
    }
    if (!ok) { // (uniform) the records of the round at k0 did not land
        if (t == 0) atomicOr(&v.stats[c.r].flags, F_TIMEOUT);
        // copies still on their way are waited for, again with a limit: that round's (its parity was stepped on) and,
        // if there is one, the round after's
        tc::mbar_wait_bounded(&sh.full[half], ((phase >> half) & 1u) ^ 1u, EX_WAIT_TRIES);
        if (k0 + D < na) tc::mbar_wait_bounded(&sh.full[half ^ 1], (phase >> (half ^ 1)) & 1u, EX_WAIT_TRIES);
        return false;
    }
    // a lane per particle: outcome, accepted trial state to the master arrays, and the pairs its attempt met
    // (the partners before it that were accepted in their trial state, every other in its old one)
    unsigned A[J]; // accepted slots of chunk c0 + j
#pragma unroll
    for (int j = 0; j < J; j++) A[j] = __ballot_sync(0xffffffffu, (accm >> j) & 1u);
    unsigned npairs = 0u, nhard = 0u;
    for (int k = 32 * w + lane; k < na; k += 32 * EX_WARPS) {
        const int q = q13 + k, g = c.cs + k;
        const ExactHead *hd = reinterpret_cast<const ExactHead *>(rows + (size_t)k * RPP * 32);
        const int code = hd->code, id = v.id[g];
        unsigned mk[4][J];
        int np = 0;
        if (!code) {
            np = hd->nstat;
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < J; j++) mk[i][j] = hd->mask[i][j];
        }
        bool acc = false;
#pragma unroll
        for (int j = 0; j < J; j++)
            if ((q >> 5) - c0 == j) acc = (A[j] >> (q & 31)) & 1u;
        v.outcome[p.p_off + id] = code == 1 ? 2 : (acc ? 1 : 0);
        if (acc) {
            v.px[g] = v.tnx[g];
            v.py[g] = v.tny[g];
            v.pz[g] = v.tnz[g];
            v.ox[g] = v.tux[g];
            v.oy[g] = v.tuy[g];
            v.oz[g] = v.tuz[g];
        }
        if (!code) {
#pragma unroll
            for (int j = 0; j < J; j++) {
                const int d = q - 32 * (c0 + j); // slots of this chunk before the particle's own
                const unsigned B = d <= 0 ? 0u : (d >= 32 ? A[j] : A[j] & ((1u << d) - 1u));
                np += __popc((mk[0][j] & ~B) | (mk[2][j] & B)) + __popc((mk[1][j] & ~B) | (mk[3][j] & B));
            }
        }
        npairs += (unsigned)np;
        nhard += code == 1;
    }
    npairs = __reduce_add_sync(0xffffffffu, npairs);
    nhard = __reduce_add_sync(0xffffffffu, nhard);
    if (lane == 0) sh.pairs[w] = npairs, sh.hard[w] = nhard;
    __syncthreads();
    if (t == 0) {
        unsigned long long n = 0ull;
        int nh = 0, nacc = 0;
        for (int i = 0; i < EX_WARPS; i++) n += sh.pairs[i], nh += sh.hard[i];
#pragma unroll
        for (int j = 0; j < J; j++) nacc += __popc(A[j]);
        double dE_sum = 0.0, dE_abs = 0.0; // in the attempts' order (0 for those that were not accepted)
#pragma unroll 8
        for (int k = 0; k < na; k++) {
            dE_sum += sh.dE[k];
            dE_abs += fabs(sh.dE[k]);
        }
        v.cell_e0[c.cell] = dE_sum;
        v.cell_abs[c.cell] = dE_abs;
        v.cell_fp64[c.cell] = 0;
        v.cell_n0[c.cell] = nacc;
        v.cell_n1[c.cell] = nh;
        v.cell_pairs[c.cell] = n;
        v.cell_cands[c.cell] = (unsigned long long)(c.total - 1) * (unsigned long long)na;
    }
    return true;
}

__global__ void __launch_bounds__(EX_WARPS * 32) k_exact_decide(const __grid_constant__ DevView v, int ci, int b)
{
    extern __shared__ double2 ex_buf[]; // [2][D][PF][32]
    phase_begin();
    __shared__ ExactShared sh;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        tc::mbar_init(&sh.full[0], 1);
        tc::mbar_init(&sh.full[1], 1);
        sh.failed[0] = sh.failed[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    unsigned phase = 0u; // bit h: parity of full[h]'s next completion
    bool left = false;   // a cell to be attempted sequentially
    const int *off = v.act_off + ci * (v.R + 1);
    const long long *er = v.ex_r + (size_t)ci * (v.ex_act + 1);
    const ExactBatch eb = exact_batch(v, off, er, b);
    const int a1 = b == v.ex_nb - 1 ? off[v.r_hi] : eb.hi; // the last batch takes the cells beyond the scratch
    for (int a = eb.lo + blockIdx.x; a < a1; a += gridDim.x) {
        __syncthreads(); // the cell before this one is done with the shared memory
        if (threadIdx.x < 32) {
            CellView c;
            active_cell(v, off, ci, a, c);
            if (!v.rep[c.r].use_fast && c.na > 0) cell_stencil(v, c, lane, sh.first, sh.base);
            if (lane == 0) sh.c = c;
        }
        __syncthreads();
        const CellView c = sh.c;
        if (v.rep[c.r].use_fast || c.na == 0) continue; // (an empty cell has its results from the rebin)
        if (a >= eb.hi || v.ex_flag[(size_t)ci * v.ex_act + a]) {
            left = true;
            continue;
        }
        const double2 *rows = v.ex_rows + (size_t)(er[a] - eb.row0) * 32;
        const int q13 = sh.base[c.own];
        bool ok;
        switch (ex_chunks(c.na)) {
        case 2: ok = exact_decide_cell<2>(v, c, q13, rows, ex_buf, sh, phase); break;
        case 3: ok = exact_decide_cell<3>(v, c, q13, rows, ex_buf, sh, phase); break;
        case 5: ok = exact_decide_cell<5>(v, c, q13, rows, ex_buf, sh, phase); break;
        default: ok = exact_decide_cell<EX_J>(v, c, q13, rows, ex_buf, sh, phase); break;
        }
        if (!ok) return; // (uniform)
    }
    if (left) exact_cells_left(&v, eb, ci, a1, sh.first, sh.base);
}

__device__ __forceinline__ void cp_row_async(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// The attempts of one cell by one warp, for phases with more cells than the chip
// has SMs: several such blocks share an SM, and evaluating only what is needed
// costs less than the patterns (262,144 particles: 6.3 ms of phases per sweep,
// 7.0 ms with a block of eight warps per cell).  Records EX_STAGES - 1 attempts
// ahead (cp.async), of the suffix rows EX_PFS.
constexpr int EX_PFS = 6;
constexpr int EX_STAGES = 4;
template <int J> struct ExactPipe {
    static constexpr int PF = 2 + 2 * J + EX_PFS; // rows fetched per attempt
};

constexpr int EX_PIPE_BYTES = EX_STAGES * ExactPipe<EX_J>::PF * 32 * 16;

template <int J>
__device__ __forceinline__ void exact_decide_cell_warp(const DevView &v, const CellView &c, int lane, int q13,
                                                  const double2 *rows, double2 *buf)
{
    constexpr int PF = ExactPipe<J>::PF, RPP = 2 + 2 * J + EX_SUF;
    const Replica &p = v.rep[c.r];
    const int na = c.na, c0 = q13 >> 5;
    const double beta = p.k.beta;
    const bool coll = p.k.coll_on;
    const double2 *src = rows + lane;
    double2 *mine = buf + lane;
    int kf = 0, sf = 0; // next record to fetch and its stage
    auto fetch = [&]() {
        if (kf < na) {
            double2 *dst = mine + sf * (PF * 32);
#pragma unroll
            for (int i = 0; i < PF; i++) cp_row_async(dst + i * 32, src + i * 32);
            src += RPP * 32;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        kf++;
        sf = sf == EX_STAGES - 1 ? 0 : sf + 1;
    };
#pragma unroll
    for (int k = 0; k < EX_STAGES - 1; k++) fetch();
    unsigned accm = 0u; // bit j: the particle at slot 32 (c0 + j) + lane was accepted
    double dE_sum = 0.0, dE_abs = 0.0;
    int nacc = 0, nhard = 0, st = 0;
    for (int k = 0; k < na; k++) {
        fetch();
        asm volatile("cp.async.wait_group %0;" ::"n"(EX_STAGES - 1) : "memory");
        __syncwarp();
        const double2 *rw = mine + st * (PF * 32);
        st = st == EX_STAGES - 1 ? 0 : st + 1;
        const ExactHead *hd = reinterpret_cast<const ExactHead *>(rw - lane);
        const int code = hd->code, nsuf = hd->nsuf;
        const double lu = hd->lu;
        double dE = 0.0;
        if (code) {
            nhard += code == 1;
        } else {
            double2 x[J], y[4];
            double po = rw[32].x, pn = rw[32].y;
#pragma unroll
            for (int j = 0; j < J; j++) x[j] = rw[((accm >> j) & 1u ? 2 + J + j : 2 + j) * 32];
#pragma unroll
            for (int s = 0; s < 4; s++) y[s] = s < nsuf ? rw[(2 + 2 * J + s) * 32] : make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < J; j++) {
                po += x[j].x;
                pn += x[j].y;
            }
#pragma unroll
            for (int s = 0; s < 4; s++) {
                po += y[s].x;
                pn += y[s].y;
            }
            for (int s = 4; s < nsuf; s++) {
                const double2 z = s < EX_PFS ? rw[(2 + 2 * J + s) * 32]
                                             : rows[((size_t)k * RPP + 2 + 2 * J + s) * 32 + lane];
                po += z.x;
                pn += z.y;
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) {
                const double yo = __shfl_xor_sync(0xffffffffu, po, o), yn = __shfl_xor_sync(0xffffffffu, pn, o);
                po = po + yo;
                pn = pn + yn;
            }
            if (coll) {
                po = po + hd->uo;
                pn = pn + hd->un;
            }
            dE = pn - po;
            if ((dE <= 0.0) || (lu <= -beta * dE)) {
                const int q = q13 + k;
                if (lane == (q & 31)) accm |= 1u << ((q >> 5) - c0);
                dE_sum += dE;
                dE_abs += fabs(dE);
                nacc++;
            }
        }
        if (v.rec_dE && lane == 0) {
            const int id = v.id[c.cs + k];
            v.rec_dE[p.p_off + id] = dE;
            v.rec_lu[p.p_off + id] = lu;
        }
        __syncwarp(); // the stage may be refilled
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // a lane per particle: outcome, accepted trial state to the master arrays, and the pairs its attempt met
    // (the partners before it that were accepted in their trial state, every other in its old one)
    unsigned long long npairs = 0ull;
    for (int k0 = 0; k0 < na; k0 += 32) {
        const int k = k0 + lane, q = q13 + k, g = c.cs + k;
        const bool on = k < na;
        const unsigned m = __shfl_sync(0xffffffffu, accm, q & 31);
        const bool acc = on && ((m >> ((q >> 5) - c0)) & 1u);
        const ExactHead *hd = reinterpret_cast<const ExactHead *>(rows + (size_t)(on ? k : 0) * RPP * 32);
        const int code = on ? hd->code : 3;
        if (on) v.outcome[p.p_off + v.id[g]] = code == 1 ? 2 : (acc ? 1 : 0);
        if (acc) {
            v.px[g] = v.tnx[g];
            v.py[g] = v.tny[g];
            v.pz[g] = v.tnz[g];
            v.ox[g] = v.tux[g];
            v.oy[g] = v.tuy[g];
            v.oz[g] = v.tuz[g];
        }
        int np = code ? 0 : hd->nstat;
#pragma unroll
        for (int j = 0; j < J; j++) {
            const unsigned A = __ballot_sync(0xffffffffu, (accm >> j) & 1u); // accepted slots of chunk c0 + j
            if (!code) {
                const int d = q - 32 * (c0 + j); // slots of this chunk before the particle's own
                const unsigned B = d <= 0 ? 0u : (d >= 32 ? A : A & ((1u << d) - 1u));
                np += __popc((hd->mask[0][j] & ~B) | (hd->mask[2][j] & B)) +
                      __popc((hd->mask[1][j] & ~B) | (hd->mask[3][j] & B));
            }
        }
        npairs += (unsigned long long)np;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) npairs += __shfl_xor_sync(0xffffffffu, npairs, o);
    if (lane == 0) {
        v.cell_e0[c.cell] = dE_sum;
        v.cell_abs[c.cell] = dE_abs;
        v.cell_fp64[c.cell] = 0;
        v.cell_n0[c.cell] = nacc;
        v.cell_n1[c.cell] = nhard;
        v.cell_pairs[c.cell] = npairs;
        v.cell_cands[c.cell] = (unsigned long long)(c.total - 1) * (unsigned long long)na;
    }
    __syncwarp();
}

__global__ void __launch_bounds__(32) k_exact_decide_warp(const __grid_constant__ DevView v, int ci, int b)
{
    extern __shared__ double2 ex_buf[]; // [EX_STAGES][PF][32]
    phase_begin();
    __shared__ int s_first[27], s_base[28];
    const int lane = threadIdx.x;
    bool left = false; // a cell to be attempted sequentially
    const int *off = v.act_off + ci * (v.R + 1);
    const long long *er = v.ex_r + (size_t)ci * (v.ex_act + 1);
    const ExactBatch eb = exact_batch(v, off, er, b);
    const int a1 = b == v.ex_nb - 1 ? off[v.r_hi] : eb.hi; // the last batch takes the cells beyond the scratch
    for (int a = eb.lo + blockIdx.x; a < a1; a += gridDim.x) {
        CellView c;
        active_cell(v, off, ci, a, c);
        if (v.rep[c.r].use_fast || c.na == 0) continue; // (an empty cell has its results from the rebin)
        cell_stencil(v, c, lane, s_first, s_base);
        if (a >= eb.hi || v.ex_flag[(size_t)ci * v.ex_act + a]) {
            left = true;
            continue;
        }
        const double2 *rows = v.ex_rows + (size_t)(er[a] - eb.row0) * 32;
        const int q13 = s_base[c.own];
        switch (ex_chunks(c.na)) {
        case 2: exact_decide_cell_warp<2>(v, c, lane, q13, rows, ex_buf); break;
        case 3: exact_decide_cell_warp<3>(v, c, lane, q13, rows, ex_buf); break;
        case 5: exact_decide_cell_warp<5>(v, c, lane, q13, rows, ex_buf); break;
        default: exact_decide_cell_warp<EX_J>(v, c, lane, q13, rows, ex_buf); break;
        }
    }
    if (left) exact_cells_left(&v, eb, ci, a1, s_first, s_base);
}

// Total energy (tot_ene, MCnptColloid.c:1598-1622) in FP64, warp per particle:
// sum over unordered pairs (r < rc, minimum image) found in the 27-cell
// stencil, plus the colloid term of every particle, with pair_exact (the
// reference-order term).  SCALED: the NPT volume move's energies of the
// current configuration and of the one scaled by lam about the origin
// (colloid at the scaled box centre), with pair_energy64.  Works on any grid,
// including boxes of fewer than 3 cells per axis (the wrapped stencil is
// deduplicated).
//
// Each pair is evaluated once: slots are sorted by cell, so particle i takes
// the rest of its own cell (slots > i) and the whole of every stencil cell
// with a larger index; e0[i] (e1[i] scaled) holds those pair terms plus its
// colloid term, and the slot sums add up to the total.  Only about one
// candidate in eight is inside the cutoff, so pairs are not evaluated where
// they are found: a distance pass over 32 candidates at a time appends the
// in-cutoff (candidate, configuration) items to a per-warp queue, and every
// 32 queued items are evaluated with all lanes busy.  The order of the FP64
// additions is fixed by the data, so results repeat bit for bit.
constexpr int EQ = 96; // queue entries per warp: < 32 pending + 64 from one chunk
#ifndef LCMC_ENERGY_MIN_BLOCKS
#define LCMC_ENERGY_MIN_BLOCKS 8
#endif

template <bool SCALED>
__global__ void __launch_bounds__(128, LCMC_ENERGY_MIN_BLOCKS) k_energy_exact(DevView v, double *e0, double *e1, int *hard,
                                                                                      bool all)
{
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const int nw = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    __shared__ int s_start[4][28]; // flat index of the first candidate of each cell
    __shared__ int s_base[4][28];  // particle slot minus flat index, per cell
    __shared__ int s_qj[4][EQ];    // queued candidate slot, configuration in bit 31
    // nothing to do when the cell kernel serves every replica that needs the energies
    bool any = false;
    for (int r = lane; r < v.R; r += 32) {
        const Replica &p = v.rep[r];
        any = any || (SCALED ? p.ensemble == 2 && !(p.da_on && !p.vol_stage1) && !cells_serve<0>(p) : all || !cells_serve<2>(p));
    }
    if (!__any_sync(0xffffffffu, any)) return;
    for (int i = blockIdx.x * nw + wib; i < v.ntot; i += gridDim.x * nw) {
        const int r = v.p2r[i];
        const Replica &p = v.rep[r];
        const int nc0 = p.nc[0], nc1 = p.nc[1], nc2 = p.nc[2];
        // NVT, screened out, or served by the cell kernel (>= 4 cells per axis)
        if (SCALED ? p.ensemble != 2 || (p.da_on && !p.vol_stage1) || cells_serve<0>(p) : !all && cells_serve<2>(p)) continue;
        const int own = v.scid[i];
        const int cell = own - p.cell_off;
        const int cx = cell % nc0, cy = (cell / nc0) % nc1, cz = cell / (nc0 * nc1);
        int c = -1;
        if (lane < 27) {
            int dz = lane / 9 - 1, dy = (lane / 3) % 3 - 1, dx = lane % 3 - 1;
            int x = (cx + dx + nc0) % nc0, y = (cy + dy + nc1) % nc1, z = (cz + dz + nc2) % nc2;
            c = p.cell_off + (z * nc1 + y) * nc0 + x;
        }
        const unsigned same = __match_any_sync(0xffffffffu, c);
        const bool keep = lane < 27 && (__ffs(same) - 1) == lane && c >= own;
        const unsigned kb = __ballot_sync(0xffffffffu, keep);
        const int ncell = __popc(kb);
        const int slot = __popc(kb & lt);
        int first = 0, cnt = 0;
        if (keep) {
            const int b = v.cell_start[c], e = v.cell_start[c + 1];
            first = c == own ? i + 1 : b;
            cnt = e - first;
        }
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (keep) {
            s_start[wib][slot] = inc - cnt;
            s_base[wib][slot] = first - (inc - cnt);
        }
        const int total = __shfl_sync(0xffffffffu, inc, 31);
        if (lane == 0) s_start[wib][ncell] = total;
        __syncwarp();

        const double lam = SCALED ? p.vol_lambda : 1.0;
        const double Ls[3] = {p.L[0] * lam, p.L[1] * lam, p.L[2] * lam};
        const double ri[3] = {v.px[i], v.py[i], v.pz[i]};
        const double ei[3] = {v.ox[i], v.oy[i], v.oz[i]};
        const double rs[3] = {ri[0] * lam, ri[1] * lam, ri[2] * lam};
        // the scaled distance is lam^2 r2 up to a few ulp: decide the scaled
        // cutoff from it unless it lies within 1e-10 of rc^2
        const double lam2 = lam * lam, rc2 = p.k.rc2, band = 1e-10 * rc2;
        double a0 = 0.0, a1 = 0.0;
        int qn = 0;
        int sc = 0; // this lane's current cell (its candidates only move forward)

        for (int t0 = 0; t0 < total; t0 += 32) {
            const int q = t0 + lane;
            bool f0 = false, f1 = false;
            int j = 0;
            if (q < total) {
                while (s_start[wib][sc + 1] <= q) sc++;
                j = s_base[wib][sc] + q;
                const double rj[3] = {v.px[j], v.py[j], v.pz[j]};
                double d[3];
                const double r2 = dist_fold(ri[0], ri[1], ri[2], rj[0], rj[1], rj[2], p.L, d);
                f0 = r2 < rc2;
                if (SCALED) {
                    const double r2s = lam2 * r2;
                    if (fabs(r2s - rc2) > band) f1 = r2s < rc2;
                    else f1 = dist_fold(rs[0], rs[1], rs[2], rj[0] * lam, rj[1] * lam, rj[2] * lam, Ls, d) < rc2;
                }
            }
            const unsigned b0 = __ballot_sync(0xffffffffu, f0);
            const unsigned b1 = __ballot_sync(0xffffffffu, f1);
            if (f0) s_qj[wib][qn + __popc(b0 & lt)] = j;
            if (f1) s_qj[wib][qn + __popc(b0) + __popc(b1 & lt)] = j | (int)0x80000000u;
            qn += __popc(b0) + __popc(b1);
            __syncwarp();
            // evaluate full batches of 32 queued pairs
            while (qn >= 32 || (qn > 0 && t0 + 32 >= total)) {
                const int m = qn < 32 ? qn : 32;
                if (lane < m) {
                    const int e = s_qj[wib][lane];
                    const int jj = e & 0x7fffffff;
                    const double rj[3] = {v.px[jj], v.py[jj], v.pz[jj]};
                    const double ej[3] = {v.ox[jj], v.oy[jj], v.oz[jj]};
                    double d[3], r2;
                    if (e < 0) {
                        r2 = dist_fold(rs[0], rs[1], rs[2], rj[0] * lam, rj[1] * lam, rj[2] * lam, Ls, d);
                        a1 += pair_energy64(p.k, r2, d, ei, ej);
                    } else {
                        r2 = dist_fold(ri[0], ri[1], ri[2], rj[0], rj[1], rj[2], p.L, d);
                        a0 += SCALED ? pair_energy64(p.k, r2, d, ei, ej) : pair_exact(p.k, r2, d, ei, ej);
                    }
                }
                // move entries [m, qn) to the front
                int mv0 = 0, mv1 = 0;
                if (m + lane < qn) mv0 = s_qj[wib][m + lane];
                if (m + 32 + lane < qn) mv1 = s_qj[wib][m + 32 + lane];
                __syncwarp();
                if (m + lane < qn) s_qj[wib][lane] = mv0;
                if (m + 32 + lane < qn) s_qj[wib][32 + lane] = mv1;
                __syncwarp();
                qn -= m;
            }
        }
        a0 = warp_sum_butterfly(a0);
        a1 = warp_sum_butterfly(a1);
        if (lane == 0) {
            double u0 = a0, u1 = a1;
            if (p.k.coll_on) {
                u0 += colloid_rod(p.k, ri, ei, p.L);
                if (SCALED) u1 += colloid_rod(p.k, rs, ei, Ls);
            }
            e0[i] = u0;
            if (SCALED) {
                e1[i] = u1;
                double d[3];
                double r2 = dist_fold(rs[0], rs[1], rs[2], 0.5 * Ls[0], 0.5 * Ls[1], 0.5 * Ls[2], Ls, d);
                hard[i] = !(r2 > p.k.coll_R * p.k.coll_R);
            }
        }
        __syncwarp();
    }
}

} // namespace lcmc


namespace lcmc {

// Scratch rows (of 512 bytes) for ntot particles on the FP64 kernel: *cap rows
// per batch, at most `most` (EX_MOST, 256 MB, less where there is no room), and
// *nb batches per phase.  Most systems run in one batch.  Active particles of a
// phase are about an eighth of the system (all of it in a one-cell box); cells
// that the batches do not reach are attempted sequentially.
void exact_scratch_size(int ntot, long long most, long long *cap, long long *alloc, int *nb)
{
    const long long all = (long long)ntot * ex_rows_per_particle(EX_NA);
    *cap = all < most ? all : most;
    *alloc = *cap + (long long)EX_NA * ex_rows_per_particle(EX_NA);
    const long long typical = (long long)ntot * ex_rows_per_particle(64) / 4;
    *nb = all <= most ? 1 : (int)((typical + most - 1) / most) + 1;
    if (most < EX_MOST) *nb = std::min(*nb, 16);
}

void exact_init()
{
    cudaFuncSetAttribute(k_exact_decide, cudaFuncAttributeMaxDynamicSharedMemorySize, EX_BYTES);
    // the rest is L1, for the cells that are attempted sequentially (the default leaves it to blocks that a phase of at
    // most a cell per SM does not have)
    cudaFuncSetAttribute(k_exact_decide, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (100 * (EX_BYTES + (int)sizeof(ExactShared) + 2048) + 233471) / 233472);
    cudaFuncSetAttribute(k_exact_decide_warp, cudaFuncAttributeMaxDynamicSharedMemorySize, EX_PIPE_BYTES);
}

void launch_exact_offsets(const DevView &v, cudaStream_t s) { k_exact_offsets<<<v.nphase, 1024, 0, s>>>(v); }

void launch_phase_exact(const DevView &v, cudaStream_t s, int ci, int grid)
{
    const int gt = min(4 * grid, v.ntot), gd = min(grid, v.ex_act);
    for (int b = 0; b < v.ex_nb; b++) {
        launch_phase(k_exact_terms, gt, 128, 0, s, v, ci, b);
        // up to a cell per SM the patterns' warps are idle ones: 1000 particles (one active cell or eight) 0.655 ->
        // 0.48 ms of phases per sweep, 8192 (27) 0.51 -> 0.465; 65,536 (343) would take 1.72 instead of 1.50.  What is
        // compared is the most active cells the context was made for, ex_act: cells of its FP32 systems and of NPT
        // boxes at 1.25 times their edge count too, so a few FP64 boxes among them take a warp per cell
        if (v.ex_act <= EX_SMS) launch_phase(k_exact_decide, gd, EX_WARPS * 32, EX_BYTES, s, v, ci, b);
        else launch_phase(k_exact_decide_warp, gd, 32, EX_PIPE_BYTES, s, v, ci, b);
    }
}

int energy_exact_blocks_per_sm()
{
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_energy_exact<true>, 128, 0) != cudaSuccess || b < 1) {
        cudaGetLastError();
        b = 4;
    }
    return b;
}

// resident blocks of a cell kernel on this device (queried once)
template <int MODE>
static int cell_energy_grid()
{
    static const int grid = [] {
        int dev = 0, sms = 0, b = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_cell_energy<MODE, false>, 128, 0) != cudaSuccess || b < 1) {
            cudaGetLastError();
            b = 2;
        }
        return b * (sms > 0 ? sms : 1);
    }();
    return grid;
}

// The volume move's U(V), U(V'): the cell kernel for systems with >= 4 cells
// per axis, the per-particle kernel for the rest (launched when there may be any).
void launch_volume_energies(const DevView &v, cudaStream_t s, double *e0, double *e1, int *hard, int grid,
                            bool per_particle)
{
    k_cell_energy<0, false><<<cell_energy_grid<0>(), 128, 0, s>>>(v);
    if (per_particle) k_energy_exact<true><<<grid, 128, 0, s>>>(v, e0, e1, hard, false);
}

// The total energy, likewise (by_cells: there may be systems the cell kernel
// serves); cells = false: per particle for every system.
// That is the order an uploaded configuration's energy is summed in: a start
// with overlapping rods has terms of 1e20 and more, whose rounding stays in the
// running energy after the overlaps have gone.
void launch_total_energy(const DevView &v, cudaStream_t s, double *e0, double *e1, int *hard, int grid, bool cells,
                         bool by_cells, bool per_particle)
{
    cells = cells && by_cells;
    if (cells) k_cell_energy<2, false><<<cell_energy_grid<2>(), 128, 0, s>>>(v);
    if (!cells || per_particle) k_energy_exact<false><<<grid, 128, 0, s>>>(v, e0, e1, hard, !cells);
}

} // namespace lcmc
