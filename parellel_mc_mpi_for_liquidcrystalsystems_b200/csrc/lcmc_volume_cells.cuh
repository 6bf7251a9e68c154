// lcmc_volume_cells.cuh - energy sums over whole configurations, one block per
// cell: U(V) and U(V') of an NPT volume move (no reference counterpart: the
// reference has no NPT move, MCnptColloid.c:3978), and the total energy
// (tot_ene, MCnptColloid.c:1598-1622).  The pair term is pij_GB, 2607-2681.
//
// The own cell's particles and those of its 13 forward neighbours, the stencil
// slots u = 9 (dz + 1) + 3 (dy + 1) + dx + 1 > 13 (each unordered cell pair once
// under periodic wrap; >= 4 cells per axis), are staged in shared memory: FP64
// position, the orientation, and a half-precision test vector relative to the
// own cell's centre.  Each warp takes eight own particles and 128 staged slots:
// the matrix unit tests which pairs lie within reach (cutoff at V or V', plus the
// operands' rounding), the sign bits become a list, and the four warps' lists
// together are evaluated by the whole block, all lanes busy.  The cutoff itself is decided on the
// FP64 minimum-image distance of every listed pair, so the pair set is the FP64
// kernel's exactly.
//   MODE 0  FP64 terms at V and V' (pair_energy64_x2): the volume move's energies
//   MODE 1  FP32 pair terms on the FP64 vectors rounded to FP32, with the FP32
//           copy's orientations: the delayed-acceptance screen U32 (FP32-kernel
//           systems, whose FP32 state copy exists)
//   MODE 2  FP64 terms at V only: the total energy
// Each cell's sums (lane order, then warps, then 32 lanes: fixed by the data)
// go to cell_e0, cell_e1 and its count of centres inside the colloid at V' to
// cell_n1.
//
// What bounds it: MODE 0 and 2 the FP64 pipe (about 150 FP64 instructions per
// in-cutoff pair for both volumes; two terms from their own expressions took
// 350), MODE 1 issue slots.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "lcmc_gb.cuh"
#include "lcmc_internal.h"
#include "lcmc_tc.cuh"
#include "lcmc_trial.cuh"

namespace lcmc {

constexpr int VC_CAP = 512;  // staged particles: the own cell and (part of) its forward neighbours
constexpr int VC_OWN = 384;  // own-cell particles (more: pair by pair from global memory)
constexpr int VC_BLK = 128;  // staged slots a warp tests at a time
constexpr int VC_REP = 128;  // replicas whose used cells are enumerated directly (more: every allocated cell)

// replica owning cell slot c (cell ranges are laid out in replica order)
__device__ __forceinline__ int replica_of_cell(const DevView &v, int c)
{
    int lo = 0, hi = v.R;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (v.rep[mid].cell_off <= c) lo = mid;
        else hi = mid;
    }
    return lo;
}

// replicas whose energies a cell kernel computes
template <int MODE>
__device__ __forceinline__ bool cells_serve(const Replica &p)
{
    const bool grid = p.nc[0] >= 4 && p.nc[1] >= 4 && p.nc[2] >= 4;
    if (MODE == 2) return grid && p.n >= ENERGY_PER_CELL * (p.nc[0] * p.nc[1] * p.nc[2]);
    if (p.ensemble != 2) return false;
    if (MODE == 1) return p.da_kind == 2 && p.use_fast;
    if (p.da_on && !p.vol_stage1) return false; // screened out: no exact recompute
    return p.vol_cells && grid;
}

// FP64 pair terms of one pair at separation d (r^2 given) and at lambda d, unit
// orientations.  Scaling leaves every angle unchanged, so both terms share all
// but the distance: three reciprocal square roots and three divisions for two
// terms (five and three for each on its own).  dist: the shifted distance of e0.
template <bool TWO>
__device__ __forceinline__ void pair_energy64_x2(const GBConsts &k, double r2, const double d[3], const double ui[3],
                                                 const double uj[3], double lam, double &e0, double &e1, double &dist)
{
    const double ir = rsqrt(r2);
    const double r = r2 * ir;
    const double c = __fma_rn(ui[2], uj[2], __fma_rn(ui[1], uj[1], ui[0] * uj[0]));
    const double a = ir * __fma_rn(d[2], ui[2], __fma_rn(d[1], ui[1], d[0] * ui[0]));
    const double b = ir * __fma_rn(d[2], uj[2], __fma_rn(d[1], uj[1], d[0] * uj[0]));
    const double sp = (a + b) * (a + b), sm = (a - b) * (a - b);
    const double wp = k.chi_prime * c, wc = k.chi * c;
    const double eps1 = rsqrt(__fma_rn(-wc, wc, 1.0));
    const double gp = __fma_rn(sp, 1.0 - wp, sm * (1.0 + wp)), gc = __fma_rn(sp, 1.0 - wc, sm * (1.0 + wc));
    const double eps2 = __fma_rn(-0.5 * k.chi_prime, gp / __fma_rn(-wp, wp, 1.0), 1.0);
    const double s_chi = __fma_rn(-0.5 * k.chi, gc * (eps1 * eps1), 1.0);
    const double well = k.four_eps0 * (ipow_d(eps1, k.nu_code, k.nu) * ipow_d(eps2, k.mu_code, k.mu));
    const double sig = k.sigma0 * rsqrt(s_chi);
    const double D0 = (r - sig) + k.sigma0;
    const double R0 = k.sigma0 / D0, q0 = R0 * R0, w0 = q0 * q0 * q0;
    e0 = D0 < 0.001 ? 1000000000.0 : well * w0 * (w0 - 1.0); // MCnptColloid.c:2670
    dist = D0;
    if (TWO) {
        const double D1 = __fma_rn(lam, r, -sig) + k.sigma0;
        const double R1 = k.sigma0 / D1, q1 = R1 * R1, w1 = q1 * q1 * q1;
        e1 = D1 < 0.001 ? 1000000000.0 : well * w1 * (w1 - 1.0);
    }
}

template <int MODE>
struct CellEnergySmem {
    double px[VC_CAP], py[VC_CAP], pz[VC_CAP];
    double ux[MODE == 1 ? 1 : VC_CAP], uy[MODE == 1 ? 1 : VC_CAP], uz[MODE == 1 ? 1 : VC_CAP]; // unit orientation
    float fx[MODE == 1 ? VC_CAP : 1], fy[MODE == 1 ? VC_CAP : 1], fz[MODE == 1 ? VC_CAP : 1];  // FP32 copy's
    uint2 ch[VC_CAP + VC_BLK]; // (x, y, z, |c|^2 rounded down), half precision, from the own cell's centre, scaled
    unsigned list[4 * 8 * VC_BLK]; // own particle << 16 | staged slot, of four pieces of work
    int nlist[4];
    int slot[MODE == 2 ? VC_CAP : 1]; // particle slot of a staged one
    double red[4][2];
    int ucell[VC_REP + 1]; // used-cell prefix over the replicas
    int start[14];         // first particle slot of stencil position o (slot 13 + o)
    int pre_n[15];         // particle prefix per stencil position
};

// The reference-order term of particles at slots i, j (its orientations as they
// are stored), within the cutoff.
static __device__ __noinline__ double pair_exact_at(const DevView *__restrict__ vp, int r, int i, int j)
{
    const DevView &v = *vp;
    const Replica &p = v.rep[r];
    const double ei[3] = {v.ox[i], v.oy[i], v.oz[i]}, ej[3] = {v.ox[j], v.oy[j], v.oz[j]};
    double d[3];
    const double r2 = dist_fold(v.px[i], v.py[i], v.pz[i], v.px[j], v.py[j], v.pz[j], p.L, d);
    return pair_exact(p.k, r2, d, ei, ej);
}

// One pair of particles (slots si, sj) at FP64 positions ri, rj: terms of both configurations
// (0 beyond the cutoff) added to a0, a1.
template <int MODE, bool SPEC21>
__device__ __forceinline__ void cell_pair(const DevView &v, int r, int si, int sj, const Replica &p, const FastK &K, const double ri[3], const double rj[3],
                                          const double ui[3], const double uj[3], const float fi[3], const float fj[3],
                                          double lam, double lam2, const double Ls[3], double &a0, double &a1)
{
    double d[3];
    const double rc2 = p.k.rc2;
    const double r2 = dist_fold(ri[0], ri[1], ri[2], rj[0], rj[1], rj[2], p.L, d);
    const bool in0 = r2 < rc2;
    if (MODE == 2) {
        if (in0) {
            double e0, e1, dist;
            pair_energy64_x2<false>(p.k, r2, d, ui, uj, 1.0, e0, e1, dist);
            // near an overlap R^12 magnifies a rounding of the distance by 12 r / dist: the total takes the
            // reference-order term there, so that it agrees with that sum to 1e-12 whatever the configuration
            if (dist < 0.3) e0 = pair_exact_at(&v, r, si, sj);
            a0 += e0;
        }
        return;
    }
    // the scaled configuration as the volume scaling forms it (positions r lambda, box L lambda, rounded products)
    if (MODE == 0) {
        // its distance is lam^2 r2 up to a few ulp: decide from it unless within 1e-10 of rc^2
        const double r2s = lam2 * r2;
        bool in1 = r2s < rc2;
        if (fabs(r2s - rc2) <= 1e-10 * rc2) {
            double ds[3];
            in1 = dist_fold(__dmul_rn(ri[0], lam), __dmul_rn(ri[1], lam), __dmul_rn(ri[2], lam), __dmul_rn(rj[0], lam),
                            __dmul_rn(rj[1], lam), __dmul_rn(rj[2], lam), Ls, ds) < rc2;
        }
        if (in0 || in1) {
            double e0, e1, dist;
            pair_energy64_x2<true>(p.k, r2, d, ui, uj, lam, e0, e1, dist);
            a0 += in0 ? e0 : 0.0;
            a1 += in1 ? e1 : 0.0;
        }
    } else {
        double ds[3];
        const bool in1 = dist_fold(__dmul_rn(ri[0], lam), __dmul_rn(ri[1], lam), __dmul_rn(ri[2], lam),
                                   __dmul_rn(rj[0], lam), __dmul_rn(rj[1], lam), __dmul_rn(rj[2], lam), Ls, ds) < rc2;
        if (in0 || in1) {
            float e0, e1;
            bool c0, c1; // the FP64 distances decide
            pair_fast_x2<SPEC21>(K, pack2((float)d[0], (float)ds[0]), pack2((float)d[1], (float)ds[1]),
                                 pack2((float)d[2], (float)ds[2]), dup2(fi[0]), dup2(fi[1]), dup2(fi[2]), dup2(fj[0]),
                                 dup2(fj[1]), dup2(fj[2]), e0, e1, c0, c1);
            a0 += in0 ? (double)e0 : 0.0;
            a1 += in1 ? (double)e1 : 0.0;
        }
    }
}

// Cells with more particles than are staged: pair by pair from global memory.
template <int MODE, bool SPEC21>
__device__ __noinline__ void cell_pairs_global(const DevView *__restrict__ vp, int r, const int *start, const int *pre_n,
                                               const double *Ls, double *out)
{
    const DevView &v = *vp;
    const Replica &p = v.rep[r];
    const FastK K = fast_consts(p.k);
    const int na = pre_n[1], nall = pre_n[14], g0 = start[0];
    const double lam = p.vol_lambda;
    double a0 = 0.0, a1 = 0.0;
    for (int k = 0; k < na; k++) {
        const int i = g0 + k;
        const double ri[3] = {v.px[i], v.py[i], v.pz[i]};
        double ui[3] = {v.ox[i], v.oy[i], v.oz[i]};
        const double in = rsqrt(ui[0] * ui[0] + ui[1] * ui[1] + ui[2] * ui[2]);
        for (int a = 0; a < 3; a++) ui[a] *= in;
        float fi[3] = {0.0f, 0.0f, 0.0f}, fj[3] = {0.0f, 0.0f, 0.0f};
        if (MODE == 1) fi[0] = v.cl4[i].w, fi[1] = v.cl2[i].x, fi[2] = v.cl2[i].y;
        int o = 0;
        for (int f = k + 1 + (int)threadIdx.x; f < nall; f += blockDim.x) {
            while (pre_n[o + 1] <= f) o++;
            const int j = start[o] + (f - pre_n[o]);
            const double rj[3] = {v.px[j], v.py[j], v.pz[j]};
            double uj[3] = {v.ox[j], v.oy[j], v.oz[j]};
            const double jn = rsqrt(uj[0] * uj[0] + uj[1] * uj[1] + uj[2] * uj[2]);
            for (int a = 0; a < 3; a++) uj[a] *= jn;
            if (MODE == 1) fj[0] = v.cl4[j].w, fj[1] = v.cl2[j].x, fj[2] = v.cl2[j].y;
            cell_pair<MODE, SPEC21>(v, r, i, j, p, K, ri, rj, ui, uj, fi, fj, lam, lam * lam, Ls, a0, a1);
        }
    }
    out[0] = a0;
    out[1] = a1;
}

template <int MODE> struct CellEnergyBlocks { static constexpr int value = MODE == 1 ? 5 : 4; };

template <int MODE, bool SPEC21>
__global__ void __launch_bounds__(128, CellEnergyBlocks<MODE>::value) k_cell_energy(const __grid_constant__ DevView v)
{
    __shared__ __align__(16) CellEnergySmem<MODE> sm;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    // the cells this kernel serves: the used cells (nc0 nc1 nc2 of the nc_max^3
    // allocated) of the replicas it serves, enumerated through a prefix
    const bool direct = v.R <= VC_REP;
    if (direct) {
        int n = 0;
        if (t < v.R) {
            const Replica &p = v.rep[t];
            if (cells_serve<MODE>(p)) n = p.nc[0] * p.nc[1] * p.nc[2];
        }
        int inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) sm.start[w] = inc;
        __syncthreads();
        for (int q = 0; q < w; q++) inc += sm.start[q];
        sm.ucell[t + 1] = inc;
        if (t == 0) sm.ucell[0] = 0;
        __syncthreads();
    }
    const int ncells = direct ? sm.ucell[v.R] : v.ctot;
    for (int e = blockIdx.x; e < ncells; e += gridDim.x) {
        int r, l;
        if (direct) { // replica: the largest r with ucell[r] <= e (replicas it does not serve are empty)
            int lo_ = 0, hi_ = v.R;
            while (hi_ - lo_ > 1) {
                const int mid = (lo_ + hi_) >> 1;
                if (sm.ucell[mid] <= e) lo_ = mid;
                else hi_ = mid;
            }
            r = lo_;
            l = e - sm.ucell[r];
        } else {
            r = replica_of_cell(v, e);
            l = e - v.rep[r].cell_off;
        }
        const Replica &p = v.rep[r];
        if (!cells_serve<MODE>(p)) continue; // uniform across the block
        const int nc0 = p.nc[0], nc1 = p.nc[1], nc2 = p.nc[2];
        if (l >= nc0 * nc1 * nc2) continue;
        const int cell = p.cell_off + l;
        const int cx = l % nc0, cy = (l / nc0) % nc1, cz = l / (nc0 * nc1);
        // stencil position o = lane: slot 13 + o (the own cell first)
        if (t < 32) {
            int st = 0, cnt = 0;
            if (lane < 14) {
                const int u = 13 + lane;
                int x = cx + u % 3 - 1, y = cy + (u / 3) % 3 - 1, z = cz + u / 9 - 1;
                x += x < 0 ? nc0 : (x >= nc0 ? -nc0 : 0);
                y += y < 0 ? nc1 : (y >= nc1 ? -nc1 : 0);
                z += z < 0 ? nc2 : (z >= nc2 ? -nc2 : 0);
                const int cn = p.cell_off + (z * nc1 + y) * nc0 + x;
                st = v.cell_start[cn];
                cnt = v.cell_start[cn + 1] - st;
            }
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane < 14) {
                sm.start[lane] = st;
                sm.pre_n[lane] = inc - cnt;
            }
            if (lane == 13) sm.pre_n[14] = inc;
        }
        __syncthreads();
        const int na = sm.pre_n[1], nall = sm.pre_n[14], g0 = sm.start[0];
        const double lam = MODE == 2 ? 1.0 : p.vol_lambda, lam2 = lam * lam;
        const double Ls[3] = {__dmul_rn(p.L[0], lam), __dmul_rn(p.L[1], lam), __dmul_rn(p.L[2], lam)};
        const FastK K = fast_consts(p.k);
        const float wx = (float)p.w[0], wy = (float)p.w[1], wz = (float)p.w[2];
        // reach tests in half precision, as the FP32 phase kernel's: the power of two that brings two cells into
        // [4, 8), and the slack for the operands' rounding; the cutoff at the larger volume's scale
        const float wmax = fmaxf(wx, fmaxf(wy, wz));
        const float sc = __int_as_float((129 + 127 - ((__float_as_int(2.0f * wmax) >> 23) & 0xff)) << 23);
        const float slack = 1.75f / 2048.0f * 2.5f * wmax + 1e-3f;
        const float reach = ((float)p.k.rc * fmaxf(1.0f, 1.0f / (float)lam) * 1.00001f + slack) * sc;
        double a0 = 0.0, a1 = 0.0;
        int hard = 0;
        // colloid term of own-cell particle k at V (thread 2k) and at V' with the hard-core test (thread 2k + 1)
        if (MODE != 2 || p.k.coll_on)
            for (int s = t; s < 2 * na; s += 128) {
                const int i = g0 + (s >> 1);
                const double ri[3] = {v.px[i], v.py[i], v.pz[i]};
                if (s & 1) {
                    if (MODE == 2) continue;
                    const double rs[3] = {__dmul_rn(ri[0], lam), __dmul_rn(ri[1], lam), __dmul_rn(ri[2], lam)};
                    if (p.k.coll_on) {
                        const double ei[3] = {v.ox[i], v.oy[i], v.oz[i]};
                        a1 = __dadd_rn(a1, colloid_rod(p.k, rs, ei, Ls)); // (not contracted into the term)
                    }
                    double d[3];
                    const double r2 = dist_fold(rs[0], rs[1], rs[2], __dmul_rn(0.5, Ls[0]), __dmul_rn(0.5, Ls[1]),
                                                __dmul_rn(0.5, Ls[2]), Ls, d);
                    hard += !(r2 > __dmul_rn(p.k.coll_R, p.k.coll_R));
                } else if (p.k.coll_on) {
                    const double ei[3] = {v.ox[i], v.oy[i], v.oz[i]};
                    a0 = __dadd_rn(a0, colloid_rod(p.k, ri, ei, p.L));
                }
            }
        if (na > VC_OWN) { // (uniform)
            double s[2];
            cell_pairs_global<MODE, SPEC21>(&v, r, sm.start, sm.pre_n, Ls, s);
            a0 += s[0];
            a1 += s[1];
        } else {
            const int fcap = VC_CAP - na; // forward particles per chunk
            for (int cs = na; cs == na || cs < nall; cs += fcap) {
                const bool first = cs == na;
                const int total = na + min(fcap, nall - cs); // staged slots of this chunk
                // own cell (first chunk) at slots [0, na), forward particles [cs, cs + fcap) after it
                for (int s_ = first ? t : na + t; s_ < total; s_ += 128) {
                    const int f = s_ < na ? s_ : cs + (s_ - na); // particle index over the stencil positions
                    // largest stencil position whose prefix is <= f (empty positions never match)
                    int o = 0, hi_ = 14;
                    while (hi_ - o > 1) {
                        const int mid = (o + hi_) >> 1;
                        if (sm.pre_n[mid] <= f) o = mid;
                        else hi_ = mid;
                    }
                    const int u = 13 + o;
                    const int g = sm.start[o] + (f - sm.pre_n[o]);
                    const double x = v.px[g], y = v.py[g], z = v.pz[g];
                    sm.px[s_] = x;
                    sm.py[s_] = y;
                    sm.pz[s_] = z;
                    if (MODE == 2) sm.slot[s_] = g;
                    if (MODE != 1) {
                        const double e0 = v.ox[g], e1 = v.oy[g], e2 = v.oz[g];
                        const double in = rsqrt(__fma_rn(e2, e2, __fma_rn(e1, e1, e0 * e0)));
                        sm.ux[s_] = e0 * in;
                        sm.uy[s_] = e1 * in;
                        sm.uz[s_] = e2 * in;
                    }
                    // position relative to the own cell's centre: the FP32 copy's (relative to the particle's own
                    // cell's origin), or formed as the gather forms it, plus the stencil offset
                    float lx, ly, lz;
                    if (p.use_fast) {
                        const float4 c4 = v.cl4[g];
                        lx = c4.x;
                        ly = c4.y;
                        lz = c4.z;
                        if (MODE == 1) {
                            const float2 c2 = v.cl2[g];
                            sm.fx[s_] = c4.w;
                            sm.fy[s_] = c2.x;
                            sm.fz[s_] = c2.y;
                        }
                    } else {
                        int xc = cx + u % 3 - 1, yc = cy + (u / 3) % 3 - 1, zc = cz + u / 9 - 1;
                        xc += xc < 0 ? nc0 : (xc >= nc0 ? -nc0 : 0);
                        yc += yc < 0 ? nc1 : (yc >= nc1 ? -nc1 : 0);
                        zc += zc < 0 ? nc2 : (zc >= nc2 ? -nc2 : 0);
                        lx = (float)fold_rel(x, p.shift[0] + (double)xc * p.w[0], 0.5 * p.w[0], p.L[0], 1.0 / p.L[0]);
                        ly = (float)fold_rel(y, p.shift[1] + (double)yc * p.w[1], 0.5 * p.w[1], p.L[1], 1.0 / p.L[1]);
                        lz = (float)fold_rel(z, p.shift[2] + (double)zc * p.w[2], 0.5 * p.w[2], p.L[2], 1.0 / p.L[2]);
                    }
                    lx = (lx + ((float)(u % 3 - 1) - 0.5f) * wx) * sc;
                    ly = (ly + ((float)((u / 3) % 3 - 1) - 0.5f) * wy) * sc;
                    lz = (lz + ((float)(u / 9 - 1) - 0.5f) * wz) * sc;
                    const __half2 xy = __floats2half2_rn(lx, ly);
                    const __half hz = __float2half_rn(lz);
                    const float hx = __low2float(xy), hy = __high2float(xy), hzf = __half2float(hz);
                    const __half hs = __float2half_rd(hx * hx + hy * hy + hzf * hzf);
                    sm.ch[s_] = make_uint2(tc::h2_bits(xy), tc::h2_bits(__halves2half2(hz, hs)));
                }
                sm.ch[total + t] = make_uint2(0u, 0x7b000000u); // beyond the last: far from everything (VC_BLK = 128)
                __syncthreads();
                // a warp's work: eight own particles by VC_BLK staged slots (slots before both are the own cell's)
                const int nt = (na + 7) >> 3, lo = first ? 0 : na, nb = (total - lo + VC_BLK - 1) / VC_BLK;
                // four at a time, one per warp; their lists together are evaluated by the whole block
                for (int it0 = 0; it0 < nt * nb; it0 += 4) {
                    const int it = it0 + w;
                    const int k0 = 8 * (it % nt), b0s = lo + VC_BLK * (it / nt);
                    // none left, or every slot of the block is below the tile's particles
                    const bool idle = it >= nt * nb || b0s + VC_BLK <= k0;
                    unsigned x0 = 0u, x1 = 0u;
                    int n = 0, pos = 0;
                    const int g = lane >> 2, q = lane & 3;
                    if (!idle) {
                        // columns of the product: particle k0 + g (its operand), k0 + 2q and k0 + 2q + 1 (their constants)
                        auto square = [&](int k) {
                            if (k >= na) return 1e30f;
                            const uint2 h = sm.ch[k];
                            const __half2 xy = *reinterpret_cast<const __half2 *>(&h.x), zs = *reinterpret_cast<const __half2 *>(&h.y);
                            const float x = __low2float(xy), y = __high2float(xy), z = __low2float(zs);
                            return x * x + y * y + z * z - reach * reach;
                        };
                        const float c0 = square(k0 + 2 * q), c1 = square(k0 + 2 * q + 1);
                        unsigned bq = 0u;
                        if (q < 2) {
                            const __half2 m2 = __floats2half2_rn(-2.0f, -2.0f);
                            const uint2 h = sm.ch[min(k0 + g, na - 1)];
                            const unsigned y = q == 0 ? h.x : (h.y & 0xffffu);
                            bq = tc::h2_bits(__hmul2(*reinterpret_cast<const __half2 *>(&y), m2));
                            if (q == 1) bq = (bq & 0xffffu) | 0x3c000000u; // (-2z, 1)
                        }
                        const unsigned *ah = reinterpret_cast<const unsigned *>(sm.ch) + 2 * (b0s + g) + (q & 1);
#pragma unroll
                        for (int i = 0; i < VC_BLK / 16; i++) {
                            float d[4];
                            tc::mma_16x8x8(d, ah[32 * i], ah[32 * i + 16], bq, c0, c1);
                            x0 = __funnelshift_l(__float_as_uint(d[0]), x0, 1);
                            x1 = __funnelshift_l(__float_as_uint(d[1]), x1, 1);
                            x0 = __funnelshift_l(__float_as_uint(d[2]), x0, 1);
                            x1 = __funnelshift_l(__float_as_uint(d[3]), x1, 1);
                        }
                        // bit 15 - z of a mask: slot b0s + g + 8 z; only slots after the particle itself
                        const int ka = k0 + 2 * q, kb = ka + 1;
                        const int za = (ka - b0s - g) >> 3, zb = (kb - b0s - g) >> 3; // slots z <= za are at or below ka
                        x0 &= za < 0 ? 0xffffu : (za >= 15 ? 0u : 0xffffu >> (za + 1));
                        x1 &= zb < 0 ? 0xffffu : (zb >= 15 ? 0u : 0xffffu >> (zb + 1));
                        n = __popc(x0) + __popc(x1);
                        pos = n;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const int y = __shfl_up_sync(0xffffffffu, pos, o);
                            if (lane >= o) pos += y;
                        }
                    }
                    if (lane == 31) sm.nlist[w] = pos;
                    __syncthreads();
                    int ne = 0;
                    for (int i = 0; i < 4; i++) {
                        if (i < w) pos += sm.nlist[i];
                        ne += sm.nlist[i];
                    }
                    unsigned *out = sm.list + pos - n;
                    const unsigned ea = (unsigned)(k0 + 2 * q) << 16 | (unsigned)(b0s + g);
                    while (x0) {
                        const int z = __clz(x0) - 16;
                        x0 ^= 0x8000u >> z;
                        *out++ = ea + 8 * z;
                    }
                    while (x1) {
                        const int z = __clz(x1) - 16;
                        x1 ^= 0x8000u >> z;
                        *out++ = ea + (1u << 16) + 8 * z;
                    }
                    __syncthreads();
                    for (int i = t; i < ne; i += 128) {
                        const unsigned en = sm.list[i];
                        const int k = (int)(en >> 16), j = (int)(en & 0xffffu);
                        const double ri[3] = {sm.px[k], sm.py[k], sm.pz[k]}, rj[3] = {sm.px[j], sm.py[j], sm.pz[j]};
                        double ui[3], uj[3];
                        float fi[3], fj[3];
                        if (MODE == 1) {
                            fi[0] = sm.fx[k], fi[1] = sm.fy[k], fi[2] = sm.fz[k];
                            fj[0] = sm.fx[j], fj[1] = sm.fy[j], fj[2] = sm.fz[j];
                        } else {
                            ui[0] = sm.ux[k], ui[1] = sm.uy[k], ui[2] = sm.uz[k];
                            uj[0] = sm.ux[j], uj[1] = sm.uy[j], uj[2] = sm.uz[j];
                        }
                        cell_pair<MODE, SPEC21>(v, r, MODE == 2 ? sm.slot[k] : 0, MODE == 2 ? sm.slot[j] : 0, p, K, ri, rj,
                                                ui, uj, fi, fj, lam, lam2, Ls, a0, a1);
                    }
                    __syncthreads(); // the lists are written again
                }
            }
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, o);
            a1 += __shfl_xor_sync(0xffffffffu, a1, o);
        }
        if (lane == 0) {
            sm.red[w][0] = a0;
            sm.red[w][1] = a1;
        }
        const int nh = __syncthreads_count(hard > 0); // threads with a centre inside the colloid
        if (t == 0) {
            v.cell_e0[cell] = (sm.red[0][0] + sm.red[1][0]) + (sm.red[2][0] + sm.red[3][0]);
            v.cell_e1[cell] = (sm.red[0][1] + sm.red[1][1]) + (sm.red[2][1] + sm.red[3][1]);
            v.cell_n1[cell] = nh;
        }
        // (the next cell's stencil is written before its barrier; red is read by thread 0 before that)
    }
}

} // namespace lcmc
