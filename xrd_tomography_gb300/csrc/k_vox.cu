// k_vox.cu -- the model with per-voxel coefficients: forward, adjoint and
// the MLEM update, matrix-free, for a batch of independent problems.
//
// The reference's model matrix has one unknown per (coarse q bin, material):
// Amatrix[k, m, ray] = sum over the voxels of material m of the coarse-q
// term of integrate_diffraction.cu:311-315,
//
//   Av[ray, v, k] = sum_{e in window(nrg)} RF[e,nrg] Pin Pout geom Rayleigh
//                   * G(wvt(v,e) - q_k; sigma(v,e)) * dq_k .
//
// With one unknown per (voxel, coarse bin), x[v, k], the forward model is
// y = Av x and its adjoint g = Av^T w.  Both are computed on the fly; the
// source-side attenuation comes from the per-(source, voxel) table.
//
// Every kernel takes a batch of problems (phantoms and scanners of any
// size, VoxJob); a single operator is a batch of one.  The two heavy kernels
// are persistent: a grid sized to the GPU takes work items from an atomic
// counter -- the (source, pixel) pairs of all problems for the forward, the
// (voxel chunk, pair group) tiles of all problems for the adjoint -- so that
// uneven problems share one launch and the tail stays short.
//
// The detector-side integrals of each (pair, voxel) come from a table: the
// operator's own (VoxOp::walk, walked once by k_walk.cu when the operator is
// created) or the current tile of a walk streamed inside the call.
//
//  * forward (k_vox_fwd): one item = one (source, pixel) pair, as in
//    k_fwd.cu: tiles of voxels with their scattering geometry and their
//    coefficients x[v, k] dq_k in shared memory, runs of 32-voxel steps of two
//    neighbouring energies off a counter, lane = voxel; a lane sums the coarse
//    bins within 7.5 sigma of either wavevector transfer, two per instruction,
//    and reads a voxel's constants and a bin's coefficient once for both.  The banded
//    spectrum weights give the detector bins.  In MLEM mode the block goes on
//    to form the ratios y / (Av x + c + 1e-20) of main.m:162 for its detector
//    bins and folds them back through the same weights, what[pair, e].
//  * adjoint (k_vox_adj): voxel-major, so that g stays on chip.  A warp owns
//    32 voxels, one per lane, and loops over a group of pairs: geometry once
//    per pair, then per two energies the lane adds what[pair,e] times their
//    terms to its own column of sums over the bins within 13.25 sigma, two
//    bins per instruction; at a pair's end the column goes into the partial
//    row with a two-sum.  The groups' partial sums
//    (float pairs) are added in FP64 by k_vox_reduce, which also applies the
//    MLEM update (main.m:163-176).
//
// Both are bound by instruction issue.  The bins of a window come from a table
// over the wavevector axis (VoxOp::qlut) instead of two square roots and
// quotients, whose index is clamped by the addition that forms it.  Measured on
// 128x128 voxels, 32 views x 128 px, 40 energies, 32 bins: forward 4.6 ms (5.3 with
// one energy at a time, which kept shared memory busy 58 % of the time; 5.5 with
// integer clamps and renormalised pairs), 10.1 with lane = energy; 7.9 before the scattering geometry lost
// its component-wise form (vox_geom) and the coefficients' transposition moved
// out of the tiles.  Adjoint of 96x78 voxels, 27 views x 110 px, 40 energies, 40
// bins: 2.1 ms (2.2), 8.7 with lane = energy for the terms, scans over the energies for
// each bin's range and lane = bin for the sums; 3.8 with compensated sums in
// shared memory, one energy per visit to a bin.
#include "scatter.cuh"

namespace xrdt {

namespace {

// Two blocks of 8 warps per SM at 128 registers: two energies at a time spill at
// 80 (three blocks: 4.9 ms against 4.75 at 128x128, 4.6 with the larger tiles; 10
// and 12 warps 4.6 and 5.0).
constexpr int kFwdWarps = 8;
constexpr int kFwdThreads = 32 * kFwdWarps;
constexpr int kMaxSteps = 24;   // 32-voxel steps of a tile

// A voxel's constants against one (source, pixel) pair.
struct VoxTerm {
    ff ax, ay;        // sums of both line integrals, unrounded: the rounding would be
                      // one error in every energy's and bin's term of the pair
    ff t1, b;         // sigma^2 = t1 + c2(e) b: c1 s^2 and sg / s^2 as pairs
    float sh, sl;     // sin(theta/2)
    float wr;         // geom Rayleigh / sqrt(2 pi)
};

// Per-(voxel, energy) factors shared by the forward and the adjoint: the
// prefactor pref = Pin Pout geom Rayleigh / (sigma sqrt(2 pi)) without RF,
// the wavevector transfer as a pair, the Gaussian exponent scale (log2
// units, as a pair) and sigma.
struct EnergyTerm {
    float pref, w_hi, w_lo, c_hi, c_lo, sigma;
};

__device__ __forceinline__ EnergyTerm energy_term(const VoxEnergy &q, const VoxTerm &v)
{
    EnergyTerm t;
    // exp(-X) with 1/f1 and 1/f2 as pairs in units of log2
    const float low = fmaf(v.ax.hi, q.f1l, fmaf(v.ay.hi, q.f2l, fmaf(v.ax.lo, q.f1, v.ay.lo * q.f2)));
    const float PP = ex2_approx(fmaf(v.ax.hi, q.f1, fmaf(v.ay.hi, q.f2, low)));
    // (the pairs here stay as they come out: their low parts are an ulp or two
    // of the high ones, and every use takes both)
    t.w_hi = __fmul_rn(q.wh, v.sh);
    t.w_lo = fmaf(q.wh, v.sh, -t.w_hi) + fmaf(q.wh, v.sl, q.wl * v.sh);
    // sigma^2 as a pair: deep in the Gaussian's tail the exponent amplifies
    // its relative error by (q distance / sigma)^2 / 2
    const float p = __fmul_rn(q.c2, v.b.hi);
    const float e = fmaf(q.c2, v.b.lo, fmaf(q.c2l, v.b.hi, fmaf(q.c2, v.b.hi, -p)));
    ff s2 = two_sum(v.t1.hi, p);
    s2.lo += e + v.t1.lo;
    // 1/sigma to within an ulp: one Newton step on rsqrt, with the low part
    const float r0 = rsqrt_approx(s2.hi);
    const float h = fmaf(-0.5f * s2.hi * r0, r0, 0.5f) - 0.5f * s2.lo * r0 * r0;
    const float rs = fmaf(r0, h, r0);
    const ff c = gauss_scale(s2, rs * rs);
    t.c_hi = c.hi;
    t.c_lo = c.lo;
    t.pref = PP * v.wr * rs;
    t.sigma = s2.hi * rs;
    return t;
}

// The scattering geometry and line integrals of a voxel against a pair.
__device__ __forceinline__ VoxTerm vox_term(const PairGeom &G, const F32Consts &c, ff c1, int xy, float2 As, float2 Ad)
{
    const float vx = ((float)(xy & 0xffff) + 0.5f) * c.vox;
    const float vy = ((float)(xy >> 16) + 0.5f) * c.vox;
    const VoxGeom g = vox_geom<true>(G, vx, vy);
    VoxTerm v;
    v.ax = two_sum(Ad.x, As.x);
    v.ay = two_sum(Ad.y, As.y);
    v.t1 = ff_mul(c1, g.s2);
    v.b = ff_mul(g.sg, ffl_rcp(g.s2));
    v.sh = g.s.hi;
    v.sl = g.s.lo;
    v.wr = g.Wg * c.rsqrt2pi;
    return v;
}

// The window table as the kernels index it: entry round(M u) of shared memory,
// u = w scale + offset clamped to [0, 1] by the addition that forms it.
struct WindowTable {
    float scale, offset;   // ((w - q_lo) cells + 1/2) / M
    uint32_t base;         // address of entry 0, less the magic number's bits
};
constexpr float kLutM = (float)(kLutCells + 1);

__device__ __forceinline__ WindowTable window_table(const unsigned *lut, float scale, float q_lo)
{
    WindowTable t;
    t.scale = scale * (1.f / kLutM);
    t.offset = fmaf(-q_lo, t.scale, 0.5f / kLutM);
    t.base = (uint32_t)__cvta_generic_to_shared(lut) - (0x4B400000u << 2);
    return t;
}

// The first and last coarse bin that may lie within `half` (times the table's
// scale) of w: the table's cells of both ends, entry 0 below the grid and
// kLutCells + 1 above it.
__device__ __forceinline__ void bin_window(const WindowTable &L, float w, float half, int *k0, int *k1)
{
    const float x = fmaf(w, L.scale, L.offset);
    // to the nearest entry through the float mantissa
    const uint32_t i0 = __float_as_uint(fmaf(__saturatef(x - half), kLutM, 12582912.f));
    const uint32_t i1 = __float_as_uint(fmaf(__saturatef(x + half), kLutM, 12582912.f));
    unsigned short lo, hi;   // the entry's halves: first bin, last bin
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(lo) : "r"(L.base + (i0 << 2)));
    asm volatile("ld.shared.s16 %0, [%1+2];" : "=h"(hi) : "r"(L.base + (i1 << 2)));
    *k0 = lo;
    *k1 = (short)hi;
}

// 2^(c (w - q)^2) at two neighbouring bins, q = (hi, hi, lo, lo): the
// argument in FP32 but c as a pair -- the scale carries the systematic part of
// the error (sigma), the difference and its square round independently per
// term.
__device__ __forceinline__ float2 gauss2(const EnergyTerm &t, float4 q)
{
    const float2 d = __fadd2_rn(__fadd2_rn(make_float2(t.w_hi, t.w_hi), make_float2(-q.x, -q.y)),
                                __fadd2_rn(make_float2(t.w_lo, t.w_lo), make_float2(-q.z, -q.w)));
    const float2 d2 = __fmul2_rn(d, d);
    const float2 x = __ffma2_rn(make_float2(t.c_hi, t.c_hi), d2, __fmul2_rn(make_float2(t.c_lo, t.c_lo), d2));
    return make_float2(ex2_approx(x.x), ex2_approx(x.y));
}

__device__ __forceinline__ VoxEnergy load_energy(const VoxEnergy *en, int el)
{
    const float4 a = ((const float4 *)en)[2 * el], b = ((const float4 *)en)[2 * el + 1];
    return VoxEnergy{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

// Stages the tables of a job with every thread of the block: energy rows, bin
// pairs (negative would be the pad of an odd count: far off the grid) and the
// window table.
__device__ __forceinline__ void stage_tables(const VoxJob &J, VoxEnergy *en, float4 *cq, unsigned *lut)
{
    const int K = J.op.P.nwt;
    const float4 *src = (const float4 *)(J.op.vox_energy + J.op.P.e_lo);
    for (int i = threadIdx.x; i < 2 * J.E; i += blockDim.x) ((float4 *)en)[i] = __ldg(src + i);
    for (int i = threadIdx.x; 2 * i < K; i += blockDim.x) {
        const float4 a = J.op.coarse_q[2 * i];
        const float4 b = 2 * i + 1 < K ? J.op.coarse_q[2 * i + 1] : make_float4(1e15f, 0.f, 0.f, 0.f);
        cq[i] = make_float4(a.x, b.x, a.y, b.y);
    }
    for (int i = threadIdx.x; i < kLutCells + 2; i += blockDim.x) lut[i] = __ldg(J.op.qlut + i);
}

// The problem that work item t belongs to: the last p with off[p] <= t.
__device__ __forceinline__ int find_job(const int64_t *__restrict__ off, int n, int64_t t)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(off + mid) <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Copies a job into shared memory with every thread of the block.
__device__ __forceinline__ void load_job(const VoxJob *__restrict__ jobs, int p, VoxJob *dst)
{
    static_assert(sizeof(VoxJob) % 4 == 0, "job size");
    const int *src = reinterpret_cast<const int *>(jobs + p);
    int *d = reinterpret_cast<int *>(dst);
    for (int i = threadIdx.x; i < (int)(sizeof(VoxJob) / 4); i += blockDim.x) d[i] = __ldg(src + i);
}

struct FwdLayout {
    size_t rec, xs, en, cq, lut, tns, tn, ratio, total;
    int xstride;   // floats of a row of two bins
};

__host__ __device__ inline size_t al16(size_t x) { return (x + 15) & ~(size_t)15; }

__host__ __device__ inline FwdLayout vox_fwd_layout(const DevProblem &P, int E, int steps, int runs)
{
    FwdLayout L;
    L.xstride = 64 * steps;   // two bins of every voxel of the tile side by side
    size_t o = 0;
    L.rec = o; o = al16(o + sizeof(float4) * 3 * 32 * (size_t)steps);
    L.xs = o; o = al16(o + sizeof(float) * (size_t)((P.nwt + 1) / 2) * L.xstride);
    L.en = o; o = al16(o + sizeof(VoxEnergy) * E);
    L.cq = o; o = al16(o + sizeof(float4) * ((P.nwt + 1) / 2));
    L.lut = o; o = al16(o + sizeof(unsigned) * (kLutCells + 2));
    L.tns = o; o = al16(o + sizeof(float2) * (size_t)E * runs);
    L.tn = o; o = al16(o + sizeof(double) * E);
    L.ratio = o; o = al16(o + sizeof(double) * P.nrg_det);
    L.total = o;
    return L;
}

// A voxel's constants from its record i of a tile of 32 nst voxels.
__device__ __forceinline__ VoxTerm load_term(const float4 *rec, int nst, int i)
{
    const float4 r0 = rec[i], r1 = rec[32 * nst + i], r2 = rec[64 * nst + i];
    return {{r0.x, r2.y}, {r0.y, r2.z}, {r0.z, r0.w}, {r1.z, r1.w}, r1.x, r1.y, r2.x};
}

// The window bin by bin; every bin where sigma is NaN -- sigma^2 is negative for a
// detector of negative area (adet12 < 0) -- whose term is NaN at each.
__device__ __forceinline__ void own_window(const WindowTable &L, const EnergyTerm &t, float sigmas, int K, int *k0,
                                           int *k1)
{
    bin_window(L, t.w_hi, sigmas * L.scale * t.sigma, k0, k1);
    if (isnan(t.sigma)) {
        *k0 = 0;
        *k1 = K - 1;
    }
}

// Component k & 1 of a pair of bins.
__device__ __forceinline__ float bin_of(float2 v, int k) { return k & 1 ? v.y : v.x; }

// A run's sum at one energy, bin by bin over that energy's own window: for runs
// whose sum is not finite and detectors of negative area.  An infinite coefficient outside the window -- within a
// neighbouring energy's, or beside it in a pair -- must not reach the sum, nor one
// whose term underflows, as 0 x inf.
__device__ __noinline__ float run_by_window(const float4 *rec, const float *xs, const float4 *cq, int x_row,
                                            const VoxEnergy *en, int el, int nst, int s0, int s1, WindowTable window,
                                            int K)
{
    const int lane = threadIdx.x & 31;
    const VoxEnergy q = load_energy(en, el);
    float sum = 0.f;
    for (int st = s0; st < s1; st++) {
        const int i = 32 * st + lane;
        const EnergyTerm t = energy_term(q, load_term(rec, nst, i));
        if (t.pref == 0.f) continue;
        int k0, k1;
        own_window(window, t, kSig, K, &k0, &k1);
        float acc = 0.f;
        for (int k = k0; k <= k1; k++) {
            const float g = bin_of(gauss2(t, cq[k >> 1]), k);
            if (g != 0.f) acc = fmaf(g, xs[(k >> 1) * x_row + 2 * i + (k & 1)], acc);
        }
        sum = fmaf(t.pref, acc, sum);
    }
    return warp_sum(sum);
}

// One (source, pixel) pair of job J, by the whole block; the job's tables are
// staged.
template <bool MLEM>
__device__ __forceinline__ void vox_fwd_pair(const VoxJob &J, int64_t pidx, unsigned char *sm, PairRec &pair,
                                             int &next_run)
{
    const DevProblem &P = J.op.P;
    const F32Consts &c = J.c;
    const int E = J.E, K = P.nwt, W = 2 * P.dnrg + 1, nv = J.op.nv;
    const int nst = J.steps, H = J.runs, run_len = (nst + H - 1) / H;
    const FwdLayout L = vox_fwd_layout(P, E, nst, H);
    float4 *rec = (float4 *)(sm + L.rec);          // [3][32 nst]
    float *xs = (float *)(sm + L.xs);              // [(K + 1)/2][32 nst] x dq of bins 2i, 2i + 1
    const VoxEnergy *en = (const VoxEnergy *)(sm + L.en);
    const float4 *cq = (const float4 *)(sm + L.cq);
    const unsigned *lut = (const unsigned *)(sm + L.lut);
    float2 *TNs = (float2 *)(sm + L.tns);          // [E][runs] compensated sums
    double *TN = (double *)(sm + L.tn);
    double *ratio = (double *)(sm + L.ratio);      // kept in FP64: see the weights below
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t npairs = (int64_t)P.n_src * P.n_det;

    for (int i = tid; i < (int)(sizeof(PairRec) / 4); i += kFwdThreads)
        reinterpret_cast<int *>(&pair)[i] = reinterpret_cast<const int *>(J.op.pairs + pidx)[i];
    for (int i = tid; i < E * H; i += kFwdThreads) TNs[i] = make_float2(0.f, 0.f);
    const ff c1 = {J.op.c1, J.op.c1l};
    const WindowTable window = window_table(lut, J.op.lut_scale, J.c.q_lo);
    const float half_sig = kSig * window.scale;
    const int x_row = L.xstride;

    for (int tile = 0; tile < J.tiles; tile++) {
        const int t0 = 32 * nst * tile;
        __syncthreads();   // the tables and the pair are staged; the last tile is no longer read
        if (tid == 0) next_run = 0;
        // the tile's coefficients (rows of two bins of the tile's voxels),
        // copied while the geometry is formed
        const int steps = min(nst, (nv - t0 + 31) >> 5);
        for (int k = wid; k < (K + 1) >> 1; k += kFwdWarps) {
            const float *src = J.xd + 2 * ((int64_t)k * J.xd_stride + t0) + 4 * lane;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(xs + k * x_row + 4 * lane);
            for (int i = 0; i < 16 * steps; i += 32)
                if (i + lane < 16 * steps)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * i), "l"(src + 4 * i)
                                 : "memory");
        }
        for (int i = tid; i < 32 * nst && t0 + (i & ~31) < nv; i += kFwdThreads) {
            const int v = min(t0 + i, nv - 1);
            const VoxTerm t = vox_term(pair.G, c, c1, J.op.vox_xy[v], J.op.atten_src[(int64_t)pair.src * nv + v],
                                       J.op.walk[(pidx - J.pair0) * nv + v]);
            rec[i] = make_float4(t.ax.hi, t.ay.hi, t.t1.hi, t.t1.lo);
            rec[32 * nst + i] = make_float4(t.sh, t.sl, t.b.hi, t.b.lo);
            // a lane past the last voxel repeats it with a weight of zero
            rec[64 * nst + i] = make_float4(t0 + i < nv ? t.wr : 0.f, t.ax.lo, t.ay.lo, 0.f);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // ---- lane = voxel: runs of 32-voxel steps of two neighbouring energies,
        // the widest windows first ----
        const int EP = (E + 1) >> 1;
        for (;;) {
            int item = 0;
            if (lane == 0) item = atomicAdd(&next_run, 1);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= EP * H) break;
            const int el = 2 * (EP - 1 - item / H), run = item % H;
            const int two = el + 1 < E;   // 0: the second energy is the first again, not kept
            const int s0 = run * run_len, s1 = min(s0 + run_len, steps);
            const VoxEnergy q = load_energy(en, el), q1 = load_energy(en, el + two);
            float sum = 0.f, sum1 = 0.f;
            for (int st = s0; st < s1; st++) {
                const int i = 32 * st + lane;
                const VoxTerm v = load_term(rec, nst, i);
                const EnergyTerm t = energy_term(q, v), u = energy_term(q1, v);
                // Both take the bins of both windows, which lie a source bin
                // apart: a fraction of their length, as sigma holds the width of
                // the source bin.  (pref 0: attenuation underflow, no contribution)
                int k0, k1, l0, l1;
                bin_window(window, t.w_hi, half_sig * t.sigma, &k0, &k1);
                bin_window(window, u.w_hi, half_sig * u.sigma, &l0, &l1);
                if (k0 > k1) k0 = 0xffff, k1 = -1;
                if (l0 > l1) l0 = 0xffff, l1 = -1;
                k0 = min(k0, l0) >> 1;
                k1 = max(k1, l1) >> 1;
                if (k0 <= k1 && (t.pref != 0.f || u.pref != 0.f)) {
                    float2 acc = make_float2(0.f, 0.f), bcc = make_float2(0.f, 0.f);
                    const float2 *x2 = (const float2 *)xs + i;
                    for (int k = k0; k <= k1; k++) {
                        const float4 b = cq[k];
                        const float2 x = x2[k * (x_row >> 1)];
                        acc = __ffma2_rn(gauss2(t, b), x, acc);
                        bcc = __ffma2_rn(gauss2(u, b), x, bcc);
                    }
                    sum = fmaf(t.pref, acc.x + acc.y, sum);
                    sum1 = fmaf(u.pref, bcc.x + bcc.y, sum1);
                }
            }
            sum = warp_sum(sum);
            sum1 = warp_sum(sum1);
            if (!(isfinite(sum) && isfinite(sum1) && pair.G.adet12 >= 0.f)) {
                sum = run_by_window(rec, xs, cq, x_row, en, el, nst, s0, s1, window, K);
                sum1 = run_by_window(rec, xs, cq, x_row, en, el + two, nst, s0, s1, window, K);
            }
            if (lane <= two) {
                const int at = (el + lane) * H + run;
                float2 k = TNs[at];
                kahan_add(k.x, k.y, lane ? sum1 : sum);
                TNs[at] = k;
            }
        }
    }
    __syncthreads();
    for (int el = tid; el < E; el += kFwdThreads) {
        double s = 0.0;
        for (int h = 0; h < H; h++) s += (double)TNs[el * H + h].x - (double)TNs[el * H + h].y;
        TN[el] = s;
    }
    __syncthreads();
    const int lo_e = P.e_lo;
    const float *rf = J.op.rf_win;
    const int *winlo = J.op.win_lo, *wn = J.op.win_n;
    for (int n = tid; n < P.nrg_det; n += kFwdThreads) {
        double acc = 0.0;
        const int w0 = __ldg(winlo + n) - lo_e;
        for (int j = 0; j < W; j++) acc += (double)__ldg(rf + n * W + j) * TN[w0 + j];
        const int64_t ray = pidx + (int64_t)n * npairs;
        if (MLEM) ratio[n] = (double)J.ymeas[ray] / (acc + (double)J.cbg[ray] + 1e-20);   // main.m:162
        else J.y[ray] = (float)acc;
    }
    if (MLEM) {
        __syncthreads();
        // what[pair, e] = sum over the detector bins whose window holds e
        for (int el = tid; el < E; el += kFwdThreads) {
            const int e = lo_e + el;
            double s = 0.0;
            const int n1 = __ldg(wn + 2 * e + 1);
            for (int n = __ldg(wn + 2 * e); n <= n1; n++) {
                const int j = e - __ldg(winlo + n);
                if (j >= 0 && j < W) s += (double)__ldg(rf + n * W + j) * ratio[n];
            }
            J.what[pidx * E + el] = (float)s;
        }
    }
}

// Persistent forward over the pairs of every job (offsets off[0 .. n]).
template <bool MLEM>
__global__ void __launch_bounds__(kFwdThreads, 2)
k_vox_fwd(const VoxBatch B)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ PairRec pair;
    __shared__ VoxJob job;
    __shared__ long long item_s;
    __shared__ int next_run;
    const int64_t *off = B.off + 0 * (B.n + 1);
    const int64_t total = off[B.n];
    int cur = -1;
    for (;;) {
        __syncthreads();   // the previous item is done with shared memory
        if (threadIdx.x == 0) item_s = (long long)atomicAdd(B.counters + 0, 1ull);
        __syncthreads();
        const int64_t item = item_s;
        if (item >= total) break;
        const int p = find_job(off, B.n, item);
        if (p != cur) {
            load_job(B.jobs, p, &job);
            cur = p;
            __syncthreads();
            const FwdLayout L = vox_fwd_layout(job.op.P, job.E, job.steps, job.runs);
            stage_tables(job, (VoxEnergy *)(sm + L.en), (float4 *)(sm + L.cq), (unsigned *)(sm + L.lut));
        }
        vox_fwd_pair<MLEM>(job, job.pair0 + (item - off[p]), sm, pair, next_run);
    }
}

// Shared memory of the adjoint: the job's tables, then per warp the current
// pair's record and weights and its sums, [(K + 1)/2][32] of two bins side by
// side.
struct AdjLayout {
    size_t en, cq, lut, warp0, per_warp, sums, weights, total;
};

__host__ __device__ inline AdjLayout vox_adj_layout(const DevProblem &P, int E, int warps)
{
    AdjLayout L;
    size_t o = 0;
    L.en = o; o = al16(o + sizeof(VoxEnergy) * E);
    L.cq = o; o = al16(o + sizeof(float4) * ((P.nwt + 1) / 2));
    L.lut = o; o = al16(o + sizeof(unsigned) * (kLutCells + 2));
    L.warp0 = o;
    size_t w = al16(sizeof(PairRec));
    L.weights = w; w = al16(w + sizeof(float) * E);
    L.sums = w; w = al16(w + sizeof(float2) * 32 * (size_t)((P.nwt + 1) / 2));
    L.per_warp = w;
    L.total = L.warp0 + w * warps;
    return L;
}

// What a pair adds to this lane's column of sums, energy by energy over each one's own
// window: for pairs with a weight that is not finite, or with a detector of negative area
// (run_by_window).  Returns the first and the last pair of bins touched.
__device__ __noinline__ int2 pair_by_window(VoxTerm v, const VoxEnergy *en, const float4 *cq, const float *ws, int E,
                                            WindowTable window, int K, float2 *sums)
{
    int2 r = {0xffff, -1};
    for (int el = 0; el < E; el++) {
        const EnergyTerm t = energy_term(load_energy(en, el), v);
        const float ct = ws[el] * t.pref;
        int k0, k1;
        own_window(window, t, kSigAdj, K, &k0, &k1);
        if (ct == 0.f || k0 > k1) continue;
        r = make_int2(min(r.x, k0 >> 1), max(r.y, k1 >> 1));
        for (int k = k0; k <= k1; k++) {
            const float g = bin_of(gauss2(t, cq[k >> 1]), k);
            float *s = (float *)(sums + 32 * (k >> 1)) + (k & 1);
            if (g != 0.f) *s = fmaf(ct, g, *s);
        }
    }
    return r;
}

// Adjoint tile (voxel-chunk block bx, pair group by) of job J.  A pair's sums
// over the energies are plain FP32 sums in shared memory, two energies per
// visit to a bin (the visits' loads and stores would bind before the FMA
// pipe); at the pair's end they go into the tile's partial rows in global
// memory with a two-sum, whose low parts are kept: rounded to one float, each
// row would carry the same relative error into every MLEM iteration, where
// the update multiplies it in again and again.  The rows of the tiles in
// flight stay in L2, and shared memory holds twice the warps that it would
// with compensated sums beside the plain ones.
__global__ void __launch_bounds__(128, 6)
k_vox_adj(const VoxBatch B)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ VoxJob J;
    __shared__ long long item_s;
    const int nwarps = blockDim.x >> 5;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int64_t *off = B.off + 1 * (B.n + 1);
    const int64_t total = off[B.n];
    int cur = -1;
    for (;;) {
        __syncthreads();
        if (tid == 0) item_s = (long long)atomicAdd(B.counters + 1, 1ull);
        __syncthreads();
        const int64_t item = item_s;
        if (item >= total) break;
        const int p = find_job(off, B.n, item);
        if (p != cur) {
            load_job(B.jobs, p, &J);
            cur = p;
            __syncthreads();
            const AdjLayout L = vox_adj_layout(J.op.P, J.E, nwarps);
            stage_tables(J, (VoxEnergy *)(sm + L.en), (float4 *)(sm + L.cq), (unsigned *)(sm + L.lut));
            __syncthreads();
        }
        const DevProblem &P = J.op.P;
        const int E = J.E, K2 = (P.nwt + 1) >> 1;
        const AdjLayout L = vox_adj_layout(P, E, nwarps);
        const VoxEnergy *en = (const VoxEnergy *)(sm + L.en);
        const float4 *cq = (const float4 *)(sm + L.cq);
        const unsigned *lut = (const unsigned *)(sm + L.lut);
        unsigned char *mine = sm + L.warp0 + L.per_warp * wid;
        PairRec &pr = *(PairRec *)mine;
        float *ws = (float *)(mine + L.weights);
        float2 *sums = (float2 *)(mine + L.sums) + lane;   // this lane's column

        const int64_t r = item - off[p];
        const int bx = (int)(r % J.chunk_blocks), by = (int)(r / J.chunk_blocks);
        const int nv = J.op.nv, chunks = (nv + 31) >> 5;
        const int chunk = bx * nwarps + wid;
        if (chunk >= chunks) continue;   // an idle warp; the next item starts with a barrier
        const int64_t p0 = J.pair0 + (int64_t)by * J.ppg;
        const int64_t p1 = min(J.pair1, p0 + J.ppg);
        const int v = min(chunk * 32 + lane, nv - 1);   // a lane past the last voxel repeats it
        const int xy = J.op.vox_xy[v];
        const ff c1 = {J.op.c1, J.op.c1l};
        const WindowTable window = window_table(lut, J.op.lut_scale, J.c.q_lo);
        const float half_sig = kSigAdj * window.scale;
        // this lane's column of the partial row: sums of two bins and their low parts
        float4 *row = J.part + ((int64_t)by * chunks + chunk) * K2 * 32 + lane;
        for (int k = 0; k < K2; k++) sums[32 * k] = make_float2(0.f, 0.f);
        // a job that is one tile of a problem adds to what the earlier tiles left
        // (tiles run in a fixed order on one stream)
        if (!J.accumulate)
            for (int k = 0; k < K2; k++) row[32 * k] = make_float4(0.f, 0.f, 0.f, 0.f);

        for (int64_t pp = p0; pp < p1; pp++) {
            __syncwarp();   // the previous pair's constants are no longer read
            for (int i = lane; i < (int)(sizeof(PairRec) / 4); i += 32)
                reinterpret_cast<int *>(&pr)[i] = reinterpret_cast<const int *>(J.op.pairs + pp)[i];
            bool finite = true;
            for (int i = lane; i < E; i += 32) {
                const float w = __ldg(J.what + pp * E + i);
                ws[i] = w;
                finite &= isfinite(w);
            }
            __syncwarp();   // (the vote orders no memory)
            const int by_two = __all_sync(0xffffffffu, finite && pr.G.adet12 >= 0.f);
            const VoxTerm vt = vox_term(pr.G, J.c, c1, xy, J.op.atten_src[(int64_t)pr.src * nv + v],
                                        J.op.walk[(pp - J.pair0) * nv + v]);
            int kmin = K2, kmax = -1;   // the pairs of bins this lane adds to
            if (!by_two) {
                const int2 k = pair_by_window(vt, en, cq, ws, E, window, P.nwt, sums);
                kmin = min(kmin, k.x);
                kmax = k.y;
            }
            for (int el = by_two ? 0 : E; el < E; el += 2) {
                const EnergyTerm t = energy_term(load_energy(en, el), vt);
                const int e1 = min(el + 1, E - 1);
                const EnergyTerm u = energy_term(load_energy(en, e1), vt);
                const float ct = ws[el] * t.pref, cu = el + 1 < E ? ws[e1] * u.pref : 0.f;
                // the bins within 13.25 sigma: every term FP32 can represent
                int k0, k1, l0, l1;
                bin_window(window, t.w_hi, half_sig * t.sigma, &k0, &k1);
                bin_window(window, u.w_hi, half_sig * u.sigma, &l0, &l1);
                if (ct == 0.f || k0 > k1) k0 = 0xffff, k1 = -1;
                if (cu == 0.f || l0 > l1) l0 = 0xffff, l1 = -1;
                k0 = min(k0, l0) >> 1;
                k1 = max(k1, l1) >> 1;
                if (k0 > k1) continue;
                kmin = min(kmin, k0);
                kmax = max(kmax, k1);
                for (int k = k0; k <= k1; k++) {
                    const float4 q = cq[k];
                    const float2 g = gauss2(t, q), h = gauss2(u, q);
                    sums[32 * k] = __ffma2_rn(make_float2(cu, cu), h, __ffma2_rn(make_float2(ct, ct), g, sums[32 * k]));
                }
            }
            kmin = __reduce_min_sync(0xffffffffu, kmin);
            kmax = __reduce_max_sync(0xffffffffu, kmax);
            for (int k = kmin; k <= kmax; k++) {
                const float4 o = row[32 * k];
                const float2 b = sums[32 * k];
                sums[32 * k] = make_float2(0.f, 0.f);
                const ff x = two_sum(o.x, b.x), y = two_sum(o.y, b.y);
                row[32 * k] = make_float4(x.hi, y.hi, o.z + x.lo, o.w + y.lo);
            }
        }
        __syncwarp();
    }
}

// what[p, e] = sum_nrg RF[e, nrg] w[p + nrg * npairs].  mode 0: the weights
// w; mode 1: every w = 1, the sum rounded to float; mode 2: every w = 1, the
// part of the sum that rounding to float dropped.  The sensitivity is the
// adjoint of mode 1 plus that of mode 2: with one float per energy shared by
// every pair, its rounding would be the same relative error in every term of
// an energy, which no sum over pairs averages out, and MLEM multiplies each
// unknown by (1 + that error) again in every iteration.
__global__ void k_vox_wtab(const VoxBatch B, int mode)
{
    const int64_t *off = B.off + 4 * (B.n + 1);
    const int64_t total = off[B.n];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int pj = find_job(off, B.n, t);
        const VoxJob &J = B.jobs[pj];
        const DevProblem &P = J.op.P;
        const int W = 2 * P.dnrg + 1, E = J.E;
        const int64_t npairs = (int64_t)P.n_src * P.n_det;
        const int64_t loc = t - off[pj];
        const int64_t p = loc / E;
        const int el = (int)(loc - p * E), e = P.e_lo + el;
        double s = 0.0;
        for (int n = J.op.win_n[2 * e]; n <= J.op.win_n[2 * e + 1]; n++) {
            const int j = e - J.op.win_lo[n];
            if (j < 0 || j >= W) continue;
            const double wv = mode ? 1.0 : (double)J.w[p + (int64_t)n * npairs];
            s += (double)J.op.rf_win[n * W + j] * wv;
        }
        J.what[loc] = mode == 2 ? (float)(s - (double)(float)s) : (float)s;
    }
}

// Where x dq of (voxel, bin) lies: rows of two bins, [(K + 1)/2][xd_stride][2],
// as the forward's tiles copy them.
__device__ __forceinline__ int64_t xd_index(const VoxJob &J, int64_t v, int k)
{
    return 2 * ((int64_t)(k >> 1) * J.xd_stride + v) + (k & 1);
}

// Sum of the adjoint's partial rows in FP64, times the bins' widths, and what
// follows from it:
//   mode 0: sens = sum (the sensitivity, Av^T 1)
//   mode 4: sens += sum (its second part, k_vox_wtab)
//   mode 1: the MLEM update x <- x * sum / (sens + 1e-7), non-finite -> 0,
//           negative -> 0 (main.m:162-176), and xd = x dq
//   mode 2: g[voxel] = sum in the full-grid layout (nx + ny*NX)*nwt + k
//   mode 3: g = sum in the compact voxel order [nv][nwt]
// A block takes 32 voxels and two bins, 512 bytes of every partial row.  Its
// warps split the rows and add theirs with two-sums (whose low parts FP32
// holds as well as it held the rows'), then the warps' sums are added in FP64:
// in FP64 throughout and by one thread per entry, 200 rows of 2224 voxels x 40
// bins took 250 us against 65, on a pipe of 1/64 of the FP32 rate.
constexpr int kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps)
k_vox_reduce(const VoxBatch B, int mode)
{
    __shared__ double part_s[kReduceWarps][2][32];
    const int64_t *off = B.off + 5 * (B.n + 1);
    const int64_t total = off[B.n] >> 5;   // (chunk, pair of bins) of every job
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
        const int pj = find_job(off, B.n, 32 * t);
        const VoxJob &J = B.jobs[pj];
        const int K = J.op.P.nwt, K2 = (K + 1) >> 1, nv = J.op.nv;
        const int64_t loc = t - (off[pj] >> 5);
        const int64_t chunk = loc / K2;
        const int k2 = (int)(loc - chunk * K2);
        const int64_t n = off[pj + 1] - off[pj];
        const float4 *part = J.part + 32 * loc + lane;
        ff a = {0.f, 0.f}, b = {0.f, 0.f};
#pragma unroll 4
        for (int gi = wid; gi < J.groups; gi += kReduceWarps) {
            const float4 pv = part[(int64_t)gi * n];
            const ff x = two_sum(a.hi, pv.x), y = two_sum(b.hi, pv.y);
            a = ff{x.hi, a.lo + (x.lo + pv.z)};
            b = ff{y.hi, b.lo + (y.lo + pv.w)};
        }
        part_s[wid][0][lane] = (double)a.hi + (double)a.lo;
        part_s[wid][1][lane] = (double)b.hi + (double)b.lo;
        __syncthreads();
        const int64_t vi = 32 * chunk + lane;
        const int k = 2 * k2 + wid;
        if (wid < 2 && vi < nv && k < K) {
            double sum = 0.0;
#pragma unroll
            for (int w = 0; w < kReduceWarps; w++) sum += part_s[w][wid][lane];
            const float dq = J.op.coarse_q[k].z;
            const double s = sum * (double)dq;
            const int64_t i = vi * K + k;
            if (mode == 0) {
                J.sens[i] = s;
            } else if (mode == 4) {
                J.sens[i] += s;
            } else if (mode == 1) {
                float v = (float)((double)J.xc[i] * s / (J.sens[i] + 1e-7));
                if (!isfinite(v)) v = 0.f;
                if (v < 0.f) v = 0.f;
                J.xc[i] = v;
                J.xd[xd_index(J, vi, k)] = v * dq;
            } else if (mode == 2) {
                const int xy = J.op.vox_xy[vi];
                J.g[((int64_t)(xy & 0xffff) + (int64_t)(xy >> 16) * J.op.P.nx) * K + k] = (float)s;
            } else {
                J.g[i] = (float)s;
            }
        }
        __syncthreads();
    }
}

// Full grid -> compact voxel order: xd = x dq (and xc = x when with_xc).
__global__ void k_vox_gather(const VoxBatch B, int with_xc)
{
    const int64_t *off = B.off + 2 * (B.n + 1);
    const int64_t total = off[B.n];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int pj = find_job(off, B.n, t);
        const VoxJob &J = B.jobs[pj];
        const int K = J.op.P.nwt;
        const int64_t loc = t - off[pj];
        const int64_t vi = loc / K;
        const int k = (int)(loc - vi * K);
        const int xy = J.op.vox_xy[vi];
        const float v = J.xfull[((int64_t)(xy & 0xffff) + (int64_t)(xy >> 16) * J.op.P.nx) * K + k];
        if (with_xc) J.xc[loc] = v;
        J.xd[xd_index(J, vi, k)] = v * J.op.coarse_q[k].z;
    }
}

// Rows [nv][K] of x dq into the forward's layout.
__global__ void k_vox_pack(const float *__restrict__ rows, int64_t nv, int K, int64_t stride, float *__restrict__ xd)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nv * K; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = t / K;
        const int k = (int)(t - v * K);
        xd[2 * ((int64_t)(k >> 1) * stride + v) + (k & 1)] = rows[t];
    }
}

// Compact -> full grid (the other voxels are left as they are).
__global__ void k_vox_scatter(const VoxBatch B)
{
    const int64_t *off = B.off + 2 * (B.n + 1);
    const int64_t total = off[B.n];
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int pj = find_job(off, B.n, t);
        const VoxJob &J = B.jobs[pj];
        const int K = J.op.P.nwt;
        const int64_t loc = t - off[pj];
        const int64_t vi = loc / K;
        const int xy = J.op.vox_xy[vi];
        J.xout[((int64_t)(xy & 0xffff) + (int64_t)(xy >> 16) * J.op.P.nx) * K + (loc - vi * K)] = J.xc[loc];
    }
}

// Pair table: the (source, pixel) constants of a list of pairs or of the
// linear pairs from p0 on.
__global__ void k_pair_table(DevProblem P, const SrcGeom *__restrict__ sg, const int2 *__restrict__ list, int64_t p0,
                             int64_t n, PairRec *__restrict__ out)
{
    allow_dependents();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = p0 + i;
        const int2 pr = list ? list[i] : make_int2((int)(p % P.n_src), (int)(p / P.n_src));
        PairRec r;
        pair_geom(P, sg[pr.x], pr.y, &r.G, &r.Rdx, &r.Rdy);
        r.src = pr.x;
        r.pad = 0;
        out[i] = r;
    }
    await_predecessor();   // launched early it must not end before what came before
}

// a grid-stride loop over n items: at most 32 blocks per SM
int grid_for(int64_t n, int threads)
{
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = 32LL * current_sm_count();
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

template <class F>
cudaError_t allow_dynamic_smem(F *kernel, int max_smem)
{
    // the limit covers static and dynamic shared memory together
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem - (int)fa.sharedSizeBytes);
}

template <class F>
size_t static_smem(F *kernel)
{
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return fa.sharedSizeBytes;
}

} // namespace

size_t pair_rec_bytes() { return sizeof(PairRec); }

cudaError_t launch_pair_table(const DevProblem &P, const SrcGeom *sg, const int2 *list, long long p0, long long n,
                              PairRec *out, cudaStream_t s, int64_t *launches, bool early)
{
    // small blocks: the records are FP64 work, spread over the SMs
    if (launches) (*launches)++;
    return launch_after(k_pair_table, grid_for(n, 32), 32, 0, s, early, P, sg, list, (int64_t)p0, (int64_t)n, out);
}

cudaError_t vox_set_attributes(int max_smem)
{
    // the launches stay free of attribute calls, so they can be captured
    cudaError_t e = allow_dynamic_smem(k_vox_fwd<true>, max_smem);
    if (e == cudaSuccess) e = allow_dynamic_smem(k_vox_fwd<false>, max_smem);
    if (e == cudaSuccess) e = allow_dynamic_smem(k_vox_adj, max_smem);
    return e;
}

size_t vox_fwd_static_smem() { return static_smem(k_vox_fwd<true>); }
size_t vox_adj_static_smem() { return static_smem(k_vox_adj); }

// Bytes of one block with the sums of 32 voxels, as the operator's limit on
// the coarse bins is stated: 256 bytes per bin and the tables.
size_t vox_limit_smem(const DevProblem &P)
{
    const int E = P.e_hi - P.e_lo + 1, K = P.nwt;
    return al16(sizeof(float) * 8 * E) + sizeof(float4) * K + sizeof(float4) * E + sizeof(float2) * 32 * (size_t)K +
           sizeof(PairRec) + sizeof(float) * E + 16 + sizeof(int2) * E + 2 * K;
}

// The forward's tiles and runs: as many voxels per tile as two blocks per SM
// leave room for (up to 768; a voxel takes 48 bytes and 4 per coarse bin), fewer
// blocks only where not even one step of 32 voxels would fit; four runs or
// more per warp.  They depend on the problem alone, so that a batch gives
// the same bits as the operators by themselves.
size_t vox_fwd_split(const DevProblem &P, int nv, int *steps, int *tiles, int *runs)
{
    const int E = P.e_hi - P.e_lo + 1;
    const int chunks = nv > 0 ? (nv + 31) / 32 : 1;
    const size_t stat = vox_fwd_static_smem() + 1024;
    auto runs_of = [&](int st) {
        const int ep = (E + 1) / 2, r = (4 * kFwdWarps + ep - 1) / ep;
        return r < 1 ? 1 : (r > st ? st : r);
    };
    int cap = 1;
    for (int st = 2; st <= kMaxSteps; st++)
        if (vox_fwd_layout(P, E, st, runs_of(st)).total + stat <= 113 * 1024) cap = st;
    *tiles = (chunks + cap - 1) / cap;
    *steps = (chunks + *tiles - 1) / *tiles;
    *runs = runs_of(*steps);
    return vox_fwd_layout(P, E, *steps, *runs).total;
}

size_t vox_adj_smem(const DevProblem &P, int warps) { return vox_adj_layout(P, P.e_hi - P.e_lo + 1, warps).total; }

int vox_fwd_blocks_per_sm(size_t smem)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_vox_fwd<true>, kFwdThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 1;
    }
    return n < 1 ? 1 : n;
}

int vox_adj_blocks_per_sm(int warps, size_t smem)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_vox_adj, 32 * warps, smem) != cudaSuccess) {
        cudaGetLastError();
        n = 1;
    }
    return n < 1 ? 1 : n;
}

cudaError_t launch_vox_forward(const VoxBatch &B, bool mlem, int grid, size_t smem, cudaStream_t s,
                               int64_t *launches)
{
    cudaError_t e = cudaMemsetAsync(B.counters + 0, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    if (mlem) k_vox_fwd<true><<<grid, kFwdThreads, smem, s>>>(B);
    else k_vox_fwd<false><<<grid, kFwdThreads, smem, s>>>(B);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_vox_adjoint(const VoxBatch &B, int grid, size_t smem, cudaStream_t s, int64_t *launches)
{
    cudaError_t e = cudaMemsetAsync(B.counters + 1, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    k_vox_adj<<<grid, 32 * B.adj_warps, smem, s>>>(B);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_vox_wtab(const VoxBatch &B, int64_t total, int mode, cudaStream_t s, int64_t *launches)
{
    k_vox_wtab<<<grid_for(total, 256), 256, 0, s>>>(B, mode);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_vox_reduce(const VoxBatch &B, int64_t total, int mode, cudaStream_t s, int64_t *launches)
{
    k_vox_reduce<<<grid_for(total, 32), 32 * kReduceWarps, 0, s>>>(B, mode);   // a block per 32 entries
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_vox_gather(const VoxBatch &B, int64_t total, bool with_xc, cudaStream_t s, int64_t *launches)
{
    k_vox_gather<<<grid_for(total, 256), 256, 0, s>>>(B, with_xc ? 1 : 0);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_vox_pack(const float *rows, int64_t nv, int K, int64_t stride, float *xd, cudaStream_t s,
                            int64_t *launches)
{
    k_vox_pack<<<grid_for(nv * K, 256), 256, 0, s>>>(rows, nv, K, stride, xd);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_vox_scatter(const VoxBatch &B, int64_t total, cudaStream_t s, int64_t *launches)
{
    k_vox_scatter<<<grid_for(total, 256), 256, 0, s>>>(B);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

} // namespace xrdt
