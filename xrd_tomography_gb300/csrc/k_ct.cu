// k_ct.cu -- transmission CT sinogram: polychromatic source-to-detector
// transmission through the attenuation map, and the same without the
// phantom (gain0).
//
// The reference declares these outputs (Tphotons and gain0, one value per
// source, detector pixel and energy channel) and the two launches that would
// fill them -- integrate_src2det over (SRC, COL) and polychromatic_src2det --
// only as comments (Forward_XRD.cu:125-140,169-199,263-276); no kernel body
// ships.  The definition used here, restated in the oracle:
//
//   chord: the segment source -> pixel clipped to the region of interest
//          [0,NX] x [0,NY] (slab clipping, FP64); samples at
//          r_in + k DQ u for k DQ <= chord length, bilinear in the (a1, a2)
//          map exactly as the line integrals of attenuator.cu:9-109;
//          (A1, A2) = DQ * sum of the samples
//   Tphotons[src, det, nrg] = sum_{e in window(nrg)} RF[e, nrg] exp(-(A1/ein^3 + A2/KN(ein)))
//   gain0[src, det, nrg]    = sum_{e in window(nrg)} RF[e, nrg]
//
// with the energy window and spectrum weights of find_src_nrg_range.cu and
// the attenuation model of integrate_diffraction.cu:291-296.  Outputs use the
// Nphotons layout, index src + det*SRC + nrg*SRC*DET.
//
// Lane = chord.  A block walks 8 views x 16 pixels with neighbouring pixels side
// by side -- their rays cross the same cells -- and then turns the line integrals
// round in shared memory, so that the stores of every detector bin, views fastest,
// are whole sectors: 71 us at the size below against 89 with 32 views side by side
// in both (12 of them in the walk, the rest from two bins' sums at a time and
// tables staged without a chain of loads).  Few chords are split among 2 to 32 lanes
// each (see the launch).  The chord's entry point and sample count are decided in
// float pairs, near a threshold in FP64 (which issues at 1/64 of the FP32 rate:
// all chords in FP64 took 16 us more), the chord is walked cell by cell
// (walk_cells), then the transmission of every source bin is formed once per
// chord -- each detector bin's window holds 2 DNRG + 1 of them -- and the windows
// are summed out of shared memory.  256x256 voxels, 180 views x
// 512 px, 64 energies: 71 us; with a warp per chord, one sample per lane, the set-up
// in FP64 by all 32 lanes alike and every window's exponentials on their own
// 660 us, and its line integrals were off by 1e-6 (positions in FP32).
#include <algorithm>

#include "scatter.cuh"

namespace xrdt {

namespace {

// Slab clipping of (sx,sy) -> (dx,dy) against [0,NX] x [0,NY]: the walk of the
// clipped chord, anchored at its entry point r (n = 0 when the segment misses
// the region).
__device__ void chord_setup(const DevProblem &P, double sx, double sy, double dx, double dy, WalkSetup *w, double *rx,
                            double *ry)
{
    const double ex = dsub(dx, sx), ey = dsub(dy, sy);
    double t0 = 0.0, t1 = 1.0;
    const double lo[2] = {0.0, 0.0}, hi[2] = {(double)P.nx, (double)P.ny};
    const double o[2] = {sx, sy}, d[2] = {ex, ey};
    for (int a = 0; a < 2; a++) {
        if (d[a] == 0.0) {
            if (o[a] < lo[a] || o[a] > hi[a]) t1 = -1.0;
            continue;
        }
        double ta = dsub(lo[a], o[a]) / d[a], tb = dsub(hi[a], o[a]) / d[a];
        if (ta > tb) {
            const double t = ta;
            ta = tb;
            tb = t;
        }
        if (ta > t0) t0 = ta;
        if (tb < t1) t1 = tb;
    }
    w->n = 0;
    w->dlt = w->ux = w->uy = ff{0.f, 0.f};
    *rx = *ry = 0.0;
    if (!(t1 > t0)) return;
    const double len = sqrt(dadd(dmul(ex, ex), dmul(ey, ey)));
    *rx = dadd(sx, dmul(t0, ex));
    *ry = dadd(sy, dmul(t0, ey));
    const double L = dmul(dsub(t1, t0), len);
    long long k = (long long)floor(L / P.DQ);
    while (dmul(P.DQ, (double)(k + 1)) <= L) k++;
    while (k >= 0 && !(dmul(P.DQ, (double)k) <= L)) k--;
    long long n = k + 1;
    if (n > P.kmax) n = P.kmax;
    const double inv = 1.0 / len;
    w->n = (int)n;
    w->ux = ff_from_double(ex * inv);
    w->uy = ff_from_double(ey * inv);
}

// The same in float pairs: false within 1e-9 of a threshold, 1e-8 of a step for the
// sample count, or within the pairs' error where that is more, and for rays along
// an axis.  Rounding moves a crossing along the chord by some 2^-44 of the distances
// over the chord's extent across the side, so by more the flatter it crosses it:
// where 256 voxels are left at 1e-3 of a voxel per length, by 2e-6 of a step, and on
// 1024 voxels, or from a source 5000 away, by 3e-5.
__device__ __forceinline__ bool chord_setup_pairs(const DevProblem &P, const F32Consts &C, ff sx, ff sy, ff dx, ff dy,
                                                  WalkSetup *w, ff *rx, ff *ry)
{
    const ff ex = ff_sub(dx, sx), ey = ff_sub(dy, sy);
    if (!(fabsf(ex.hi) > 1e-3f && fabsf(ey.hi) > 1e-3f)) return false;
    const ff ix = ff_rcp(ex), iy = ff_rcp(ey);
    // entry and exit of both slabs
    const ff x0 = ff_neg(ff_mul(sx, ix)), x1 = ff_mul(ff_fsub(C.nxf, sx), ix);
    const ff y0 = ff_neg(ff_mul(sy, iy)), y1 = ff_mul(ff_fsub(C.nyf, sy), iy);
    const ff tx0 = ex.hi > 0.f ? x0 : x1, tx1 = ex.hi > 0.f ? x1 : x0;
    const ff ty0 = ey.hi > 0.f ? y0 : y1, ty1 = ey.hi > 0.f ? y1 : y0;
    auto less = [](ff a, ff b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); };
    ff t0 = {0.f, 0.f}, t1 = {1.f, 0.f};
    if (less(t0, tx0)) t0 = tx0;
    if (less(t0, ty0)) t0 = ty0;
    if (less(tx1, t1)) t1 = tx1;
    if (less(ty1, t1)) t1 = ty1;
    const ff dt = ff_sub(t1, t0);
    const float err = 2.f * kUnitPairs * walk_extent(C, fabsf(sx.hi) + fabsf(ex.hi), fabsf(sy.hi) + fabsf(ey.hi)) *
                      fmaxf(fabsf(ix.hi), fabsf(iy.hi));
    if (!(fabsf(dt.hi) > fmaxf(1e-9f, err))) return false;
    w->n = 0;
    w->dlt = w->ux = w->uy = ff{0.f, 0.f};
    *rx = *ry = ff{0.f, 0.f};
    if (dt.hi < 0.f) return true;
    const ff len = ff_sqrt(ff_dot2(ex, ex, ey, ey));
    const ff t = ff_div(ff_mul(dt, len), ff{C.DQ, C.DQ_lo});
    if (!(t.hi < 4194304.f)) return false;
    float ft = floorf(t.hi);
    float fr = (t.hi - ft) + t.lo;
    if (fr < 0.f) {
        ft -= 1.f;
        fr = (t.hi - ft) + t.lo;
    }
    const float gt = fmaf(err, len.hi * C.inv_DQ, 1e-8f);
    if (!(fr > gt && fr < 1.f - fmaxf(gt, 1e-7f))) return false;
    long long n = (long long)ft + 1;
    if (n > P.kmax) n = P.kmax;
    const ff il = ff_rcp(len);
    w->n = (int)n;
    w->ux = ff_mul(ex, il);
    w->uy = ff_mul(ey, il);
    *rx = ff_add(sx, ff_mul(t0, ex));
    *ry = ff_add(sy, ff_mul(t0, ey));
    return true;
}

// FP64 out of line, for the chords that the pairs leave open.
__device__ __noinline__ void chord_setup_f64(const DevProblem &P, const SrcGeom *g, int det, WalkSetup *w, ff *rx,
                                             ff *ry)
{
    double Rdx, Rdy, Rdz, x, y;
    det_position(P, g->sphi, g->cphi, det, &Rdx, &Rdy, &Rdz);
    chord_setup(P, g->Rsrc_x, g->Rsrc_y, Rdx, Rdy, w, &x, &y);
    *rx = ff_from_double(x);
    *ry = ff_from_double(y);
}

constexpr int kCtWarps = 4;
constexpr int kCtMaxSmem = 200 * 1024;

// A detector's position per column pitch and a source's trigonometry as pairs.
struct CtConsts {
    ff cx, cy, r_det, pitch;
    int n_col;
};

// Views of a strip of chords: 8 floats of an output row are a 32-byte sector.
constexpr int kStrip = 8;

// Shared memory: per warp the transmission of a pass's source bins
// [e_pass][chords of the warp], then (STAGED) the spectrum windows [nrg_det][W],
// their sums and their first bins.  Windows too wide for that (!STAGED) are read
// through L1, and every bin forms its own transmissions.
template <bool STAGED, bool FINE>
__global__ void __launch_bounds__(32 * kCtWarps)
k_ct_sinogram(DevProblem P, F32Consts c, CtConsts q, const SrcGeom *__restrict__ sg, const float4 *__restrict__ cells,
              const FwdEnergy *__restrict__ energy, const float *__restrict__ rf_win, const int *__restrict__ win_lo,
              float *__restrict__ T, float *__restrict__ G0, int e_pass, int lg_split, int strip_w)
{
    extern __shared__ float att_s[];
    __shared__ float2 A_s[32 * kCtWarps];   // the block's line integrals
    const int lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    // 2^lg_split neighbouring lanes share a chord: its samples, source bins and detector bins
    const int split = 1 << lg_split, sub = lane & (split - 1), cols = 32 >> lg_split;
    const int nch = blockDim.x >> lg_split, ch = threadIdx.x >> lg_split;   // chords of the block, this thread's
    float *att = att_s + (size_t)(threadIdx.x >> 5) * cols * e_pass + (lane >> lg_split);   // this chord's column
    const int64_t npairs = (int64_t)P.n_src * P.n_det;
    const int W = 2 * P.dnrg + 1;
    const int64_t ncell = (int64_t)(P.nx + 1) * (P.ny + 1);
    float *rf_s = att_s + (size_t)nwarps * cols * e_pass, *g0_s = rf_s + P.nrg_det * W;
    int *lo_s = (int *)(g0_s + P.nrg_det);
    if (STAGED) {
        for (int i = threadIdx.x; i < P.nrg_det * W; i += blockDim.x) rf_s[i] = rf_win[i];
        for (int i = threadIdx.x; i < P.nrg_det; i += blockDim.x) lo_s[i] = win_lo[i];
        __syncthreads();
        for (int n = threadIdx.x; n < P.nrg_det; n += blockDim.x) {
            float g0 = 0.f;
            for (int j = 0; j < W; j++) g0 += rf_s[n * W + j];
            g0_s[n] = g0;
        }
    }
    // Blocks take the chords of a strip of strip_w views (the last may be
    // narrower) in the order of the outputs, views fastest, nch at a time.
    const int64_t full = ((int64_t)strip_w * P.n_det + nch - 1) / nch;   // blocks of a full strip
    const int strips = P.n_src / strip_w, rest = P.n_src - strips * strip_w;
    const int64_t nblocks = strips * full + ((int64_t)rest * P.n_det + nch - 1) / nch;
    for (int64_t blk = blockIdx.x; blk < nblocks; blk += gridDim.x) {
        const int strip = (int)min(blk / full, (int64_t)strips);
        const int width = strip < strips ? strip_w : rest;
        const int64_t first = (blk - strip * full) * nch;     // of the strip's chords
        const int count = (int)min((int64_t)nch, (int64_t)width * P.n_det - first);
        // ---- line integrals, in a strip of kStrip with neighbouring lanes on
        // neighbouring pixels of one view, whose rays cross the same cells (a
        // chord past the end repeats the last) ----
        {
            int k = ch;
            if (width == kStrip && nch >= 2 * kStrip) k = (ch % (nch / kStrip)) * kStrip + ch / (nch / kStrip);
            const int64_t s = first + min(k, count - 1);
            const int src = strip * strip_w + (int)(s % width), det = (int)(s / width);
            const SrcGeom *g = sg + src;
            // det_position in pairs: the column's offset is a multiple of 1/2
            const ff sphi = ff_from_double(g->sphi), cphi = ff_from_double(g->cphi);
            const ff rdet = ff_mulf(q.pitch, (float)(det % q.n_col) - 0.5f * (float)q.n_col + 0.5f);
            const ff dx = ff_add(ff_sub(q.cx, ff_mul(q.r_det, sphi)), ff_mul(rdet, cphi));
            const ff dy = ff_add(ff_add(q.cy, ff_mul(q.r_det, cphi)), ff_mul(rdet, sphi));
            WalkSetup ws;
            ff ax, ay;
            if (!chord_setup_pairs(P, c, ff_from_double(g->Rsrc_x), ff_from_double(g->Rsrc_y), dx, dy, &ws, &ax, &ay))
                chord_setup_f64(P, g, det, &ws, &ax, &ay);
            const int per = (ws.n + split - 1) >> lg_split;
            ws.n = min(ws.n, (sub + 1) * per);
            float2 A = walk_cells<true, FINE>(cells, 1, P.nx + 1, (unsigned)(ncell - 1), ws, ax.hi, ay.hi, c,
                                        make_float2(ax.lo, ay.lo), (float)(sub * per));
            for (int o = split >> 1; o > 0; o >>= 1) {
                A.x += __shfl_xor_sync(0xffffffffu, A.x, o);
                A.y += __shfl_xor_sync(0xffffffffu, A.y, o);
            }
            if (sub == 0) A_s[k] = A;
        }
        __syncthreads();
        // ---- energies: neighbouring lanes on neighbouring outputs ----
        const float2 A = A_s[ch];
        const bool mine = ch < count;
        const int64_t s = first + min(ch, count - 1);
        const int64_t p = strip * strip_w + s % width + s / width * P.n_src;
        auto transmission = [&](int e) {   // -log2(e)/f1, -log2(e)/f2 as pairs
            const float4 f = __ldg(reinterpret_cast<const float4 *>(energy + e));
            return ex2_approx(fmaf(A.x, f.x, fmaf(A.y, f.z, fmaf(A.x, f.y, A.y * f.w))));
        };
        auto store = [&](int n, float t, float g0) {
            if (mine) {
                const int64_t ray = p + (int64_t)n * npairs;
                T[ray] = t;
                G0[ray] = g0;
            }
        };
        if (STAGED) {
            // per pass the bins whose windows lie in its source bins (win_lo rises with n)
            for (int n = 0; n < P.nrg_det;) {
                const int e0 = lo_s[n];
                const int ne = min(e_pass, P.nrg_src - e0);
                __syncwarp();   // the windows of the pass before are done with their bins
#pragma unroll 4
                for (int e = sub; e < ne; e += split) att[cols * e] = transmission(e0 + e);
                __syncwarp();
                for (n += sub; n < P.nrg_det; n += split) {
                    const int lo = lo_s[n] - e0;
                    if (lo + W > ne) break;
                    const float *a = att + cols * lo, *rf = rf_s + n * W;
                    // two bins at a time, for their loads to overlap
                    const int m = n + split;
                    const int lo1 = m < P.nrg_det ? lo_s[m] - e0 : ne;
                    if (lo1 + W <= ne) {
                        const float *a1 = att + cols * lo1, *rf1 = rf_s + m * W;
                        float t = 0.f, t1 = 0.f;
#pragma unroll 4
                        for (int j = 0; j < W; j++) {
                            t = fmaf(rf[j], a[cols * j], t);
                            t1 = fmaf(rf1[j], a1[cols * j], t1);
                        }
                        store(n, t, g0_s[n]);
                        store(m, t1, g0_s[m]);
                        n = m;
                    } else {
                        float t = 0.f;
#pragma unroll 4
                        for (int j = 0; j < W; j++) t = fmaf(rf[j], a[cols * j], t);
                        store(n, t, g0_s[n]);
                    }
                }
                n = __reduce_min_sync(0xffffffffu, n);   // the first bin of the next pass
            }
        } else {
            for (int n = sub; n < P.nrg_det; n += split) {
                float t = 0.f, g0 = 0.f;
                for (int j = 0; j < W; j++) {
                    const float rf = __ldg(rf_win + n * W + j);
                    t = fmaf(rf, transmission(__ldg(win_lo + n) + j), t);
                    g0 += rf;
                }
                store(n, t, g0);
            }
        }
        __syncthreads();   // before the next chords' line integrals
    }
}

} // namespace

cudaError_t launch_ct_sinogram(const DevProblem &P, const SrcGeom *sg, const float4 *cells, const FwdEnergy *energy,
                               const float *rf_win, const int *win_lo, float *T, float *G0, cudaStream_t s,
                               int64_t *launches)
{
    const int64_t npairs = (int64_t)P.n_src * P.n_det;
    const int W = 2 * P.dnrg + 1;
    // lanes per chord: as many as 32 warps per SM have.  Kernel time at 1, 2, 4,
    // 8, 16, 32 lanes: 38400 chords (200x180 voxels, 64 bins) 62.4, 46.6, 38.4,
    // 40.5, 52.7, 75.3 us; 9600 (110x100, 32 bins) 42.1, 27.2, 22.0, 18.0, 17.2,
    // 21.9; 1000 (72x56, 48 bins) 44.6, 28.2, 20.0, 14.9, 11.8, 11.8; a warp's
    // serial walk and its serial bins are what the small ones wait for.
    int lg_split = 0;
    while (lg_split < 5 && (npairs << (lg_split + 1)) <= 1024LL * current_sm_count()) lg_split++;
    const size_t bin_bytes = sizeof(float) * (32 >> lg_split);
    // the source bins of a pass: all that the windows reach, or as many as one
    // warp's columns have room for beside the windows, one window at least
    const int E = P.e_hi - P.e_lo + 1;
    const size_t tables = sizeof(float) * ((size_t)P.nrg_det * W + 2 * P.nrg_det);
    int warps = kCtWarps;
    int64_t e_pass = E;
    size_t smem = bin_bytes * warps * E + tables;
    if (smem > 56 * 1024) {   // four blocks per SM
        warps = 1;
        e_pass = tables < kCtMaxSmem ? std::min<int64_t>(E, (int64_t)((kCtMaxSmem - tables) / bin_bytes)) : 0;
        smem = bin_bytes * (size_t)e_pass + tables;
    }
    const bool staged = e_pass >= W;
    if (!staged) {
        warps = kCtWarps;
        e_pass = 0;
        smem = 0;
    }
    const F32Consts c = make_f32_consts(P);
    auto *kernel = c.grain > 1.f ? (staged ? k_ct_sinogram<true, true> : k_ct_sinogram<false, true>)
                                 : (staged ? k_ct_sinogram<true, false> : k_ct_sinogram<false, false>);
    // (the limit of every size: one call must not lower it between another thread's setting and launch)
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCtMaxSmem);
    if (e != cudaSuccess) return e;
    const int64_t nch = (int64_t)(32 >> lg_split) * warps;
    // strips of kStrip views where a lane has a chord to itself (38400 chords,
    // four lanes each: 39 us either way; 9600, sixteen: 20 us in strips, 17 in rows)
    const int strip_w = lg_split == 0 && P.n_src >= kStrip ? kStrip : P.n_src;
    const int strips = P.n_src / strip_w, rest = P.n_src - strips * strip_w;
    int64_t blocks = strips * (((int64_t)strip_w * P.n_det + nch - 1) / nch) + ((int64_t)rest * P.n_det + nch - 1) / nch;
    if (blocks > 64LL * current_sm_count()) blocks = 64LL * current_sm_count();
    const CtConsts q = {ff_from_double(P.cx), ff_from_double(P.cy), ff_from_double(P.r_det), ff_from_double(P.col_pitch),
                        P.n_col};
    kernel<<<(int)blocks, 32 * warps, smem, s>>>(P, c, q, sg, cells, energy, rf_win, win_lo, T, G0,
                                                 (int)e_pass, lg_split, strip_w);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

} // namespace xrdt
