// k_matrix.cu -- the model matrix (Amatrix) of the forward projector.
//
//   Amatrix[k, m, ray] = sum_{v of material m} sum_{e in window(nrg)} RF[e,nrg]
//                        Pin Pout geom Rayleigh G(wvt(v,e) - q_k; sigma(v,e)) dq_k
//
// (integrate_diffraction.cu:311-315, 365).  As in k_fwd.cu a block takes a
// (source, pixel) pair and sums over its voxels per source energy first,
// T[e, m, k], then applies the banded spectrum weights.
//
// Tiles of up to 768 voxels: lane = voxel forms the scattering geometry; then a
// warp takes one energy at a time off a counter, so that T[e] has one writer.
// Per 32 voxels lane = voxel forms the Gaussian's factors, which go through the
// warp's shared memory four voxels side by side, and lane = coarse bin adds the
// terms of two voxels per packed instruction, 32 bins at a time, skipping the
// groups of 32 bins that none of the four windows (7.5 sigma) reaches.  Sums
// stay in registers while the material stays the same.
//
// Bound by instruction issue: about half of the bins evaluated lie beyond 7.5
// sigma of their own term, the two packed pair differences and products cost
// more than the exp2, and four voxels' window tests and materials nearly as much
// again.  64x64 voxels, 32 views x 128 px, 40 energies, 4 materials x 64 bins: 3.5
// ms, and 3.8 with the groups' range compared per group instead of a bit each;
// the projection (1.8 ms) included 5.8 ms; two voxels at a time instead of four
// (6.2 then) 8.0 ms; lane = energy with shared-memory float
// atomics per (energy, material, bin) -- compare-and-swap loops here -- 21.4 ms.
#include <algorithm>

#include "scatter.cuh"

namespace xrdt {

namespace {

constexpr int kMaxMatrixWarps = 24;
constexpr int kStaticSmem = 256;   // of a block, rounded up; 1 KB more is the system's
constexpr int kMaxSmem = 227 * 1024 - kStaticSmem;   // dynamic, of a block by itself
static_assert(sizeof(PairRec) + 16 <= kStaticSmem, "the static part of a block's shared memory");

// words of four voxels' terms: pref, w_hi, w_lo and the exponent's scale of each
// voxel, then the bin groups of the pass they reach (a bit each), their common
// material (-1: they differ) and the four materials; a stride of 20 words
// keeps the stores of lane = voxel free of bank conflicts
constexpr int kQuad = 20;

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// warps per block, 32-voxel steps per tile, energies per pass
struct MatrixSplit {
    int warps, steps, e_pass;
};

struct Layout {
    size_t rec, term, cq, rf, winlo, ta, total;
};

__host__ __device__ inline Layout matrix_layout(const DevProblem &P, const MatrixSplit &sp)
{
    Layout L;
    size_t o = 0;
    L.rec = o; o = align16(o + sizeof(float4) * 2 * 32 * (size_t)sp.steps);
    L.term = o; o = align16(o + sizeof(float) * kQuad * 8 * (size_t)sp.warps);
    L.cq = o; o = align16(o + sizeof(float4) * P.nwt);
    L.rf = o; o = align16(o + sizeof(float) * P.nrg_det * (2 * P.dnrg + 1));
    L.winlo = o; o = align16(o + sizeof(int) * P.nrg_det);
    L.ta = o; o = align16(o + sizeof(float) * (size_t)sp.e_pass * P.n_mat * P.nwt);
    L.total = o;
    return L;
}

struct MatrixArgs {
    DevProblem P;
    const PairRec *recs;       // [block] the blocks' pairs
    FwdTables T;
    const int *vox_xy, *vox_mat, *vox_order;
    const float2 *atten_src;
    float *A;
    long long p0, n_cols;      // block b writes output column p0 + b of n_cols
    const float2 *walk;        // [block][nv] detector-side line integrals (k_walk.cu)
    int nv, E, tiles;
    MatrixSplit split;
    F32Consts c;
};

// NG: groups of 32 coarse bins that a warp keeps in registers at a time.
// COUNT: count the exp2 evaluations (profiling).
template <int NG, bool COUNT>
__global__ void __launch_bounds__(32 * kMaxMatrixWarps, 1)
k_matrix(const MatrixArgs args)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ PairRec pair;
    __shared__ int next_e;
    const DevProblem &P = args.P;
    const F32Consts &c = args.c;
    const int E = args.E, W = 2 * P.dnrg + 1, K = P.nwt, MW = P.n_mat * K;
    const int nst = args.split.steps, nv = args.nv, nthr = 32 * args.split.warps;
    const Layout L = matrix_layout(P, args.split);
    float4 *rec = (float4 *)(sm + L.rec);      // [2][32 nst]
    float4 *cq = (float4 *)(sm + L.cq);
    float *rf = (float *)(sm + L.rf);
    int *winlo = (int *)(sm + L.winlo);
    float *TA = (float *)(sm + L.ta);          // [e_pass][n_mat][K]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    float *term = (float *)(sm + L.term) + 8 * kQuad * wid;   // this warp's terms
    const float2 *walk = args.walk + (int64_t)blockIdx.x * nv;
    const int64_t colidx = args.p0 + blockIdx.x;

    for (int i = tid; i < (int)(sizeof(PairRec) / 4); i += nthr)
        reinterpret_cast<int *>(&pair)[i] = reinterpret_cast<const int *>(args.recs + blockIdx.x)[i];
    for (int i = tid; i < K; i += nthr) cq[i] = args.T.coarse_q[i];
    for (int i = tid; i < P.nrg_det * W; i += nthr) rf[i] = args.T.rf_win[i];
    for (int i = tid; i < P.nrg_det; i += nthr) winlo[i] = args.T.win_lo[i];
    unsigned nexp = 0;   // exp2 evaluations of this lane (profiling only)

    for (int pe0 = 0; pe0 < E; pe0 += args.split.e_pass) {
        const int ne = min(args.split.e_pass, E - pe0);
        __syncthreads();   // the tables are staged; the last pass's sums are written out
        for (int i = tid; i < ne * MW; i += nthr) TA[i] = 0.f;
        for (int tile = 0; tile < args.tiles; tile++) {
            const int t0 = 32 * nst * tile;
            __syncthreads();   // the last tile's records are no longer read
            if (tid == 0) next_e = 0;
            // ---- lane = voxel: scattering geometry (integrate_diffraction.cu:192-255) ----
            for (int i = tid; i < 32 * nst && t0 + (i & ~31) < nv; i += nthr) {
                const int v = args.vox_order[min(t0 + i, nv - 1)];
                const int xy = args.vox_xy[v];
                const float vx = ((float)(xy & 0xffff) + 0.5f) * c.vox;
                const float vy = ((float)(xy >> 16) + 0.5f) * c.vox;
                // sigma through pairs: a row's small entries are Gaussian tails
                const VoxGeom vg = vox_geom<true>(pair.G, vx, vy);
                const float2 As = args.atten_src[(int64_t)pair.src * nv + v];
                const float2 Ad = walk[v];
                const float wr = t0 + i < nv ? vg.Wg * c.rsqrt2pi : 0.f;
                rec[i] = make_float4(Ad.x + As.x, Ad.y + As.y, ff_mul(vg.sg, ffl_rcp(vg.s2)).hi, wr);
                rec[32 * nst + i] = make_float4(vg.s.hi, vg.s.lo, __int_as_float(args.vox_mat[v]), 0.f);
            }
            __syncthreads();
            const int steps = min(nst, (nv - t0 + 31) >> 5);
            // ---- one energy per warp at a time ----
            for (;;) {
                int item = 0;
                if (lane == 0) item = atomicAdd(&next_e, 1);
                item = __shfl_sync(0xffffffffu, item, 0);
                if (item >= ne) break;
                const int el = ne - 1 - item, e = P.e_lo + pe0 + el;   // the widest windows first
                const FwdEnergy q = args.T.fwd_energy[e];
                const EnergyRow er = args.T.energy[e];
                float *ta = TA + (size_t)el * MW;
                for (int gb = 0; 32 * gb < K; gb += NG) {
                    float2 acc[NG];
                    float qh[NG], ql[NG];
#pragma unroll
                    for (int g = 0; g < NG; g++) {
                        const float4 b = cq[min(32 * (gb + g) + lane, K - 1)];
                        qh[g] = -b.x;
                        ql[g] = -b.y;
                        acc[g] = make_float2(0.f, 0.f);
                    }
                    int mat = -1;   // the material the sums belong to
                    auto flush = [&]() {
#pragma unroll
                        for (int g = 0; g < NG; g++) {
                            const int k = 32 * (gb + g) + lane;
                            if (k < K) ta[mat * K + k] += acc[g].x + acc[g].y;
                            acc[g] = make_float2(0.f, 0.f);
                        }
                    };
                    for (int st = 0; st < steps; st++) {
                        // lane = voxel: the Gaussian's factors
                        {
                            const float4 r0 = rec[32 * st + lane], r1 = rec[32 * (nst + st) + lane];
                            const float sh = r1.x;
                            const float PP =
                                ex2_approx(fmaf(r0.x, q.f1, fmaf(r0.y, q.f2, fmaf(r0.x, q.f1l, r0.y * q.f2l))));
                            const float w_p = er.wfac_hi * sh;
                            const float w_r = fmaf(er.wfac_hi, sh, -w_p) + fmaf(er.wfac_hi, r1.y, er.wfac_lo * sh);
                            const float w_hi = w_p + w_r, w_lo = w_r - (w_hi - w_p);
                            const float sig2 = fmaf(er.sig_c2, r0.z, er.sig_c1 * (sh * sh));
                            const float rs = rsqrt_approx(sig2);
                            const float pref = PP * r0.w * rs;
                            // bit g: the window reaches group gb + g
                            unsigned groups = 0;
                            if (pref != 0.f) {
                                int klo, khi;
                                coarse_window(w_hi, kSig * sig2 * rs, c.q_lo, c.qpar_a, c.qpar_b, K, &klo, &khi);
                                const int g0 = max((klo >> 5) - gb, 0), g1 = min((khi >> 5) - gb, NG - 1);
                                if (klo <= khi && g0 <= g1) groups = (2u << g1) - (1u << g0);
                            }
                            const float pr = groups ? pref : 0.f;
                            groups |= __shfl_xor_sync(0xffffffffu, groups, 1);
                            groups |= __shfl_xor_sync(0xffffffffu, groups, 2);
                            const int m0 = __float_as_int(r1.z), m1 = __shfl_xor_sync(0xffffffffu, m0, 1);
                            const int m01 = m0 | m1 << 16, m23 = __shfl_xor_sync(0xffffffffu, m01, 2);
                            __syncwarp();   // the last step's terms have been read
                            float *t = term + kQuad * (lane >> 2) + (lane & 3);
                            t[0] = pr;
                            t[4] = w_hi;
                            t[8] = w_lo;
                            t[12] = -0.5f * kLog2e * rs * rs;
                            if (!(lane & 3)) {
                                const bool same = m01 == m23 && m0 == m1;
                                *(int4 *)(t + 16) = make_int4((int)groups, same ? m0 : -1, m01, m23);
                            }
                            __syncwarp();
                        }
                        // lane = coarse bin: four voxels at a time
#pragma unroll 2
                        for (int v = 0; v < 8; v++) {
                            const float4 *t = (const float4 *)(term + kQuad * v);
                            const int4 info = *(const int4 *)(t + 4);
                            if (!info.x) continue;   // no window reaches these groups
                            const float4 pr = t[0], wh = t[1], wl = t[2], sc = t[3];
                            // the Gaussians of two voxels at a bin
                            auto gauss = [&](float2 h, float2 l, float2 c2, float b, float bl) {
                                const float2 d = __fadd2_rn(__fadd2_rn(h, make_float2(b, b)),
                                                            __fadd2_rn(l, make_float2(bl, bl)));
                                const float2 x = __fmul2_rn(__fmul2_rn(c2, d), d);
                                return make_float2(ex2_approx(x.x), ex2_approx(x.y));
                            };
                            if (info.y >= 0) {
                                if (info.y != mat) {
                                    if (mat >= 0) flush();
                                    mat = info.y;
                                }
#pragma unroll
                                for (int g = 0; g < NG; g++)
                                    if (info.x & 1 << g) {
                                        acc[g] = __ffma2_rn(make_float2(pr.x, pr.y),
                                                            gauss(make_float2(wh.x, wh.y), make_float2(wl.x, wl.y),
                                                                  make_float2(sc.x, sc.y), qh[g], ql[g]),
                                                            acc[g]);
                                        acc[g] = __ffma2_rn(make_float2(pr.z, pr.w),
                                                            gauss(make_float2(wh.z, wh.w), make_float2(wl.z, wl.w),
                                                                  make_float2(sc.z, sc.w), qh[g], ql[g]),
                                                            acc[g]);
                                        if (COUNT) nexp += 4;
                                    }
                            } else {
                                // a border between materials: straight into the sums
#pragma unroll
                                for (int g = 0; g < NG; g++) {
                                    const int k = 32 * (gb + g) + lane;
                                    if ((info.x & 1 << g) && k < K) {
                                        const float2 a = gauss(make_float2(wh.x, wh.y), make_float2(wl.x, wl.y),
                                                               make_float2(sc.x, sc.y), qh[g], ql[g]);
                                        const float2 b = gauss(make_float2(wh.z, wh.w), make_float2(wl.z, wl.w),
                                                               make_float2(sc.z, sc.w), qh[g], ql[g]);
                                        if (COUNT) nexp += 4;
                                        ta[(info.z & 0xffff) * K + k] += pr.x * a.x;
                                        ta[(int)((unsigned)info.z >> 16) * K + k] += pr.y * a.y;
                                        ta[(info.w & 0xffff) * K + k] += pr.z * b.x;
                                        ta[(int)((unsigned)info.w >> 16) * K + k] += pr.w * b.y;
                                    }
                                }
                            }
                        }
                    }
                    if (mat >= 0) flush();
                    __syncwarp();
                }
            }
        }
        __syncthreads();
        // Amatrix[k, m, src, det, nrg] = dq_k sum_{e in window(nrg)} RF[e,nrg] T[e,m,k]
        const int64_t colbase = colidx * MW;
        const int64_t nstride = (int64_t)MW * args.n_cols;
        for (int n = wid; n < P.nrg_det; n += args.split.warps) {
            const int j0 = max(0, pe0 - (winlo[n] - P.e_lo)), j1 = min(W, pe0 + ne - (winlo[n] - P.e_lo));
            if (pe0 > 0 && j0 >= j1) continue;   // nothing to add
            const float *t0 = TA + ((int64_t)(winlo[n] - P.e_lo) - pe0) * MW;
            float *dst = args.A + colbase + (int64_t)n * nstride;
            for (int i = lane, k = lane % K; i < MW; i += 32) {
                float acc = 0.f;
                for (int j = j0; j < j1; j++) acc = fmaf(rf[n * W + j], t0[(int64_t)j * MW + i], acc);
                acc *= cq[k].z;
                if (pe0 == 0) dst[i] = acc;
                else dst[i] += acc;
                k += 32;
                while (k >= K) k -= K;
            }
        }
    }
    await_predecessor();   // launched early it must not end before what came before
    if (COUNT) {
        unsigned long long w = nexp;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (lane == 0) atomicAdd(args.T.work, w);
    }
}

template <int NG>
cudaError_t launch_groups(const MatrixArgs &a, int n_pairs, size_t smem, cudaStream_t s)
{
    auto *kernel = a.T.work ? k_matrix<NG, true> : k_matrix<NG, false>;
    // (the limit of every size: one call must not lower it between another thread's setting and launch)
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    // early: it reads nothing of the projection's, so the two overlap
    return launch_after(kernel, n_pairs, 32 * a.split.warps, smem, s, true, a);
}

// Two blocks of 12 warps per SM, or three of 8 -- whichever leaves fewer warps
// without an energy in the last round of a tile (64x64 voxels, 40 energies: the
// projection with its matrix 5.8 against 6.0 ms) -- when the sums of every energy fit beside the tile; else
// one block with as many energies per pass as fit (a pass repeats the geometry
// and adds to the rows written before), with fewer warps and shorter tiles
// only when a single energy's sums leave no room.
bool choose_split(const DevProblem &P, int E, int nv, MatrixSplit *out, size_t *smem)
{
    const int chunks = std::max(1, (nv + 31) / 32);
    const size_t per_e = sizeof(float) * (size_t)P.n_mat * P.nwt;
    auto rounds = [&](int warps) { return (E + warps - 1) / warps * warps; };
    struct Shape {
        int warps, steps, blocks;
    };
    static const Shape shapes[] = {{8, 20, 3}, {12, 24, 2}, {12, 12, 2}, {8, 8, 3}, {24, 24, 1}, {8, 8, 1}, {1, 1, 1}};
    for (const Shape &h : shapes) {
        if (h.blocks == 3 && h.steps == 20 && rounds(8) > rounds(12)) continue;
        const int tiles = (chunks + h.steps - 1) / h.steps;
        MatrixSplit sp = {h.warps, (chunks + tiles - 1) / tiles, 0};
        const size_t limit = h.blocks == 1 ? kMaxSmem : (size_t)228 * 1024 / h.blocks - 1024 - kStaticSmem;
        const size_t base = matrix_layout(P, sp).total + 16;
        if (base + per_e > limit) continue;
        const int64_t fit = (int64_t)((limit - base) / per_e);
        if (h.blocks > 1 && fit < E) continue;
        // passes of about equal length
        const int passes = (int)((E + fit - 1) / fit);
        sp.e_pass = (E + passes - 1) / passes;
        *out = sp;
        *smem = matrix_layout(P, sp).total;
        return true;
    }
    return false;
}

} // namespace

bool matrix_fits(const DevProblem &P, int nv)
{
    MatrixSplit sp;
    size_t smem;
    return choose_split(P, P.e_hi - P.e_lo + 1, nv, &sp, &smem);
}

cudaError_t launch_matrix(const DevProblem &P, const PairRec *recs, const FwdTables &T, const PrepBuffers &B, int nv,
                          bool list, long long n_list, long long p0, int n_pairs, const float2 *walk, float *A,
                          cudaStream_t s, int64_t *launches)
{
    if (!A || !B.vox_order || nv <= 0) return cudaErrorInvalidValue;
    MatrixArgs a;
    a.P = P;
    a.recs = recs;
    a.T = T;
    a.vox_xy = B.vox_xy;
    a.vox_mat = B.vox_mat;
    a.vox_order = B.vox_order;
    a.atten_src = B.atten_src;
    a.A = A;
    a.p0 = p0;
    a.n_cols = list ? n_list : (long long)P.n_src * P.n_det;
    a.walk = walk;
    a.nv = nv;
    a.E = P.e_hi - P.e_lo + 1;
    a.c = make_f32_consts(P);
    size_t smem;
    if (!choose_split(P, a.E, nv, &a.split, &smem)) return cudaErrorInvalidConfiguration;
    a.tiles = ((nv + 31) / 32 + a.split.steps - 1) / a.split.steps;
    if (launches) (*launches)++;
    const int groups = (P.nwt + 31) / 32;
    if (groups <= 1) return launch_groups<1>(a, n_pairs, smem, s);
    if (groups <= 2) return launch_groups<2>(a, n_pairs, smem, s);
    if (groups <= 4) return launch_groups<4>(a, n_pairs, smem, s);
    return launch_groups<8>(a, n_pairs, smem, s);
}

} // namespace xrdt
