// k_fwd.cu -- factored forward projector (Nphotons, Cphotons).
//
// Same model as integrate_diffraction.cu:9-409, reorganised for the GPU:
//
//  * One block per (source, detector pixel) instead of one per
//    (source, pixel, detector energy bin).  Everything except the spectrum
//    weight RF = spectrum[e, nrg] and the Compton channel overlap depends on
//    the source energy e only (:266-356), so the block accumulates
//    T[e] = sum_v W(v,e) ... once per source bin and applies the banded
//    response afterwards: Nphotons[nrg] = sum_{e in window(nrg)} RF[e,nrg] T[e].
//    The reference evaluates each (voxel, e) pair once per detector bin whose
//    window holds e (11 times).
//  * Gaussian q-resolution sums (:299-308) run over the bins within 7.5 sigma
//    of the wavevector transfer only (each dropped term is below 7e-13 of the
//    peak); the reference sums every fine bin.
//  * The detector-side line integrals of the block's pair come from the table
//    that k_det_walk (k_walk.cu) writes for the current tile of pairs, one
//    float2 per voxel; the source-side ones from a per-(source, voxel) table
//    (k_prep.cu), since they do not depend on the detector pixel.
//  * The wavevector transfer is carried as a float pair (about 48 significant
//    bits) because the Gaussian at 3 sigma amplifies its relative error by
//    several hundred; the rest is FP32, with compensated or FP64 sums over
//    the tiles of voxels.
//
// Work split inside a block: tiles of up to 768 voxels.  First lane = voxel
// computes the scattering geometry of the tile and leaves 12 floats per
// voxel in shared memory.  Then the warps take runs of 32-voxel steps of one
// source energy, again with lane = voxel.  The lanes of a step share the
// energy -- its constants are loaded once per run -- and hold neighbouring
// voxels (tiles of 8 x 4, PrepBuffers::vox_order), so their Gaussian windows
// are about equally long: the window loop wastes few lanes.  Sums over voxels
// stay in the lane until the run ends.  Runs come off a counter, the widest
// windows first, because a window's length grows with the energy.
//
// The kernel is bound by instruction issue.  With lane = energy (an energy's
// constants loaded for every voxel, a voxel's constants shuffled, a window loop
// as long as the warp's longest window) 32 terms took about 390 instructions;
// here they take about 240, and k_fwd went from 12.5 to 7.1 ms on 128x128 voxels,
// 32 views x 128 px, 40 energies, from 314 to 135 ms on the reference's own sizes
// (100x100, 32 views x 1024 px, 64 energies, 768 fine bins), and from 674 to 319 ms
// on 256x256 voxels, 45 views x 512 px, 64 energies.  Two neighbouring energies per
// step, packed two to an instruction, took 18 % fewer instructions but no less
// time (7.0, 147 and 314 ms at best): a packed FMA holds its pipe for two cycles.
// Measured on the way, 128x128: equal contiguous shares instead of the counter 9.3
// (reference sizes 227) ms, the counter 9.6 (192) ms, and voxels in tiles instead
// of strips 8.2 (149) ms.
//
// Compton counts: per step each lane adds its two channel overlaps to its own
// column of the warp's cells [channel][32] (no conflicts, no atomics); at the
// end of a run the columns are added up.  N and C are deterministic.
#include <algorithm>

#include "scatter.cuh"

namespace xrdt {

namespace {

constexpr int kMaxWarps = 12;      // 384 threads, two blocks per SM at 80 registers
constexpr int kMaxSmem = 226 * 1024 - (int)sizeof(PairRec);   // dynamic, of a block by itself
constexpr int kMaxSteps = 24;      // 32-voxel steps per energy and tile: 768 voxels, 36 KB of records
constexpr unsigned kMagicBits = 0x4B400000u;   // 1.5 * 2^23: adding it rounds to an integer in the mantissa
constexpr float kMagic = 12582912.f;

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

// How a launch is cut: warps per block, 32-voxel steps per energy and tile,
// columns of the Compton cells, whether the tables sit in shared memory, the
// highest energies whose steps of a tile are one run, and the runs that those of
// each other energy are cut into.
struct FwdSplit {
    int warps, steps, columns, tables, whole, runs;
};

struct Layout {
    size_t rec, cells, en, offs, tc, tns, cacc, tn, rf, winlo, wn, ifine, s2, s1, total;
    int slots;     // rows of a warp's Compton cells
    int istride;   // floats per material row of the patterns
};

// Shared-memory layout; identical on host and device.
__host__ __device__ inline Layout fwd_layout(const DevProblem &P, int E, int SL, const FwdSplit &sp, int tab)
{
    Layout L;
    const int W = 2 * P.dnrg + 1;
    // a slot below and one above the real ones, which are flushed in groups of
    // eight (one by one when the cells have few columns)
    L.slots = sp.columns == 32 ? ((SL + 7) & ~7) + 2 : SL + 2;
    L.istride = (P.nqf + 3) & ~3;
    size_t o = 0;
    L.rec = o; o = align16(o + sizeof(float4) * 3 * 32 * (size_t)sp.steps);
    L.cells = o; o = align16(o + sizeof(float) * (size_t)sp.warps * L.slots * sp.columns);
    L.ifine = o; if (!tab) o = align16(o + sizeof(float) * (size_t)P.n_mat * L.istride);
    L.en = o; o = align16(o + sizeof(FwdEnergy) * E);
    L.cacc = o; o = align16(o + sizeof(double) * P.nrg_det);
    L.tn = o; o = align16(o + sizeof(double) * E);
    L.tns = o; o = align16(o + sizeof(float2) * (size_t)E * sp.runs);
    L.offs = o; o = align16(o + sizeof(float) * (size_t)E * (SL + 2));
    L.tc = o; o = align16(o + sizeof(float) * (size_t)E * sp.runs * SL);
    L.rf = o; o = align16(o + sizeof(float) * P.nrg_det * W);
    L.winlo = o; o = align16(o + sizeof(int) * P.nrg_det);
    L.wn = o; o = align16(o + sizeof(int) * E);
    L.s2 = o; if (sp.tables) o = align16(o + sizeof(float) * (size_t)P.nq * P.na);
    L.s1 = o; if (sp.tables && tab) o = align16(o + sizeof(float) * (size_t)P.nq * P.na);
    L.total = o;
    return L;
}

struct FwdArgs {
    DevProblem P;
    const PairRec *recs;       // [block] the blocks' pairs
    FwdTables T;
    const int *vox_xy, *vox_mat, *vox_na, *vox_order;
    const float *vox_a2;
    const float2 *atten_src;
    const unsigned char *s2u8;
    const unsigned char *s1u8;   // the table path: the coherent table
    const float *vox_ta;         // the table path, bilinear: the Compton column as a grid coordinate
    const float *Ifine;
    float *N, *C;
    long long p0;              // block b writes output column p0 + b
    long long n_cols;          // output columns: the list's length, or SRC*DET
    const float2 *walk;        // [block][nv] detector-side line integrals (k_walk.cu)
    int nv, E, sl;
    int tiles;                 // tiles of voxels
    int narrow;                // 1: the outgoing range meets at most two channels (dEs <= dEd)
    FwdSplit split;
    F32Consts c;
    float y0h, y0l;            // q_lo / dq + 1/2: the wavevector transfer in bins is w / dq - y0
    float c1b;                 // sigma^2 of the source bin width, over s^2, in bins^2
};

__device__ __forceinline__ float4 lds128(uint32_t a)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// Sums eight values over the warp: the sum of x[i] ends in the lanes with
// ((lane >> 4 & 1) | (lane >> 2 & 2) | (lane & 4)) == i.  Nine shuffles
// instead of forty.
__device__ __forceinline__ float sum8(const float *x, int lane)
{
    float y[4], z[2];
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float keep = b4 ? x[2 * i + 1] : x[2 * i], send = b4 ? x[2 * i] : x[2 * i + 1];
        y[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const float keep = b3 ? y[2 * i + 1] : y[2 * i], send = b3 ? y[2 * i] : y[2 * i + 1];
        z[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    float s = (b2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, b2 ? z[0] : z[1], 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// The records of the tile of voxels from t0 on, with every thread of the block.  Out
// of line, so that the registers and the schedule of the runs' loop do not
// follow from this one's: inlined, the reference's own sizes take 120.7 ms against 117.9
// and 256x256 348.9 against 346.0 (the geometry alone out of line 118.3 and 347.6).
template <int TAB>
__device__ __noinline__ void tile_records(const FwdArgs &args, const PairRec &pair, const float2 *walk, float4 *rec,
                                          int istride, int t0)
{
    const DevProblem &P = args.P;
    const F32Consts &c = args.c;
    const int nst = args.split.steps, nv = args.nv;
    // ---- lane = voxel: scattering geometry (integrate_diffraction.cu:192-255) ----
    for (int i = threadIdx.x; i < 32 * nst && t0 + (i & ~31) < nv; i += blockDim.x) {
        const int v = args.vox_order[min(t0 + i, nv - 1)];
        const bool in = t0 + i < nv;
        const int xy = args.vox_xy[v];
        const float vx = ((float)(xy & 0xffff) + 0.5f) * c.vox;
        const float vy = ((float)(xy >> 16) + 0.5f) * c.vox;
        const VoxGeom vg = vox_geom<false>(pair.G, vx, vy);
        const float a2v = args.vox_a2[v];
        // labels as at integrate_diffraction.cu:259-260: the detector-side
        // integral feeds Pin, the source-side one Pout; the coherent term
        // needs their sum only
        const float2 As = args.atten_src[(int64_t)pair.src * nv + v];
        const float2 Ad = walk[v];
        // factors formed once per voxel: the Compton weight gp a2 / 2 over
        // the source bin width (the 1/2 of Cf, :347), the Rayleigh weight
        // with 1/sqrt(2 pi) (table path: with a2), and sigma_geom / s^2.
        // A lane past the last voxel repeats it with weights of zero.
        const float gpa = in ? vg.gp * a2v * 0.5f * c.inv_dEs : 0.f;
        const float wr = in ? vg.Wg * (TAB ? a2v : c.rsqrt2pi) : 0.f;
        const float sgs2 = __fdividef(vg.sg.hi, vg.s.hi * vg.s.hi);
        float last;
        if (TAB == 2) last = args.vox_ta[v];
        else if (TAB == 1) last = __int_as_float(args.vox_na[v] * P.nq);
        else last = __int_as_float((args.vox_mat[v] * istride) | ((args.vox_na[v] * P.nq) << 16));
        rec[i] = make_float4(Ad.x + As.x, Ad.y + As.y, As.x, As.y);
        rec[32 * nst + i] = make_float4(vg.s.hi, vg.s.lo, vg.omc.hi, vg.omc.lo);
        rec[64 * nst + i] = make_float4(sgs2, gpa, wr, last);
    }
}

// TAB: 0 the coherent term from the materials' fine-q patterns
// (integrate_diffraction.cu:299-308); 1 from the coherent table S1 by nearest
// bin, 2 with both tables read bilinearly (the cross-section table path).
// FAST: the tables sit in shared memory, the cells have 32 columns and an
// outgoing range meets at most two channels; the general form costs 15
// instructions more per step.  COUNT: count the exp2 evaluations (profiling).
template <int TAB, bool FAST, bool COUNT>
__global__ void __launch_bounds__(32 * kMaxWarps, 2)
k_fwd(const __grid_constant__ FwdArgs args)
{
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ PairRec pair;   // the block's (source, pixel) constants
    __shared__ int next_run;
    const DevProblem &P = args.P;
    const F32Consts &c = args.c;
    const int E = args.E, SL = args.sl, W = 2 * P.dnrg + 1;
    const int nw = args.split.warps, nst = args.split.steps, ncol = args.split.columns;
    const int H = args.split.runs, whole = args.split.whole, run_len = (nst + H - 1) / H;
    const Layout L = fwd_layout(P, E, SL, args.split, TAB);
    float4 *rec = (float4 *)(sm + L.rec);          // [3][32 nst]
    const FwdEnergy *en = (const FwdEnergy *)(sm + L.en);
    float *offs = (float *)(sm + L.offs);          // [E][SL + 2] Esrc1(e) - Edet1(channel)
    float *TC = (float *)(sm + L.tc);              // [E][runs][SL] Compton sums of a tile, before RF
    float2 *TNs = (float2 *)(sm + L.tns);          // [E][runs] compensated coherent sums
    double *Cacc = (double *)(sm + L.cacc);        // [nrg_det]
    double *TN = (double *)(sm + L.tn);            // [E]
    float *rf = (float *)(sm + L.rf);
    int *winlo = (int *)(sm + L.winlo);
    int *wn = (int *)(sm + L.wn);                  // first detector bin whose window holds e
    const float *S2 = (const float *)(sm + L.s2);  // quantised tables as floats (no u8 conversion in the loop)
    const float *S1 = (const float *)(sm + L.s1);

    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nthr = 32 * nw;
    const int64_t colidx = args.p0 + blockIdx.x;   // output column of this block
    const int64_t ncols = args.n_cols;
    const float2 *walk = args.walk + (int64_t)blockIdx.x * args.nv;

    // ---- stage the tables ----
    {
        const float4 *e4 = (const float4 *)(args.T.fwd_energy + P.e_lo);
        float4 *d4 = (float4 *)(sm + L.en);
        for (int i = tid; i < E * (int)(sizeof(FwdEnergy) / 16); i += nthr) d4[i] = __ldg(e4 + i);
    }
    for (int i = tid; i < E; i += nthr) wn[i] = args.T.win_n[2 * (P.e_lo + i)];
    for (int i = tid; i < E * H; i += nthr) TNs[i] = make_float2(0.f, 0.f);
    for (int i = tid; i < P.nrg_det * W; i += nthr) rf[i] = args.T.rf_win[i];
    for (int i = tid; i < E * (SL + 2); i += nthr) offs[i] = args.T.offs_e[(int64_t)P.e_lo * (SL + 2) + i];
    for (int i = tid; i < nw * L.slots * ncol; i += nthr) ((float *)(sm + L.cells))[i] = 0.f;
    for (int i = tid; i < P.nrg_det; i += nthr) {
        winlo[i] = args.T.win_lo[i];
        Cacc[i] = 0.0;
    }
    if (!TAB) {
        // rows of a multiple of four bins, the pads zero
        float *Is = (float *)(sm + L.ifine);
        for (int i = tid; i < P.n_mat * L.istride; i += nthr) {
            const int mm = i / L.istride, j = i - mm * L.istride;
            Is[i] = j < P.nqf ? __ldg(args.Ifine + mm * P.nqf + j) : 0.f;
        }
    }
    if (args.split.tables) {
        for (int i = tid; i < P.nq * P.na; i += nthr) ((float *)(sm + L.s2))[i] = (float)args.s2u8[i];
        if (TAB)
            for (int i = tid; i < P.nq * P.na; i += nthr) ((float *)(sm + L.s1))[i] = (float)args.s1u8[i];
    }
    auto table2 = [&](int i) { return FAST || args.split.tables ? S2[i] : (float)__ldg(args.s2u8 + i); };
    auto table1 = [&](int i) { return FAST || args.split.tables ? S1[i] : (float)__ldg(args.s1u8 + i); };

    // the tables were written long before; the pair's record and walk are from here
    await_predecessor();
    allow_dependents();
    // ---- per-(source, pixel) geometry, integrate_diffraction.cu:81-128 (k_pair_table) ----
    for (int i = tid; i < (int)(sizeof(PairRec) / 4); i += nthr)
        reinterpret_cast<int *>(&pair)[i] = reinterpret_cast<const int *>(args.recs + blockIdx.x)[i];
    const float qmin_t = c.qmin_t, inv_dqt = c.inv_dqt;
    const float dEdf = c.dEd, dEsf = c.dEs, kn0 = c.kn0;
    const int jlast = (int)kMagicBits + P.nqf - 1;
    const uint32_t rec_a = (uint32_t)__cvta_generic_to_shared(rec);
    const uint32_t plane = 512u * (uint32_t)nst;     // bytes of one of the three planes of records
    // the pattern's address from a bin number in the magic number's mantissa
    const uint32_t ifine_a = (uint32_t)__cvta_generic_to_shared(sm + L.ifine) - (kMagicBits << 2);
    float *cell = (float *)(sm + L.cells) + (size_t)wid * L.slots * ncol;
    const int nv = args.nv;
    unsigned int nexp = 0;   // exp2 evaluations of this lane (profiling only)

    for (int tile = 0; tile < args.tiles; tile++) {
        const int t0 = tile * 32 * nst;
        __syncthreads();   // the tables are staged; the last tile's records are no longer read
        if (tid == 0) next_run = 0;
        tile_records<TAB>(args, pair, walk, rec, L.istride, t0);
        __syncthreads();
        const int steps = min(nst, (nv - t0 + 31) >> 5);   // steps of this tile

        // ---- lane = voxel: runs of 32-voxel steps of one energy ----
        // Warps take the runs from a counter, the highest energies, whose
        // windows are the widest, first.
        for (;;) {
            int item = 0;
            if (lane == 0) item = atomicAdd(&next_run, 1);
            item = __shfl_sync(0xffffffffu, item, 0);
            if (item >= whole + (E - whole) * H) break;
            const int part = max(item - whole, 0);   // 0 for an energy in one run
            const int el = E - 1 - min(item, whole) - part / H, row = el * H + part % H;
            const int s0 = part % H * run_len, s1 = item < whole ? steps : min(s0 + run_len, steps);
            const FwdEnergy q = en[el];
            const float *orow = offs + el * (SL + 2);
            float accN = 0.f;
            for (int st = s0; st < s1; st++) {
                const uint32_t ra = rec_a + 16u * (uint32_t)(32 * st + lane);
                const float4 r0 = lds128(ra), r1 = lds128(ra + plane), r2 = lds128(ra + 2 * plane);
                const float sh = r1.x, oh = r1.z;
                // ---- attenuation: exponents in units of log2, with 1/f1 and
                // 1/f2 as pairs: the exponent reaches tens at the lowest
                // energies, where FP32 constants alone would move the factor
                // by a few 1e-6
                const float PP = ex2_approx(fmaf(r0.x, q.f1, fmaf(r0.y, q.f2, fmaf(r0.x, q.f1l, r0.y * q.f2l))));
                if (COUNT) nexp += 1;
                if (TAB) {
                    // the coherent term from the table S1 (the reference's
                    // commented-out kernel, integrate_diffraction.cu:701-719):
                    // Pin Pout geom Rayleigh a2 S1[wvt bin, a-ratio bin] with
                    // wvt = ein sin(theta/2) on the tables' log2 axis
                    float s1v;
                    if (TAB == 1)
                        s1v = table1(coherent_bin(P, q.ein, sh, oh, r1.w, args.T.energy + P.e_lo + el, qmin_t,
                                                  inv_dqt, c.bin_guard) +
                                     __float_as_int(r2.w));
                    else
                        s1v = table_bilinear(table1, P.nq, P.na, (lg2_approx(q.ein * sh) - qmin_t) * c.inv_dqg, r2.w);
                    accN = fmaf(PP * r2.z, s1v, accN);
                } else {
                    // ---- Gaussian q sum, :284-308, in units of the fine bin ----
                    const float sig2 = fmaf(q.c2, r2.x, args.c1b * (sh * sh));
                    const float rs = rsqrt_approx(sig2);
                    const float half = (kSig * sig2) * rs;
                    const float pref = PP * r2.z * rs;
                    // the wavevector transfer w / dq as a pair (p, pl), and the
                    // bin nearest to it: w / dq - y0 = j + frac.  y0h has few
                    // bits, so y0h + j is exact and so is its difference from p.
                    const float p = q.wh * sh;
                    const float pl = fmaf(q.wh, sh, -p) + fmaf(q.wh, r1.y, q.wl * sh);
                    const float y = (p - args.y0h) + (pl - args.y0l);
                    const float tj = y + kMagic;
                    const float frac = (p - (args.y0h + (tj - kMagic))) + (pl - args.y0l);
                    // the window's first and last bin, rounded outwards to the
                    // nearest and the first down to a multiple of four (the
                    // extra bins are exact terms of the full sum or zero pads);
                    // bin numbers stay in the magic number's mantissa, where
                    // they are integers and floats at once
                    const int jb = max(__float_as_int((y - half) + kMagic) & ~3, (int)kMagicBits);
                    const int je = min(__float_as_int((y + half) + kMagic), jlast);
                    float2 acc = make_float2(0.f, 0.f);
                    if (jb <= je && pref != 0.f) {
                        // c (u - frac)^2 as a quadratic in u = j - j0: near the
                        // peak it is A alone, far out C u^2 dominates, so the
                        // exponent keeps its relative accuracy in two FMAs,
                        // two bins per instruction
                        const float cq = (-0.5f * kLog2e) * (rs * rs);
                        const float cf = cq * frac;
                        const float2 A2 = make_float2(cf * frac, cf * frac), B2 = make_float2(-2.f * cf, -2.f * cf);
                        const float2 C2 = make_float2(cq, cq);
                        const float u = __int_as_float(jb) - tj;
                        float2 U = make_float2(u, u + 1.f);
                        uint32_t a = ifine_a + 4u * (uint32_t)((__float_as_int(r2.w) & 0xffff) + jb);
                        const uint32_t end = a + 4u * (uint32_t)(je - jb);
                        if (COUNT) nexp += (unsigned)((je - jb + 4) & ~3);
                        for (; a <= end; a += 16) {
                            const float4 I = lds128(a);
                            const float2 g0 = __ffma2_rn(__ffma2_rn(C2, U, B2), U, A2);
                            U = __fadd2_rn(U, make_float2(2.f, 2.f));
                            const float2 g1 = __ffma2_rn(__ffma2_rn(C2, U, B2), U, A2);
                            U = __fadd2_rn(U, make_float2(2.f, 2.f));
                            acc = __ffma2_rn(make_float2(ex2_approx(g0.x), ex2_approx(g0.y)), make_float2(I.x, I.y), acc);
                            acc = __ffma2_rn(make_float2(ex2_approx(g1.x), ex2_approx(g1.y)), make_float2(I.z, I.w), acc);
                        }
                    }
                    // (outside: where sigma^2 is negative, of a detector of negative area, the
                    // window is empty and pref is NaN, as the sum then is)
                    accN = fmaf(pref, acc.x + acc.y, accN);
                }
                // ---- Compton, :318-356 ----
                // eratio without contraction: the table bin's check forms it the same way
                const float x = __fmul_rn(q.ein, oh);
                const float er = __fadd_rn(1.f, x);
                const float rer = rcp_approx(er);
                // slot of the channel that holds the lower end of the outgoing
                // range [E1, E2]/eratio: 0 is the channel below the window, the
                // real ones follow; a range outside the window is skipped (a
                // misjudgement at a channel edge moves below 1e-5 of the overlap)
                const float ts = fmaf(q.es, rer, q.cs) + kMagic;
                int slot = __float_as_int(ts) - (int)kMagicBits;
                const bool hit = FAST || args.narrow ? (unsigned)slot <= (unsigned)q.ns : slot <= q.ns;
                float base = 0.f;
                // overlaps are taken times eratio: the range starts at
                // U = (Esrc1 - Edet1) - Edet1 x above a channel's left edge, is
                // one source bin long, and a channel dEd eratio
                const float re = dEdf * er;
                if (hit) {
                    // Pc = exp(-(Xin + Xc)) with Xc the source-side exponent at
                    // the outgoing energy eout = ein / eratio, formed as the
                    // Rayleigh one plus the small Compton change, so that Pc
                    // keeps the accuracy of PP:
                    //   Asx (1/eout^3 - 1/ein^3) = Asx/ein^3 ((1 + x)^3 - 1)
                    //   Asy (1/KN(eout) - 1/KN(ein))
                    //     = Asy/KN(ein) x ((k1 + 2 k2) + x (k1 + k2)) / (eratio^2 KN(eout))
                    // with k1 = kn1 ein, k2 = kn2 ein^2
                    const float cube = x * fmaf(x, x + 3.f, 3.f);   // (1 + x)^3 - 1
                    const float num = x * fmaf(x, q.qe, q.pe);
                    const float D = fmaf(er, fmaf(kn0, er, q.k1), q.k2);
                    const float dX = fmaf(r0.z * q.f1, cube, (r0.w * q.f2) * num * rcp_approx(D));
                    const float Pc = PP * ex2_approx(dX);
                    if (COUNT) nexp += 1;
                    // the table's value: nearest bin, or bilinear in the table path
                    float s2v;
                    if (TAB == 2)
                        s2v = table_bilinear(table2, P.nq, P.na,
                                             (compton_log2(q.ein * sh, er) - qmin_t) * c.inv_dqg, r2.w);
                    else
                        s2v = table2(compton_bin(P, q.ein, er, sh, oh, r1.w, args.T.energy + P.e_lo + el, qmin_t,
                                                 inv_dqt, c.bin_guard) +
                                     (TAB ? __float_as_int(r2.w) : (int)((unsigned)__float_as_int(r2.w) >> 16)));
                    // twice Cf of :347 (gpa holds the 1/2): eratio^2 (eratio + 1/eratio - 1 + cos^2)
                    const float ct = 1.f - oh;
                    const float Cf2 = er * fmaf(er, fmaf(ct, ct, x), 1.f);
                    base = Pc * r2.y * Cf2 * s2v;
                    if (FAST) {
                        // at most two channels (dEs <= dEd)
                        const float U = fmaf(-fmaf(ts - kMagic, dEdf, q.edb), x, orow[slot]);
                        const float o0 = fmaxf(fminf(dEsf, re - U), 0.f);
                        float *cl = cell + 32 * slot + lane;
                        cl[0] = fmaf(base, o0, cl[0]);
                        cl[32] = fmaf(base, dEsf - o0, cl[32]);
                    }
                }
                if (!FAST) {
                    // any number of channels; lanes that share a column take turns
                    const int last = min(__float_as_int(fmaf(fmaf(dEsf, c.inv_dEd, q.es), rer, q.cs) + kMagic) -
                                             (int)kMagicBits, q.ns);
                    for (int g = 0; g < 32; g += ncol) {
                        if (hit && lane >= g && lane < g + ncol)
                            for (int n = max(slot, 1); n <= last; n++) {
                                const float U = fmaf(-fmaf((float)n, dEdf, q.edb), x, orow[n]);
                                const float ov = fminf(U + dEsf, re) - fmaxf(U, 0.f);
                                float *cl = cell + ncol * n + (lane - g);
                                if (ov > 0.f) *cl = fmaf(base, ov, *cl);
                            }
                        __syncwarp();
                    }
                }
            }
            // ---- the run's sums at this energy ----
            accN = warp_sum(accN);
            if (lane == 0) {
                float2 k = TNs[row];
                kahan_add(k.x, k.y, accN);
                TNs[row] = k;
            }
            __syncwarp();
            float *tc = TC + row * SL;
            if (FAST || ncol == 32) {
                const int which = (lane >> 4 & 1) | (lane >> 2 & 2) | (lane & 4);
                for (int n0 = 1; n0 <= q.ns; n0 += 8) {
                    float x8[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        x8[i] = cell[32 * (n0 + i) + lane];
                        cell[32 * (n0 + i) + lane] = 0.f;
                    }
                    const float s = sum8(x8, lane);
                    const int n = n0 + which;
                    if ((lane & 3) == 0 && n <= q.ns) tc[n - 1] = s;
                }
                // the slot above the window, which a range that starts in the
                // last one also reaches
                cell[32 * (q.ns + 1) + lane] = 0.f;
            } else {
                for (int n = 1; n <= q.ns; n++) {
                    const float s = warp_sum(lane < ncol ? cell[ncol * n + lane] : 0.f);
                    if (lane == 0) tc[n - 1] = s;
                    if (lane < ncol) cell[ncol * n + lane] = 0.f;
                }
            }
            __syncwarp();
        }
        __syncthreads();
        // detector bin n gathers the tile's Compton sums of the energies whose
        // windows hold it, weighted with RF[e, n]
        for (int n = tid; n < P.nrg_det; n += nthr) {
            float s = 0.f;
            for (int j = 0; j < W; j++) {
                const int el = winlo[n] + j - P.e_lo;
                float t = 0.f;
                for (int h = 0; h < (el >= E - whole ? 1 : H); h++) t += TC[(el * H + h) * SL + (n - wn[el])];
                s = fmaf(t, rf[n * W + j], s);
            }
            Cacc[n] += (double)s;
        }
    }

    if (COUNT) {
        unsigned long long w = nexp;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
        if (lane == 0) atomicAdd(args.T.work, w);
    }

    // ---- outputs: ray index src + det*SRC + nrg*SRC*DET (:404) ----
    __syncthreads();
    for (int el = tid; el < E; el += nthr) {
        double s = 0.0;
        for (int h = 0; h < H; h++) {
            const float2 k = TNs[el * H + h];
            s += (double)k.x - (double)k.y;
        }
        TN[el] = s;
    }
    __syncthreads();
    for (int n = tid; n < P.nrg_det; n += nthr) {
        const int64_t ray = colidx + (int64_t)n * ncols;
        double acc = 0.0;
        for (int j = 0; j < W; j++) acc += (double)rf[n * W + j] * TN[winlo[n] + j - P.e_lo];
        args.N[ray] = (float)acc;
        args.C[ray] = (float)Cacc[n];
    }
}

template <int TAB, bool FAST, bool COUNT>
cudaError_t launch_variant(const FwdArgs &a, int n_pairs, size_t smem, cudaStream_t s)
{
    auto *kernel = k_fwd<TAB, FAST, COUNT>;
    // (the limit of every size: one call must not lower it between another thread's setting and launch)
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    // early: the tables are staged while the walk ends
    return launch_after(kernel, n_pairs, 32 * a.split.warps, smem, s, true, a);
}

template <int TAB>
cudaError_t launch_tab(const FwdArgs &a, int n_pairs, size_t smem, cudaStream_t s)
{
    const bool fast = a.narrow && a.split.columns == 32 && a.split.tables;
    if (a.T.work) return fast ? launch_variant<TAB, true, true>(a, n_pairs, smem, s)
                              : launch_variant<TAB, false, true>(a, n_pairs, smem, s);
    return fast ? launch_variant<TAB, true, false>(a, n_pairs, smem, s)
                : launch_variant<TAB, false, false>(a, n_pairs, smem, s);
}

// The split of a launch.  Twelve warps and tiles of up to 768 voxels wherever
// two such blocks fit on an SM (113 KB each): long runs amortise an energy's
// constants and the flush of its Compton cells.  Many detector bins per
// window or large tables take fewer warps, then narrower cells, then the
// tables read through L1.
bool choose_split(const DevProblem &P, int E, int SL, int nv, int tab, FwdSplit *out, size_t *smem)
{
    // a voxel's pattern row and table column share a word of its record (the table
    // path reads no patterns)
    if ((int64_t)P.nq * P.na > 65536 || (!tab && (int64_t)P.n_mat * ((P.nqf + 3) & ~3) > 65536)) return false;
    const int chunks = std::max(1, (nv + 31) / 32);
    static const FwdSplit candidates[] = {
        {kMaxWarps, kMaxSteps, 32, 1, 0, 1}, {kMaxWarps, 18, 32, 1, 0, 1}, {kMaxWarps, 12, 32, 1, 0, 1},
        {8, 12, 32, 1, 0, 1},                {kMaxWarps, 12, 32, 1, 0, 1}, {8, 8, 32, 1, 0, 1},
        {4, 4, 32, 1, 0, 1},                 {2, 2, 32, 1, 0, 1},          {1, 1, 32, 1, 0, 1},
        {1, 1, 1, 1, 0, 1},                  {1, 1, 1, 0, 0, 1}};
    for (int i = 0; i < (int)(sizeof candidates / sizeof candidates[0]); i++) {
        FwdSplit sp = candidates[i];
        // tiles of about equal length
        const int tiles = (chunks + sp.steps - 1) / sp.steps;
        sp.steps = (chunks + tiles - 1) / tiles;
        // four runs or more per warp; where the energies by themselves give as
        // many, the lowest, one for two warps, in two runs each, for the warps to
        // end a tile together (reference sizes 138.8 -> 134.8 ms, 256x256 326.5 -> 318.2,
        // 128x128 7.09 -> 7.08; one per warp 136.0, 321.4; every energy in two 136.3, 335)
        sp.runs = std::min(sp.steps, std::max(1, (4 * sp.warps + E - 1) / E));
        if (sp.runs == 1 && sp.steps > 1 && sp.warps > 1) {
            sp.runs = 2;
            sp.whole = std::max(0, E - sp.warps / 2);
        }
        const size_t total = fwd_layout(P, E, SL, sp, tab).total;
        const size_t limit = i < 4 ? (113 - 1) * 1024 - sizeof(PairRec) : kMaxSmem;
        if (total <= limit) {
            *out = sp;
            *smem = total;
            return true;
        }
    }
    return false;
}

__global__ void k_gather_rays(const int64_t *__restrict__ idx, int64_t n, const float *__restrict__ Nc,
                              const float *__restrict__ Cc, const float *__restrict__ Ac, int mw,
                              float *__restrict__ N, float *__restrict__ C, float *__restrict__ A)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
        N[i] = Nc[idx[i]];
        C[i] = Cc[idx[i]];
    }
    if (A)
        for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n * mw; t += stride)
            A[t] = Ac[idx[t / mw] * mw + t % mw];
}

} // namespace

bool forward_fits(const DevProblem &P, int sl, int nv, int tab)
{
    FwdSplit sp;
    size_t smem;
    return choose_split(P, P.e_hi - P.e_lo + 1, sl, nv, tab, &sp, &smem);
}

cudaError_t launch_gather_rays(const int64_t *idx, int64_t n, const float *Nc, const float *Cc,
                               const float *Ac, int mw, float *N, float *C, float *A, cudaStream_t s,
                               int64_t *launches)
{
    if (n == 0) return cudaSuccess;
    k_gather_rays<<<1024, 256, 0, s>>>(idx, n, Nc, Cc, Ac, mw, N, C, A);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_fast_forward(const DevProblem &P, const PairRec *recs, const FwdTables &T,
                                const PrepBuffers &B, int nv, const float *Ifine, bool list,
                                long long n_list, long long p0, int n_pairs, const float2 *walk, float *N,
                                float *C, cudaStream_t s, int64_t *launches, int tab)
{
    if (!N || !C || !B.vox_order || tab < 0 || tab > 2 || (tab && !B.s1u8) || (tab == 2 && !B.vox_ta)) return cudaErrorInvalidValue;
    FwdArgs a;
    a.p0 = p0;
    a.n_cols = list ? n_list : (long long)P.n_src * P.n_det;
    a.walk = walk;
    a.P = P;
    a.recs = recs;
    a.T = T;
    a.vox_xy = B.vox_xy;
    a.vox_mat = B.vox_mat;
    a.vox_na = B.vox_na;
    a.vox_order = B.vox_order;
    a.vox_a2 = B.vox_a2;
    a.atten_src = B.atten_src;
    a.s2u8 = B.s2u8;
    a.s1u8 = B.s1u8;
    a.vox_ta = B.vox_ta;
    a.Ifine = Ifine;
    a.N = N;
    a.C = C;
    a.nv = nv;
    a.E = P.e_hi - P.e_lo + 1;
    a.sl = T.sl;
    a.c = make_f32_consts(P);
    a.narrow = P.dEs <= P.dEd * (1.0 + 1e-12) ? 1 : 0;
    // y0 with at most 22 significant bits over the grid's bins, and the rest
    const double y0 = P.q_lo / P.dq_fine + 0.5;
    const double grid = ldexp(1.0, (int)ceil(log2(fabs(y0) + (double)P.nqf + 1.0)) - 22);
    a.y0h = (float)(rint(y0 / grid) * grid);
    a.y0l = (float)(y0 - (double)a.y0h);
    a.c1b = (float)((2.0 / P.hbarc) * (2.0 / P.hbarc) * P.dEs * P.dEs / 12.0 / (P.dq_fine * P.dq_fine));
    size_t smem;
    if (!choose_split(P, a.E, a.sl, nv, tab, &a.split, &smem)) return cudaErrorInvalidConfiguration;
    a.tiles = ((nv + 31) / 32 + a.split.steps - 1) / a.split.steps;
    if (launches) (*launches)++;
    // empty phantom: the caller writes the zeros of integrate_diffraction.cu:364-409
    if (nv == 0) return cudaSuccess;
    if (tab == 1) return launch_tab<1>(a, n_pairs, smem, s);
    if (tab == 2) return launch_tab<2>(a, n_pairs, smem, s);
    return launch_tab<0>(a, n_pairs, smem, s);
}

} // namespace xrdt
