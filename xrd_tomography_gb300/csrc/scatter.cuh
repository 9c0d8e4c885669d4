// scatter.cuh -- per-(source, pixel) and per-voxel scattering geometry of
// integrate_diffraction.cu:81-255 in the form the FP32 kernels consume, and
// the SFU helpers they share (k_fwd.cu: materials; k_vox.cu: per-voxel
// coefficients).
//
// The wavevector transfer is carried as a float pair (about 48 significant
// bits) because the Gaussian q resolution at 3 sigma amplifies its relative
// error by several hundred; 1 - cos(theta) comes from the cross product, so
// small angles lose nothing to cancellation.  The rest is FP32.
#pragma once

#include "xrdt_device.cuh"
#include "ff.cuh"
#include "walk.cuh"

namespace xrdt {

// Per-(source, pixel) constants of the scattering geometry.
struct PairGeom {
    ff Rsx, Rsy, Rdx, Rdy;        // source and detector positions (in plane)
    ff Rdz;                       // detector height over the source
    ff DD;                        // square of the source -> detector distance
    ff mx, my;                    // the voxel's height over the source: az = ax mx + ay my
    ff hz;                        // Hvox = az hz
    float nsx, nsy, nsz, ndx, ndy, sphi, cphi;
    float tan_full, adet12, focal2_12;
    ff vox2_12;                   // vox^2 / 12
};

// Per-voxel results of the scattering geometry.
struct VoxGeom {
    ff s;        // sin(theta/2)
    ff s2;       // sin^2(theta/2)
    ff omc;      // 1 - cos(theta)
    ff sg;       // (sS2 + vV2 + dD2) / (|a|^2 |b|^2)
    float gp;    // geom_src2vox * geom_vox2det
    float Wg;    // gp * Rayleigh factor
    float cos2;  // cos^2(theta)
};

// A pair's constants with its detector position in double and its source,
// tabulated once per operator or forward call (k_pair_table, k_vox.cu).
struct PairRec {
    PairGeom G;
    double Rdx, Rdy;
    int src, pad;
};

namespace {

constexpr float kSig = 7.5f;            // Gaussian window, in sigma (tail below 7e-13)
// The adjoint's window: every term that FP32 can represent.  2^(c d^2) flushes
// to zero below 2^-126, i.e. beyond sqrt(2 * 126 / log2(e)) = 13.2 sigma, so
// summing out to 13.25 sigma gives exactly the dense sum.  A sensitivity
// made of far-tail terms only can still be comparable to the 1e-7 that MLEM
// adds to it (main.m:162), so the adjoint cannot drop them.
constexpr float kSigAdj = 13.25f;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ void kahan_add(float &s, float &c, float x)
{
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// SFU approximations with denormals flushed (no denormal fix-up code; the
// arguments here are far from the denormal range)
__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp_approx(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2_approx(float x)
{
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sqrt_approx(float x)
{
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

constexpr float kTwelfth_hi = (float)(1.0 / 12.0);
constexpr float kTwelfth_lo = (float)(1.0 / 12.0 - (double)kTwelfth_hi);
// 0.5 log2(e) as a float pair: the Gaussian exp(-d^2 / (2 sigma^2)) is
// evaluated as 2^(c d^2) with c = -0.5 log2(e) / sigma^2
constexpr double kHalfLog2e = 0.72134752044448170368;
constexpr float kHalfLog2e_hi = (float)kHalfLog2e;
constexpr float kHalfLog2e_lo = (float)(kHalfLog2e - (double)kHalfLog2e_hi);

// c = -0.5 log2(e) / sigma^2 as a float pair, from sigma^2 as a pair and its
// reciprocal to FP32.  The residual of the quotient is exact through the FMA
// to a bit or two.
__device__ __forceinline__ ff gauss_scale(ff sig2, float rcp)
{
    const float ch = -kHalfLog2e_hi * rcp;
    float r = fmaf(-ch, sig2.hi, -kHalfLog2e_hi);
    r = fmaf(-ch, sig2.lo, r) - kHalfLog2e_lo;
    return {ch, r * rcp};
}

// Compton table bin of integrate_diffraction.cu:331-337 decided in FP64, as
// the oracle decides it; used only when the FP32 value lies within its error of
// a bin edge.  Kept out of line so that the rare FP64 path is a real branch
// and not predicated into every iteration of the energy loop.
__device__ __noinline__ int compton_bin_f64(const DevProblem &P, double ein, float omc_hi, float omc_lo)
{
    const double omcd = (double)omc_hi + (double)omc_lo;
    const double sd = sqrt(fabs(omcd) / 2.0);
    const double erd = 1.0 + ein * omcd;
    const double wd = ein * sd;
    const double l2d = log2(wd * sqrt(erd + wd * wd) / erd);
    return floor_to_int((l2d - P.q_min) / P.dq_tab);
}

// log2(w sqrt(eratio + w^2) / eratio), the Compton table's wavevector axis
// (integrate_diffraction.cu:331-333), with w = ein sin(theta/2).
__device__ __forceinline__ float compton_log2(float w, float eratio)
{
    const float w2 = w * w;
    return fmaf(0.5f, lg2_approx(w2 * (eratio + w2)), lg2_approx(rcp_approx(eratio)));
}

// Compton table bin nq = floor((compton_log2 - q_min) / dq), clamped to
// [0, NQ) (integrate_diffraction.cu:331-337).  Decided in FP32 from the voxel's
// 1 - cos(theta) (pair (oh, ol)) and sin(theta/2) (hi part sh), by rounding
// through the float mantissa; near a bin edge, where the value lies bin_guard
// or more from the middle of its bin (make_f32_consts), it is decided again
// in FP64 with the energy row's ein.  eratio = 1 + ein oh without contraction.
__device__ __forceinline__ int compton_bin(const DevProblem &P, float ein, float eratio, float sh, float oh, float ol,
                                           const EnergyRow *row, float qmin_t, float inv_dqt, float bin_guard)
{
    const float h = (compton_log2(ein * sh, eratio) - qmin_t) * inv_dqt - 0.5f;
    const float t = h + 12582912.f;
    int nq = __float_as_int(t) - 0x4B400000;            // round(h) = floor(h + 1/2); clamped below
    if (!(fabsf(h - (t - 12582912.f)) < bin_guard))   // near a table edge
        nq = compton_bin_f64(P, row->ein, oh, ol);
    return max(0, min(nq, P.nq - 1));
}

// The cross-section table path (code the reference keeps commented out,
// integrate_diffraction.cu:701-719): the coherent table's wavevector bin
// nq = floor((log2(w) - q_min) / dq) with w = ein sin(theta/2), clamped to
// [0, NQ), decided as compton_bin: in FP32 from the hi part of sin(theta/2), near
// a bin edge again in FP64 from 1 - cos(theta) (pair (oh, ol)).
__device__ __noinline__ int coherent_bin_f64(const DevProblem &P, double ein, float omc_hi, float omc_lo)
{
    const double omcd = (double)omc_hi + (double)omc_lo;
    const double sd = sqrt(fabs(omcd) / 2.0);
    return floor_to_int((log2(ein * sd) - P.q_min) / P.dq_tab);
}

__device__ __forceinline__ int coherent_bin(const DevProblem &P, float ein, float sh, float oh, float ol,
                                            const EnergyRow *row, float qmin_t, float inv_dqt, float bin_guard)
{
    const float h = (lg2_approx(ein * sh) - qmin_t) * inv_dqt - 0.5f;
    const float t = h + 12582912.f;
    int nq = __float_as_int(t) - 0x4B400000;            // as in compton_bin
    if (!(fabsf(h - (t - 12582912.f)) < bin_guard)) nq = coherent_bin_f64(P, row->ein, oh, ol);
    return max(0, min(nq, P.nq - 1));
}

// Bilinear value of a table [nq, na] (S(q + a*nq) as a float) at
// grid coordinates (tq, ta): the grid points are the table's entries,
// q_min + i (q_max - q_min)/(NQ - 1) (XSection_builder.m:121-125); clamped to
// the table (a NaN coordinate reads the first row or column).
template <class Table>
__device__ __forceinline__ float table_bilinear(const Table &S, int nq, int na, float tq, float ta)
{
    tq = fminf(fmaxf(tq, 0.f), (float)(nq - 1));
    ta = fminf(fmaxf(ta, 0.f), (float)(na - 1));
    const int i = min((int)tq, nq - 2), j = min((int)ta, na - 2);
    const float f = tq - (float)i, g = ta - (float)j;
    const int r0 = i + j * nq, r1 = r0 + nq;
    const float s00 = S(r0), s01 = S(r1);
    const float lo = fmaf(f, S(r0 + 1) - s00, s00);
    const float hi = fmaf(f, S(r1 + 1) - s01, s01);
    return fmaf(g, hi - lo, lo);
}

// integrate_diffraction.cu:93-128 for source g and pixel det: the pair's
// constants and the detector position in double.
__device__ __forceinline__ void pair_geom(const DevProblem &P, const SrcGeom &g, int det, PairGeom *G,
                                          double *Rdet_x, double *Rdet_y)
{
    double Rdz;
    det_position(P, g.sphi, g.cphi, det, Rdet_x, Rdet_y, &Rdz);
    G->Rsx = ff_from_double(g.Rsrc_x);
    G->Rsy = ff_from_double(g.Rsrc_y);
    G->Rdx = ff_from_double(*Rdet_x);
    G->Rdy = ff_from_double(*Rdet_y);
    const double Dx = *Rdet_x - g.Rsrc_x, Dy = *Rdet_y - g.Rsrc_y;   // Rsrc_z = 0
    G->Rdz = ff_from_double(Rdz);
    G->DD = ff_from_double(Dx * Dx + Dy * Dy + Rdz * Rdz);
    const double nsx = -g.sphi * P.sta, nsy = g.cphi * P.sta, nsz = -P.cta;
    const double nsxy = sqrt(nsx * nsx + nsy * nsy);
    G->nsx = (float)nsx;
    G->nsy = (float)nsy;
    G->nsz = (float)nsz;
    // Rvox_z = -(a . nsrc_xy) tan(geomphi/2) / |nsrc_xy|, Hvox with tan(geomphi):
    // their ratio by the double angle, finite at a wedge angle of 0 too
    G->mx = ff_from_double(-nsx * P.tan_half / nsxy);
    G->my = ff_from_double(-nsy * P.tan_half / nsxy);
    G->hz = ff_from_double(-2.0 / (1.0 - P.tan_half * P.tan_half));
    G->ndx = (float)g.sphi;
    G->ndy = (float)(-g.cphi);
    G->sphi = (float)g.sphi;
    G->cphi = (float)g.cphi;
    G->tan_full = (float)P.tan_full;
    G->adet12 = (float)(P.geomAdet / 12.0);
    G->vox2_12 = ff_from_double(P.vox * P.vox / 12.0);
    G->focal2_12 = (float)(P.focal * P.focal / 12.0);
}

// integrate_diffraction.cu:196-255 for one voxel.  a = voxel - source and b =
// detector - voxel as float pairs; 1 - cos(theta) from the cross product,
// |a x b|^2 / (|a||b| (|a||b| + a.b)), which has no cancellation at small
// angles.  (Everything from a and b themselves: with D = a + b in b's place, three
// products less, the errors grow with |D|/|b| and its square, sin(theta/2) to 6e-11
// with the source 5000 voxels away and 2e-9 from 10^5 on.)  The blur vectors S = ((a x b) x a)/|a|^2,
// D' = ((a x b) x b)/|b|^2 and V = -(S + D') = u x (a x b), u = a/|a|^2 +
// b/|b|^2, are perpendicular to a, b and a x b in turn, so with c = a x b
//   |S|^2 = |c|^2/|a|^2,  |D'|^2 = |c|^2/|b|^2,  |V|^2 = |D|^2 |c|^2/(|a|^2 |b|^2)
// and of the pairs only the components along the source's, the detector's and the
// z axis are left to find.  (The z component is no small one where the detector sits
// high over the fan plane.)
// SIGMA_PAIR: the terms that make up most of sigma^2 as pairs (the per-voxel
// operator, whose adjoint sums deep Gaussian tails: a tail amplifies sigma^2's
// relative error by (q distance / sigma)^2 / 2, and FP32 leaves it about two
// ulps off); otherwise in FP32 (the material forward projector, whose counts
// are dominated by the Gaussians' cores).  About 550 and 350 instructions per
// voxel; component by component with correctly rounded quotients and roots
// they were 2700 and 700, a third of the operator's forward and a tenth of
// the projector.
template <bool SIGMA_PAIR>
__device__ __forceinline__ VoxGeom vox_geom(const PairGeom &G, float vx, float vy)
{
    const ff ax = ff_fsub(vx, G.Rsx), ay = ff_fsub(vy, G.Rsy);
    const ff az = ffl_dot2(ax, G.mx, ay, G.my);
    const ff bx = ff_neg(ff_fsub(vx, G.Rdx)), by = ff_neg(ff_fsub(vy, G.Rdy)), bz = ff_sub(G.Rdz, az);
    // (tight where terms cancel: these high parts are used as floats, too)
    const ff an = ffl_dot3(ax, ax, ay, ay, az, az);
    const ff bn = ff_tight(ffl_dot3(bx, bx, by, by, bz, bz));
    const ff ab = ffl_dot3(ax, bx, ay, by, az, bz);
    const ff cx = ff_dot2(ay, bz, ff_neg(az), by);
    const ff cy = ff_dot2(az, bx, ff_neg(ax), bz);
    const ff cz = ff_dot2(ax, by, ff_neg(ay), bx);
    const ff cn = ffl_dot3(cx, cx, cy, cy, cz, cz);
    const ff nab = ffl_sqrt(ffl_mul(an, bn));
    VoxGeom r;
    if (ab.hi > 0.f) r.omc = ff_tight(ffl_mul(cn, ffl_rcp(ffl_mul(nab, ffl_add(nab, ab)))));
    else r.omc = ff_fsub(1.f, ffl_mul(ab, ffl_rcp(nab)));
    r.s2 = ff{0.5f * r.omc.hi, 0.5f * r.omc.lo};
    r.s = ff_sqrt(r.s2);
    const float costh = 1.f - r.omc.hi;
    r.cos2 = costh * costh;
    // FP32 remainder of the geometry
    const float Ax = ax.hi, Ay = ay.hi, Az = az.hi, Cx = cx.hi, Cy = cy.hi, Cz = cz.hi;
    const float Bx = bx.hi, By = by.hi;
    const ff ian = ff_rcp(an), ibn = ff_rcp(bn);
    const float ia = ian.hi, ib = ibn.hi;
    const float Sn = ((Cy * Az - Cz * Ay) * G.nsx + (Cz * Ax - Cx * Az) * G.nsy + (Cx * Ay - Cy * Ax) * G.nsz) * ia;
    const float sS2 = (cn.hi * ia - Sn * Sn) * G.focal2_12;
    if (!SIGMA_PAIR) {
        // (V by components: |V|^2 - Vz^2 would cancel where V points along z)
        const float Bz = bz.hi, H = Az * G.hz.hi;
        const float ux = fmaf(Ax, ia, Bx * ib), uy = fmaf(Ay, ia, By * ib), uz = fmaf(Az, ia, Bz * ib);
        const float Vx = uy * Cz - uz * Cy, Vy = uz * Cx - ux * Cz, Vz = ux * Cy - uy * Cx;
        const float Dn = ((Cy * Bz - Cz * By) * G.ndx + (Cz * Bx - Cx * Bz) * G.ndy) * ib;
        const float rest = fmaf((H * H) * (1.f / 12.f), Vz * Vz, sS2);
        r.sg = ff{fmaf(fmaf(Vx, Vx, Vy * Vy), G.vox2_12.hi, fmaf(fmaf(cn.hi, ib, -Dn * Dn), G.adet12, rest)) * ia * ib, 0.f};
    } else {
        const ff cb = ffl_mul(cn, ibn);
        const ff VV = ffl_mul(G.DD, ffl_mul(cb, ian));
        // Vz of V = u x c
        const ff ux = ffl_dot2(ax, ian, bx, ibn), uy = ffl_dot2(ay, ian, by, ibn);
        const ff Vz = ffl_dot2(ux, cy, ff_neg(uy), cx);
        const ff Vz2 = ffl_mul(Vz, Vz);
        // D'.n_det = ((a.b) (b.n) - (a.n) |b|^2)/|b|^2
        const ff adn = ffl_dot2(ax, ff{G.ndx, 0.f}, ay, ff{G.ndy, 0.f});
        const ff bdn = ffl_dot2(bx, ff{G.ndx, 0.f}, by, ff{G.ndy, 0.f});
        const ff Dn = ffl_sub(ffl_mul(ffl_mul(ab, ibn), bdn), adn);
        const ff dD = ffl_sub(cb, ffl_mul(Dn, Dn));
        const ff H = ffl_mul(az, G.hz);
        const ff blur = ffl_add(ffl_dot3(ffl_sub(VV, Vz2), G.vox2_12, ffl_mul(Vz2, ffl_mul(H, H)),
                                         ff{kTwelfth_hi, kTwelfth_lo}, dD, ff{G.adet12, 0.f}),
                                ff{sS2, 0.f});
        r.sg = ffl_mul(ffl_mul(blur, ian), ibn);
    }
    // geom_src2vox geom_vox2det = (a.n_src,xy / |a_xy|) (b.n_det) tan / (|a| |b|^3);
    // the roots and quotients with a correction step: the adjoint's column
    // sums inherit any bias of these factors, and MLEM amplifies it tenfold
    const float Rdotn = -G.sphi * Ax + G.cphi * Ay;
    const float axy2 = fmaf(Ax, Ax, Ay * Ay);
    float rxy = rsqrt_approx(axy2);
    rxy = fmaf(0.5f * rxy, fmaf(-axy2 * rxy, rxy, 1.f), rxy);
    const float inab = ff_rcp(nab).hi;   // (tight: rounded once)
    r.gp = (Rdotn * rxy) * (-(G.ndx * Bx + G.ndy * By) * ib) * inab * G.tan_full;
    r.Wg = r.gp * ((1.f + r.cos2) * 0.5f);
    return r;
}

// Coarse q bins that can lie within `half` of w: invert the bin edges
// edge(n) = q_lo + b n + a n^2 of wvt_value.cu:8-22 at w - half and w + half,
// widened by one bin on each side against rounding.  Returns the full range
// when the parabola has no real inverse there.
__device__ __forceinline__ void coarse_window(float w, float half, float q_lo, float qa, float qb, int nwt,
                                              int *klo, int *khi)
{
    int lo = 0, hi = nwt - 1;
    const float ua = w - half - q_lo, ub = w + half - q_lo;
    const float da = fmaf(4.f * qa, ua, qb * qb), db = fmaf(4.f * qa, ub, qb * qb);
    if (da >= 0.f && db >= 0.f) {
        // approximate root and quotient: the bin window is widened by one bin
        // on each side anyway
        const float na_ = __fdividef(2.f * ua, qb + sqrt_approx(da));
        const float nb_ = __fdividef(2.f * ub, qb + sqrt_approx(db));
        lo = max(lo, floor_nc(na_) - 1);
        hi = min(hi, floor_nc(nb_) + 1);
    }
    *klo = lo;
    *khi = hi;
}

} // namespace

} // namespace xrdt
