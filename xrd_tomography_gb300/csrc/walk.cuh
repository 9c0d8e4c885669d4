// walk.cuh -- the attenuation line integral (attenuator.cu:9-109) over the
// bilinear cell map.
//
// The integer decisions (which ROI edge is entered, how many samples the ray
// takes) are those of the reference, made in FP32 with guard bands, then in
// float pairs, then in FP64 (walk_decide).  walk_cells sums the samples, one
// lane per ray, cell by cell with closed-form sums over the samples inside
// each cell, with float-pair offsets from an anchor: the voxel for the
// projector's and the operators' walks, the entry point for the CT chords.
#pragma once

#include "xrdt_device.cuh"
#include "ff.cuh"

namespace xrdt {

constexpr float kEdgeEps = 0.00001f;   // GetIntersection's margin about an edge

struct WalkSetup {
    float Lx, Ly;   // along the ray, of any length
    int n;          // number of samples: k = 0 .. n-1
    int edge;       // ROI edge entered (GetIntersection's order: bottom, right,
                    // top, left), -1 when the segment misses the ROI
    // The same samples anchored at the voxel v, for walk_cells: sample k sits
    // at v + (dlt + (n-1-k) DQ) u with u the unit vector from the voxel back
    // to the entry point and dlt = Lr - (n-1) DQ the distance of the last
    // sample from the voxel, both as float pairs.
    ff dlt, ux, uy;
};

// GetIntersection + the sample count of attenuator.cu:19-52: every k in
// [0, kmax) with DQ*k <= Lr.  A segment that misses the ROI gives n = 0
// (the reference compares against a NaN length and takes no sample).
__device__ inline void walk_setup(const DevProblem &P, double ex, double ey, double vx, double vy,
                                  WalkSetup *w)
{
    double rx, ry;
    get_intersection(ex, ey, vx, vy, P.nx, P.ny, &rx, &ry, &w->edge);
    double Lx = vx - rx, Ly = vy - ry;
    const double L2 = dadd(dmul(Lx, Lx), dmul(Ly, Ly));
    const double Lr = sqrt(L2);
    const double rL = 1.0 / sqrt(L2);
    Lx *= rL;
    Ly *= rL;
    long long n = 0;
    if (Lr >= 0.0) {
        long long k = (long long)floor(Lr / P.DQ);
        while (dmul(P.DQ, (double)(k + 1)) <= Lr) k++;
        while (k >= 0 && !(dmul(P.DQ, (double)k) <= Lr)) k--;
        n = k + 1;
        if (n > P.kmax) n = P.kmax;
    }
    w->Lx = (float)Lx;
    w->Ly = (float)Ly;
    w->n = (int)n;
    if (n > 0) {
        w->dlt = ff_from_double(Lr - P.DQ * (double)(n - 1));
        w->ux = ff_from_double(-Lx);
        w->uy = ff_from_double(-Ly);
    } else {
        w->dlt = w->ux = w->uy = ff{0.f, 0.f};
    }
}

// The voxel-anchored form of a set-up whose edge and sample count are
// decided (walk_setup_f32), from the endpoint (ex, ey) as float pairs: with
// D = v - e, the entry point on edge x = X0 lies at Lr = |D| (vx - X0)/Dx
// from the voxel (y = Y0: |D| (vy - Y0)/Dy), and u = -D/|D|.
__device__ __forceinline__ void walk_anchor_ff(const F32Consts &C, ff ex, ff ey, float vx, float vy, WalkSetup *w)
{
    if (w->n <= 0) {
        w->dlt = w->ux = w->uy = ff{0.f, 0.f};
        return;
    }
    const ff Dx = ff_fsub(vx, ex), Dy = ff_fsub(vy, ey);
    const ff D = ff_sqrt(ff_dot2(Dx, Dx, Dy, Dy));
    const bool horizontal = w->edge == 0 || w->edge == 2;        // y = 0 or NY, else x = NX or 0
    const float far_edge = w->edge == 1 ? C.nxf : (w->edge == 2 ? C.nyf : 0.f);
    const ff ratio = ff_mulf(ff_rcp(horizontal ? Dy : Dx), (horizontal ? vy : vx) - far_edge);
    const ff Lr = ff_mul(D, ratio), iD = ff_rcp(D);
    w->dlt = ff_sub(Lr, ff_mulf(ff{(float)(w->n - 1), 0.f}, C.DQ));
    w->ux = ff_neg(ff_mul(Dx, iD));
    w->uy = ff_neg(ff_mul(Dy, iD));
}

// How far rounding may move the entry point, in voxels: `unit` times the size of
// the endpoint and of the region, and as much more as the edge's length times
// the other side over |den| -- a side over the ray's extent across the edge --
// says that the ray grazes the edge.  Of 10^7 rays per scanner (endpoints at 0.8
// to 10^5 sides, maps of 3 to 2048 voxels a side, SFU quotients an ulp off) no
// FP32 entry point was further off than 3.8 units of 2^-24; the pairs' is taken
// the same way.
constexpr float kUnitF32 = 6.f / 16777216.f, kUnitPairs = 1e-12f;

__device__ __forceinline__ float walk_extent(const F32Consts &C, float ex, float ey)
{
    return fmaf(0.25f, C.nxf + C.nyf, fabsf(ex) + fabsf(ey));
}

__device__ __forceinline__ float entry_error(const F32Consts &C, float extent_units, float inv_den)
{
    return extent_units * fmaf(0.5f * (C.nxf * C.nyf), fabsf(inv_den), 1.f);
}

// FP32 version of walk_setup for the endpoint (ex, ey) rounded to float.
// Returns false when a decision is too close to its threshold for FP32 to be
// trusted -- a nearly edge-parallel ray, a ray through an ROI corner, or a
// length within a few FP32 errors of a multiple of DQ (axis-aligned rays hit
// the latter exactly) -- and the caller then decides in float pairs or FP64
// (walk_decide).  The guards grow with the distances: rounding of the endpoint
// and of the products moves the entry point by a few 2^-24 of them, and further
// along an edge that the ray grazes (entry_error).  With fixed guards, set for
// endpoints some 300 voxels away, 0.25 % of the walks from a source 5000 voxels
// away took a sample too many or too few.
__device__ __forceinline__ bool walk_setup_f32(const DevProblem &P, const F32Consts &C, float ex, float ey,
                                               float vx, float vy, WalkSetup *w)
{
    const float NX = C.nxf, NY = C.nyf, inv_DQ = C.inv_DQ;
    const float eps = kEdgeEps;
    const float dx = vx - ex, dy = vy - ey;
    const float units = kUnitF32 * walk_extent(C, ex, ey);
    float err = 0.f;
    float rx = 0.f, ry = 0.f;
    bool found = false;
    int edge = -1;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float x3 = (i == 1 || i == 2) ? NX : 0.f;
        const float x4 = (i == 0 || i == 1) ? NX : 0.f;
        const float y3 = (i >= 2) ? NY : 0.f;
        const float y4 = (i == 1 || i == 2) ? NY : 0.f;
        const float x4_x3 = x4 - x3, y3_y1 = y3 - ey, y4_y3 = y4 - y3, x3_x1 = x3 - ex;
        const float den = x4_x3 * dy - dx * y4_y3;
        // edge-parallel within FP32 error: 1e-2, and where the side is long enough
        // for the rounding of its coordinates to reach a hundredth of |den|
        if (fabsf(den) < fmaxf(1e-2f, 4e-6f * (NX * NY))) return false;
        const float inv = __fdividef(1.f, den);
        err = entry_error(C, units, inv);
        const float G = fmaxf(2e-4f, err * C.inv_side);
        const float ua = (x4_x3 * y3_y1 - x3_x1 * y4_y3) * inv;
        if (fabsf(ua + eps) < G || fabsf(ua - (1.f + eps)) < G) return false;
        if (ua > -eps && ua < 1.f + eps) {
            const float ub = (dx * y3_y1 - x3_x1 * dy) * inv;
            if (fabsf(ub + eps) < G || fabsf(ub - (1.f + eps)) < G) return false;
            if (ub > -eps && ub < 1.f + eps) {
                rx = fmaf(dx, ua, ex);
                ry = fmaf(dy, ua, ey);
                found = true;
                edge = i;
                break;
            }
        }
    }
    if (!found) return false;
    const float Lx = vx - rx, Ly = vy - ry;
    const float t = sqrtf(fmaf(Lx, Lx, Ly * Ly)) * inv_DQ;
    float ft;
    const int it = floor_nc(t, &ft);
    const float fr = t - ft;
    const float gt = fmaf(4e-7f, t, fmaxf(1e-3f, err * inv_DQ));
    if (fr < gt || fr > 1.f - gt) return false;
    long long n = (long long)it + 1;
    if (n > P.kmax) n = P.kmax;
    w->Lx = dx;
    w->Ly = dy;
    w->n = (int)n;
    w->edge = edge;
    return true;
}

// The same decisions in float pairs, for the lanes that walk_setup_f32 leaves
// open: about 48 bits against its 24, in FP32 instructions.  Returns false
// within 1e-9 of a threshold (1e-8 of a step for the length), or within the
// pairs' error of some 2^-44 of the distances where that is more, and FP64 then
// has to round as the oracle does: rays along the grid, rays through a corner.
// FP64 issues at 1/64 of the FP32 rate, and the 0.7 % of the lanes that are
// open sit in one warp of five.  Straight to FP64 instead, the walk of 256x256
// voxels, 45 views x 512 px took 3 % longer, and the source side's, all of it in FP64
// before, 397 us against 206.
static __device__ __noinline__ bool walk_setup_pairs(const DevProblem &P, const F32Consts &C, ff ex, ff ey, float vx, float vy,
                                              WalkSetup *w)
{
    const float NX = C.nxf, NY = C.nyf;
    const ff eps = {kEdgeEps, 0.f};
    const float units = kUnitPairs * walk_extent(C, ex.hi, ey.hi);
    float err = 0.f;
    const ff dx = ff_fsub(vx, ex), dy = ff_fsub(vy, ey);
    if (!(fabsf(dx.hi) * NY > 1e-4f) || !(fabsf(dy.hi) * NX > 1e-4f)) return false;   // edge-parallel
    // how far inside [-eps, 1 + eps] a parameter lies (negative: outside)
    auto inside = [&](ff u) {
        const ff lo = ff_add(u, eps), hi = ff_add(ff_fsub(1.f, u), eps);
        return fminf(lo.hi, hi.hi);
    };
    const ff ex1 = ff_fsub(NX, ex), ey1 = ff_fsub(NY, ey);   // from the far edges
    int edge = -1;
    ff ua = {0.f, 0.f};
#pragma unroll 1
    for (int i = 0; i < 4; i++) {
        const bool horizontal = !(i & 1);                    // y = 0 or NY: bottom, (right), top, (left)
        const ff fx = i == 1 || i == 2 ? ex1 : ff_neg(ex);   // edge's first corner minus the endpoint
        const ff fy = i >= 2 ? ey1 : ff_neg(ey);
        ua = horizontal ? ff_div(fy, dy) : ff_div(fx, dx);
        err = entry_error(C, units, __fdividef(1.f, horizontal ? dy.hi * NX : dx.hi * NY));
        const float G = fmaxf(1e-9f, err * C.inv_side);
        const float in_a = inside(ua);
        if (fabsf(in_a) < G) return false;
        if (!(in_a > 0.f)) continue;
        // dx fy - fx dy over the edge's length times dy (or -dx)
        const ff cross = ff_sub(ff_mul(dx, fy), ff_mul(fx, dy));
        const ff den = horizontal ? ff_mulf(dy, i == 0 ? NX : -NX) : ff_mulf(dx, i == 1 ? -NY : NY);
        const float in_b = inside(ff_div(cross, den));
        if (fabsf(in_b) < G) return false;
        if (in_b > 0.f) {
            edge = i;
            break;
        }
    }
    if (edge < 0) return false;
    const ff D = ff_sqrt(ff_dot2(dx, dx, dy, dy));
    const ff Lr = ff_mul(D, ff_fsub(1.f, ua));
    const ff t = ff_div(Lr, ff{C.DQ, C.DQ_lo});
    if (!(t.hi > 0.f && t.hi < 4194304.f)) return false;
    // floor of the pair: of its high part, moved down when the low part crosses
    float ft = floorf(t.hi);
    float fr = (t.hi - ft) + t.lo;
    if (fr < 0.f) {
        ft -= 1.f;
        fr = (t.hi - ft) + t.lo;
    }
    const float gt = fmaf(err, C.inv_DQ, 1e-8f);
    if (fr < gt || fr > 1.f - fmaxf(gt, 1e-7f)) return false;
    long long n = (long long)ft + 1;
    if (n > P.kmax) n = P.kmax;
    w->n = (int)n;
    w->edge = edge;
    w->Lx = dx.hi;
    w->Ly = dy.hi;
    return true;
}

// In FP64, from the voxel's exact centre: (vx, vy) is that rounded to float, which
// for a side of more than eight bits is no multiple of half a side any more.
static __device__ __noinline__ void walk_setup_f64(const DevProblem &P, double ex, double ey, float vx, float vy,
                                            WalkSetup *w)
{
    walk_setup(P, ex, ey, (rint((double)vx / P.vox - 0.5) + 0.5) * P.vox,
               (rint((double)vy / P.vox - 0.5) + 0.5) * P.vox, w);
}

// A walk's decisions and its voxel-anchored form, from the endpoint as float
// pairs (and in double for the last resort).  Pairs decide for voxel centres that
// a float holds, as with a side of 1; for others FP64 does: a centre off by 1e-7
// of itself takes a sample too many or too few where a length is a multiple of DQ.
__device__ __forceinline__ void walk_decide(const DevProblem &P, const F32Consts &C, ff ex, ff ey,
                                            const double *exd, const double *eyd, float vx, float vy, WalkSetup *w)
{
    bool ok = walk_setup_f32(P, C, ex.hi, ey.hi, vx, vy, w);
    if (!ok && C.vox_exact) ok = walk_setup_pairs(P, C, ex, ey, vx, vy, w);
    if (ok) walk_anchor_ff(C, ex, ey, vx, vy, w);
    else walk_setup_f64(P, *exd, *eyd, vx, vy, w);
}

// Sum of the n samples times DQ, walked cell by cell by one lane.  Cell (ci,
// cj) holds the coefficients of the texels (ci-1..ci, cj-1..cj) of the
// zero-bordered map in the frame of the cell centre: f = c00 + c10 u + c01 v +
// c11 u v with u = x - ci and v = y - cj in [-0.5, 0.5] (k_prep.cu).  The
// bilinear patch of a cell is a polynomial in the sample index, so the samples j = 0 .. m-1 of
// a run inside one cell add up in closed form: with (u0, v0) the first
// sample's offset from the cell centre, S1 = m(m-1)/2 and
// S2 = (m-1)m(2m-1)/6,
//     sum u = m u0 + Lx S1,   sum v = m v0 + Ly S1,
//     sum uv = m u0 v0 + (u0 Ly + v0 Lx) S1 + Lx Ly S2,
//     sum f = m c00 + c10 sum u + c01 sum v + c11 sum uv.
// Each step takes the cell of its first sample (the nearest centre: rounding
// through the float mantissa, valid for |x| < 2^22) and
// the run up to the first sample beyond the cell's exit edge, at least one
// sample.  A sample within rounding of an edge may fall on either side; the
// interpolant is continuous there, so the sum changes only by rounding.  The
// runs are added with Kahan compensation.  One cell load serves the 3-4
// samples of a run (DQ = 1/4 voxel), or all of a uniform square's (below).  The
// samples are taken from the last (next to the voxel) to the first: rays that end on one voxel then start together and part slowly,
// so the lanes of a warp walking such rays read neighbouring cells.
// Cell (ci, cj) is cells[2 (ci sx + cj sy)]: sx = 1, sy = NX+1 for the
// row-major map, sx = NY+1, sy = 1 for the column-major copy.  Each step
// reads its 32-byte cell with one 256-bit load (sm_100 and later; cells are
// 32-byte aligned in a device allocation): the L1 cost of a warp-wide load
// follows the cache lines its lanes touch, so one load per cell instead of
// two halves it.  256x256 voxels, 45 views x 512 px: 63.8 ms against 65.3 for two
// 16-byte loads.
__device__ __forceinline__ void ld_cell256(const float4 *p, float4 &c0, float4 &c1)
{
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(c0.x), "=f"(c0.y), "=f"(c0.z), "=f"(c0.w), "=f"(c1.x), "=f"(c1.y), "=f"(c1.z), "=f"(c1.w)
        : "l"(p));
}

// The radius of the square of uniform cells (all four texels alike, in both
// maps) centred on a uniform cell, up to kReach - 1 cells: the map's samples are
// one constant there, so a run may reach across the whole square.  Such a
// cell's c11 is 0, and the cell carries 2 radius kReachUnit in the first one's
// place: below kReachLimit, where a coefficient counts as 0 (k_build_cells).
// Segmented phantoms are uniform but for their materials' borders, and rays
// cross them in about log2(size) steps per region instead of one per cell:
// 256x256 voxels, 45 views x 512 px 360 -> 64 ms, 128x128, 32 views x 128 px
// 6.6 -> 2.5 ms.  With noise on the materials 261 and 4.4 ms; on a map without a
// single uniform cell the wider test costs 2 % (367 and 6.7 ms).
constexpr int kReach = 31;
constexpr float kReachUnit = 0x1p-125f, kReachScale = 0x1p125f, kReachLimit = 0x1p-115f;

// LOW: the anchor is the pair (v, vlow), not an exact float, and the step a pair too:
// its rounding moves samples by up to 6e-8 of their way.  k0: the first sample to
// take.  FINE: a ray may have more than 2^24 samples, which a float counts in grains of
// two or more (C.grain): runs are whole grains long, so that k0 + m is exact and every
// run starts past the one before.  (A variant of its own: with the grain a constant of
// every walk, that of 128x128 voxels took 4 % longer.)
template <bool LOW, bool FINE>
__device__ __forceinline__ float2 walk_cells(const float4 *__restrict__ cells, int sx, int sy, unsigned ncell_m1,
                                             const WalkSetup &w, float vx, float vy, const F32Consts &C,
                                             float2 vlow = make_float2(0.f, 0.f), float k0 = 0.f)
{
    const float magic = 12582912.f, DQ = C.DQ;
    const float grain = FINE ? C.grain : 1.f, round = FINE ? C.grain_magic : magic;
    const float nf = (float)w.n;
    // samples from the voxel outwards: sample j at v + (dlt + j DQ) u
    const float2 L = make_float2(w.ux.hi * DQ, w.uy.hi * DQ);
    // minus the inverse steps, clamped so that a run is never overestimated
    const float ilx = fabsf(L.x) > 1e-4f ? -1.f / L.x : (L.x < 0.f ? 1e4f : -1e4f);
    const float ily = fabsf(L.y) > 1e-4f ? -1.f / L.y : (L.y < 0.f ? 1e4f : -1e4f);
    const float2 ninv = make_float2(ilx, ily);
    // exit edge offset h = +-0.5 (towards the step) times the inverse step
    const float2 hinv = make_float2(L.x < 0.f ? 0.5f * ilx : -0.5f * ilx, L.y < 0.f ? 0.5f * ily : -0.5f * ily);
    const float lxly = L.x * L.y;
    const float2 uhi = make_float2(w.ux.hi, w.uy.hi), ulo = make_float2(w.ux.lo, w.uy.lo);
    // LOW: whole voxels of the anchor and the rest, for the differences below to be
    // exact as they are for a voxel centre (from a float anchor the offset loses up
    // to 2e-5 voxel 250 cells on; line integrals of rough maps 512 a side 1e-6, not 6e-8)
    const float2 vt = make_float2(vx, vy), v2 = LOW ? make_float2(rintf(vx), rintf(vy)) : vt;
    if (LOW) vlow = make_float2((vx - v2.x) + vlow.x, (vy - v2.y) + vlow.y);
    // the distance of the voxel's nearest sample is below one step unless the
    // sample count was capped: then a two-sum that needs no ordering
    const bool small_dlt = w.dlt.hi <= DQ;
    float2 acc = make_float2(0.f, 0.f), comp = make_float2(0.f, 0.f);
    while (k0 < nf) {
        // distance s = dlt + k0 DQ and displacement t = s u as float pairs
        // (exact products through the FMA): the sample's offset from its cell
        // centre is then good to about 1e-7 voxel, where a position formed
        // at a magnitude of hundreds of voxels in FP32 would be off by 1e-5
        // and shift the interpolant by as much at material edges
        // (explicitly rounded operations, x and y packed in one instruction:
        // a contracted multiply-add would count a product's error twice)
        const float kq = __fmul_rn(k0, DQ);
        float kqe = fmaf(k0, DQ, -kq);
        if (LOW) kqe = fmaf(k0, C.DQ_lo, kqe);
        const float sh = __fadd_rn(w.dlt.hi, kq);
        float sl;
        if (small_dlt) {
            sl = __fadd_rn(__fsub_rn(w.dlt.hi, __fsub_rn(sh, kq)), __fadd_rn(kqe, w.dlt.lo));   // |kq| >= dlt
        } else {
            const float bb = __fsub_rn(sh, w.dlt.hi);
            sl = __fadd_rn(__fadd_rn(__fsub_rn(w.dlt.hi, __fsub_rn(sh, bb)), __fsub_rn(kq, bb)),
                           __fadd_rn(kqe, w.dlt.lo));
        }
        const float2 s2 = make_float2(sh, sh);
        const float2 p = __fmul2_rn(s2, uhi);
        float2 e = __fadd2_rn(__ffma2_rn(s2, uhi, make_float2(-p.x, -p.y)),
                              __ffma2_rn(s2, ulo, __fmul2_rn(make_float2(sl, sl), uhi)));
        if (LOW) e = __fadd2_rn(e, vlow);
        // the cell whose centre is nearest (any cell holding the point gives
        // the same value: the interpolant is continuous), then the offset
        const float2 t = __fadd2_rn(__fadd2_rn(vt, p), make_float2(magic, magic));
        const int ix = __float_as_int(t.x) - 0x4B400000, iy = __float_as_int(t.y) - 0x4B400000;
        const unsigned c = min((unsigned)(ix * sx + iy * sy), ncell_m1);
        float4 c0, c1;
        ld_cell256(cells + 2 * c, c0, c1);
        // the cell centre (exact) minus the anchor -- half or whole voxels --
        // is exact, and it cancels p but for the offset (Sterbenz), so only e rounds
        const float2 r = __fadd2_rn(t, make_float2(-magic, -magic));
        const float2 d = __fadd2_rn(__fadd2_rn(__fadd2_rn(v2, make_float2(-r.x, -r.y)), p), e);
        // steps to each exit edge of the cell, or of the uniform square around it
        const bool tiny = fabsf(c1.z) < kReachLimit;
        const float r2 = tiny ? c1.z * kReachScale : 0.f;
        if (tiny) c1.z = 0.f;
        const float2 s = __ffma2_rn(d, ninv, __ffma2_rn(make_float2(r2, r2), hinv, hinv));
        // ceil(s) as round(s + 1/2) through the float mantissa (either way at a tie)
        float m = __fadd_rn(__fadd_rn(__fadd_rn(fminf(s.x, s.y), 0.5f), round), -round);
        m = fminf(fmaxf(m, grain), nf - k0);
        const float S1 = 0.5f * __fmaf_rn(m, m, -m);
        const float S2 = S1 * __fmaf_rn(m, 2.f / 3.f, -1.f / 3.f);
        const float2 su = __ffma2_rn(d, make_float2(m, m), __fmul2_rn(L, make_float2(S1, S1)));
        float suv = __fmul_rn(__fmul_rn(d.x, d.y), m);
        suv = __fmaf_rn(__fmaf_rn(d.x, L.y, __fmul_rn(d.y, L.x)), S1, suv);
        suv = __fmaf_rn(lxly, S2, suv);
        float2 part = __fmul2_rn(make_float2(suv, suv), make_float2(c1.z, c1.w));
        part = __ffma2_rn(make_float2(su.y, su.y), make_float2(c1.x, c1.y), part);
        part = __ffma2_rn(make_float2(su.x, su.x), make_float2(c0.z, c0.w), part);
        part = __ffma2_rn(make_float2(m, m), make_float2(c0.x, c0.y), part);
        const float2 y = __fadd2_rn(part, make_float2(-comp.x, -comp.y));
        const float2 tt = __fadd2_rn(acc, y);
        comp = __fadd2_rn(__fadd2_rn(tt, make_float2(-acc.x, -acc.y)), make_float2(-y.x, -y.y));
        acc = tt;
        k0 += m;
    }
    return make_float2((acc.x - comp.x) * DQ, (acc.y - comp.y) * DQ);
}

} // namespace xrdt
