// k_walk.cu -- detector-side line integrals of a tile of (source, pixel)
// pairs: tab[item * nv + v] = attenuator(Rdet, Rvox) of
// integrate_diffraction.cu:259 (attenuator.cu:9-109), for every non-empty
// voxel v.
//
// The forward projector needs one such walk per (pair, voxel).  Walked inside
// the projector they share its registers and occupancy with the energy loop;
// here a separate kernel walks them and the projector reads the results as
// one coalesced float2 per voxel.
//
// Sampled one point per lane, the walk is bound by L1 wavefronts: a
// warp-wide 16-byte load costs at least four, and every sample needs a
// 32-byte cell.  Here each lane walks a whole ray cell by cell (walk_cells,
// walk.cuh), one cell load per run of 3-4 samples or per uniform square.  A warp takes 32 rays
// that end on 32 neighbouring pixels of one view and leave from the same
// voxel, so its lanes take about the same number of steps and stay within a
// few voxels of each other, side by side across the rays.  The warp reads
// the copy of the cell map (row- or column-major) whose rows run across its
// rays, so that neighbouring lanes mostly share cache lines.  Per voxel each
// lane sets up its own ray (in FP32, near a threshold in float pairs or FP64,
// walk_decide) and stores its float2; the stores of consecutive voxels of a row merge in L2.
#include <algorithm>

#include "scatter.cuh"

namespace xrdt {

namespace {

constexpr int kWalkThreads = 128;
constexpr int kWalkWarps = kWalkThreads / 32;
// Voxels per warp item (a strip): up to 64, so that the ray's FP64 endpoint is
// set up seldom, but no more than leaves kItemsPerSM items per SM.  A warp
// walks its strip's voxels one after the other; with 64 always, a small
// problem ran as a few warps: 45x33 voxels, 10 views x 75 px (240 warps) took
// 649 us against 82 now, 12x12, 4 views x 8 px (8 warps) 462 us against 20, and
// the last wave of 128x128, 32 views x 128 px showed too (7.8 against 6.65 ms).
// The smallest strips still pay: one voxel's walk outweighs the set-up.
constexpr int kMaxStrip = 64;
constexpr int kItemsPerSM = 256;   // 8 times the resident warps

// Row of ray r of group g of `rays` rays.  Linear pairs: the tile holds whole
// pixels (nd of them) of every view, row pixel * SRC + view; group g is view
// g % SRC and pixels rays (g / SRC) + r.  A list: entries rays g + r.
__device__ __forceinline__ bool group_row(const DevProblem &P, int list, long long n_items, int nd, int rays,
                                          long long g, int r, long long *row)
{
    if (list) {
        *row = g * rays + r;
        return *row < n_items;
    }
    const int s = (int)(g % P.n_src);
    const int dl = (int)(g / P.n_src) * rays + r;
    *row = (long long)dl * P.n_src + s;
    return dl < nd;
}

// 8 blocks (32 warps) per SM: the walk waits on L1 latency, and at 64
// registers (28 bytes spilled around the fallback calls) it takes 63.8 ms on
// 256x256 voxels, 45 views x 512 px against 68.7 at 6 blocks and 80 registers, 2.54
// against 2.72 on 128x128, 32 views x 128 px.
template <bool FINE>
__global__ void __launch_bounds__(kWalkThreads, 8)
k_det_walk(DevProblem P, F32Consts c, const PairRec *__restrict__ recs, int list,
           long long n_items, int nd, long long n_groups, int strip_len, const int *__restrict__ vox_xy, int nv,
           const float4 *__restrict__ cells, float2 *__restrict__ tab, int lg_split)
{
    const int lane = threadIdx.x & 31;
    // 2^lg_split neighbouring lanes share a ray's samples
    const int split = 1 << lg_split, sub = lane & (split - 1);
    await_predecessor();
    allow_dependents();   // (not before: the next kernel may then take every earlier result as written)
    const int64_t ncell = (int64_t)(P.nx + 1) * (P.ny + 1);
    const unsigned ncell_m1 = (unsigned)(ncell - 1);
    const float4 *cells_t = cells + 2 * ncell;   // column-major copy
    const int nstrips = (nv + strip_len - 1) / strip_len;
    const long long nwork = n_groups * nstrips;
    const long long wstride = (long long)gridDim.x * kWalkWarps;
    for (long long wk = (long long)blockIdx.x * kWalkWarps + (threadIdx.x >> 5); wk < nwork; wk += wstride) {
        const long long g = wk / nstrips;
        const int strip = (int)(wk - g * nstrips);
        long long row = -1;
        const bool valid = group_row(P, list, n_items, nd, 32 >> lg_split, g, lane >> lg_split, &row);
        // the pixel's position, tabulated per pair, as float pairs (and as
        // double for the rare FP64 set-up)
        const PairRec *rec = recs + (valid ? row : 0);
        const ff exff = rec->G.Rdx, eyff = rec->G.Rdy;
        float2 *out = tab + (valid ? row : 0) * nv;
        const int v1 = min(nv, (strip + 1) * strip_len);
        for (int v = strip * strip_len; v < v1; v++) {
            const int xy = vox_xy[v];
            const float vx = ((float)(xy & 0xffff) + 0.5f) * c.vox;
            const float vy = ((float)(xy >> 16) + 0.5f) * c.vox;
            WalkSetup ws;
            ws.Lx = ws.Ly = 0.f;
            ws.n = 0;
            ws.dlt = ws.ux = ws.uy = ff{0.f, 0.f};
            if (valid) walk_decide(P, c, exff, eyff, &rec->Rdx, &rec->Rdy, vx, vy, &ws);
            // rays mostly along x lie side by side along y: column-major copy
            const unsigned along_x = __ballot_sync(0xffffffffu, valid && fabsf(ws.Lx) > fabsf(ws.Ly));
            const unsigned any = __ballot_sync(0xffffffffu, valid);
            const bool colmajor = 2 * __popc(along_x) > __popc(any);
            const int per = (ws.n + split - 1) >> lg_split;
            ws.n = min(ws.n, (sub + 1) * per);
            const float2 none = make_float2(0.f, 0.f);
            const float k0 = (float)(sub * per);
            float2 A = colmajor ? walk_cells<false, FINE>(cells_t, P.ny + 1, 1, ncell_m1, ws, vx, vy, c, none, k0)
                                : walk_cells<false, FINE>(cells, 1, P.nx + 1, ncell_m1, ws, vx, vy, c, none, k0);
            for (int o = split >> 1; o > 0; o >>= 1) {
                A.x += __shfl_xor_sync(0xffffffffu, A.x, o);
                A.y += __shfl_xor_sync(0xffffffffu, A.y, o);
            }
            if (valid && sub == 0) out[v] = A;
        }
    }
}

} // namespace

cudaError_t launch_det_walk(const DevProblem &P, const PairRec *recs, bool list, long long n_items, const int *vox_xy,
                            int nv, const float4 *cells, float2 *tab, cudaStream_t s, int64_t *launches, bool early)
{
    if (n_items <= 0 || nv <= 0) return cudaSuccess;
    // Lanes per ray: up to 8, as far as 32 warps per SM have them with every
    // pair of the problem -- not of this launch, so that a pair's integrals do
    // not depend on the others that are asked for.
    const int sms = current_sm_count();
    const long long walks = (long long)P.n_src * P.n_det * nv;
    int lg_split = 0;
    while (lg_split < 3 && walks << (lg_split + 1) <= 1024LL * sms) lg_split++;
    const int rays = 32 >> lg_split;
    int nd = 0;
    long long n_groups;
    if (list) {
        n_groups = (n_items + rays - 1) / rays;
    } else {
        // whole pixels of every view
        if (n_items % P.n_src != 0) return cudaErrorInvalidValue;
        nd = (int)(n_items / P.n_src);
        n_groups = (long long)P.n_src * ((nd + rays - 1) / rays);
    }
    const int strip = (int)std::min<long long>(
        kMaxStrip, std::max<long long>(1, n_groups * nv / ((long long)sms * kItemsPerSM)));
    const long long nwork = n_groups * ((nv + strip - 1) / strip);
    long long blocks = (nwork + kWalkWarps - 1) / kWalkWarps;
    if (blocks > (long long)sms * 64) blocks = (long long)sms * 64;
    if (launches) (*launches)++;
    const F32Consts c = make_f32_consts(P);
    return launch_after(c.grain > 1.f ? k_det_walk<true> : k_det_walk<false>, (int)blocks, kWalkThreads, 0, s, early, P,
                        c, recs, list ? 1 : 0, n_items, nd, n_groups, strip, vox_xy, nv, cells, tab, lg_split);
}

} // namespace xrdt
