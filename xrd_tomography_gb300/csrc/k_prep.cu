// k_prep.cu -- per-call staging for the factored forward projector.
//
//  * k_build_cells: the (a1,a2) map as bilinear cells.  Replaces Copy2Vector
//    (Copy2Vector.cu:9-23) and the cudaArray/texture set-up of
//    Forward_XRD.cu:209-237: cell (ci,cj) holds the bilinear coefficients of
//    the four texels (ci-1..ci, cj-1..cj) of a zero-bordered map, about the
//    cell centre, as two float4, so one sample is two 16-byte loads and three
//    packed FMAs with no border tests.  The map is stored twice: row-major
//    (ci + cj (NX+1)) and behind it column-major (cj + ci (NY+1)), so that a
//    warp whose rays lie side by side along y reads neighbouring cells from
//    one cache line as well as one whose rays lie side by side along x.  A
//    uniform cell also carries the radius of the uniform square around it
//    (walk_cells, walk.cuh).  One block per 32 x 32 cells; coefficients from
//    float pairs (in FP64 the blocks of a small map queued on the FP64 pipes of
//    a few SMs: 24 us against 14 on 45x33).  Also
//    quantises the Compton table to u8 (integrate_diffraction.cu:66-74) and
//    gathers the spectrum windows.
//  * k_compact_voxels: non-empty voxels in the reference's loop order
//    (nx outer, ny inner; integrate_diffraction.cu:173-178) and the material
//    id check (ids above n_mat would index past Ifine in the reference).
//  * k_voxel_compton: the (a1,a2) sample of the Compton table lookup per voxel
//    (integrate_diffraction.cu:181-189), honouring the stale-coordinate quirk.
//  * k_src_atten: the source-side line integral per (source, voxel), which
//    the reference recomputes in every block (integrate_diffraction.cu:260).
#include <algorithm>

#include "xrdt_device.cuh"
#include "walk.cuh"

namespace xrdt {

namespace {

// (a + b) + (c + d) in float pairs, rounded to float (plain float sums where
// a pair's low part overflows to NaN).
__device__ __forceinline__ float sum4(float a, float b, float c, float d)
{
    const ff s = ff_add(two_sum(a, b), two_sum(c, d));
    return isfinite(s.hi) ? s.hi : (a + b) + (c + d);
}

// floor(x) clamped to 0 .. 255 (NaN: 0, as floor_to_int's lowest int), without
// a conversion: those share the FP64 pipe.
__device__ __forceinline__ unsigned char floor_u8(float x)
{
    if (!(x > 0.f)) return 0;
    if (x >= 255.f) return 255;
    return (unsigned char)(__float_as_uint(__fadd_rd(x, 8388608.f)) & 255u);   // 2^23
}

constexpr int kRows = 32 + 2 * kReach;   // cells of a tile and its surroundings, per side

__global__ void __launch_bounds__(1024)
k_build_cells(int nx, int ny, const float *__restrict__ a1, const float *__restrict__ a2,
                              float4 *__restrict__ cells, const float *__restrict__ S2,
                              unsigned char *__restrict__ s2u8, int ns2, const float *__restrict__ S1,
                              unsigned char *__restrict__ s1u8, const float *__restrict__ spec,
                              const int *__restrict__ win_lo, float *__restrict__ rf_win, int nrg_src, int nrf, int W,
                              int tiles)
{
    allow_dependents();
    if ((int)blockIdx.x >= tiles) {
        // ---- the blocks behind the cells: the tables ----
        const int i0 = ((int)blockIdx.x - tiles) * blockDim.x + threadIdx.x;
        const int step = ((int)gridDim.x - tiles) * blockDim.x;
        for (int i = i0; i < ns2; i += step) {
            s2u8[i] = floor_u8(S2[i]);
            if (S1) s1u8[i] = floor_u8(S1[i]);
        }
        // the spectrum windows: rf_win[n][j] = spectrum[win_lo[n] + j, n]
        for (int i = i0; i < nrf; i += step) {
            const int n = i / W, j = i - n * W;
            rf_win[i] = spec[win_lo[n] + j + (int64_t)n * nrg_src];
        }
        await_predecessor();
        return;
    }
    __shared__ unsigned uneven[kRows][3];
    __shared__ unsigned char row_dist[kRows][32];
    const int64_t ncell = (int64_t)(nx + 1) * (ny + 1);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int tiles_x = (nx + 1 + 31) >> 5;
    const int x0 = 32 * (int)(blockIdx.x % tiles_x), y0 = 32 * (int)(blockIdx.x / tiles_x);
    // texel (i, j) of the map with its zero border
    auto texel = [&](int i, int j) {
        const bool in = (i >= 0 && i < nx && j >= 0 && j < ny);
        const int64_t idx = in ? (int64_t)i + (int64_t)j * nx : 0;
        return in ? make_float2(a1[idx], a2[idx]) : make_float2(0.f, 0.f);
    };
    // ---- which cells of the tile and its surroundings are not uniform ----
    // row r of `uneven`: cells y0 - kReach + r, bit b: cell x0 - kReach + b;
    // cells outside the map count as uniform (no sample lies there)
#pragma unroll 3
    for (int i = wid; i < kRows * 3; i += 32) {
        const int r = i / 3, w = i - 3 * r;
        const int ci = x0 - kReach + 32 * w + lane, cj = y0 - kReach + r;
        bool odd = false;
        if (ci >= 0 && ci <= nx && cj >= 0 && cj <= ny && 32 * w + lane < kRows) {
            const float2 t = texel(ci, cj), l = texel(ci - 1, cj), d = texel(ci, cj - 1), e = texel(ci - 1, cj - 1);
            odd = !(t.x == l.x && t.x == d.x && t.x == e.x && t.y == l.y && t.y == d.y && t.y == e.y);
        }
        const unsigned m = __ballot_sync(0xffffffffu, odd);
        if (lane == 0) uneven[r][w] = m;
    }
    __syncthreads();
    // ---- per row and tile column: distance to the nearest one in the row ----
    for (int r = wid; r < kRows; r += 32) {
        const unsigned w0 = uneven[r][0], w1 = uneven[r][1], w2 = uneven[r][2];
        const int c = lane + kReach;   // this column's bit
        const unsigned right = c < 32 ? __funnelshift_r(w0, w1, c) : __funnelshift_r(w1, w2, c - 32);   // bits c ..
        const unsigned left = __funnelshift_r(w0, w1, lane);                                            // bits .. c
        const int dr = right ? __ffs(right) - 1 : 32, dl = left ? __clz(left) : 32;
        row_dist[r][lane] = (unsigned char)min(dr, dl);
    }
    __syncthreads();
    const int ci = x0 + lane, cj = y0 + wid;
    if (ci <= nx && cj <= ny) {
        int dist = row_dist[kReach + wid][lane];
        for (int dy = 1; dy < dist; dy++)
            dist = min(dist, max(dy, min((int)row_dist[kReach + wid - dy][lane], (int)row_dist[kReach + wid + dy][lane])));
        const int64_t c = (int64_t)ci + (int64_t)cj * (nx + 1);
        float v[2][2][2];
#pragma unroll
        for (int dj = 0; dj < 2; dj++)
#pragma unroll
            for (int di = 0; di < 2; di++) {
                const float2 t = texel(ci - 1 + di, cj - 1 + dj);
                v[dj][di][0] = t.x;
                v[dj][di][1] = t.y;
            }
        // bilinear coefficients per component q about the cell centre:
        // f(u,v) = c00 + c10 u + c01 v + c11 u v for u, v in [-1/2, 1/2]
        float c00[2], c10[2], c01[2], c11[2];
        for (int q = 0; q < 2; q++) {
            const float f00 = v[0][0][q], f10 = v[0][1][q], f01 = v[1][0][q], f11 = v[1][1][q];
            c00[q] = 0.25f * sum4(f00, f10, f01, f11);
            c10[q] = 0.5f * sum4(f10, -f00, f11, -f01);
            c01[q] = 0.5f * sum4(f01, -f00, f11, -f10);
            c11[q] = sum4(f11, -f01, f00, -f10);
        }
        // a uniform cell's c11 is 0: the first one carries twice the radius of
        // the uniform square around it, scaled below every coefficient that
        // is kept (walk_cells)
        if (fabsf(c11[0]) < kReachLimit) c11[0] = dist > 1 ? (float)(2 * (dist - 1)) * kReachUnit : 0.f;
        const float4 lo = make_float4(c00[0], c00[1], c10[0], c10[1]);
        const float4 hi = make_float4(c01[0], c01[1], c11[0], c11[1]);
        const int64_t ct = ncell + (int64_t)cj + (int64_t)ci * (ny + 1);
        cells[2 * c] = lo;
        cells[2 * c + 1] = hi;
        cells[2 * ct] = lo;
        cells[2 * ct + 1] = hi;
    }
    await_predecessor();   // launched early it must not end before what came before
}

// The position of each of a thread's flags (bit r of `keep`, r < 4, in order)
// among all flags of the block, after `base`; adds the block's total to base.
// cnt: [2][32], used in turn, so that one barrier per call is enough.
__device__ __forceinline__ int block_positions(unsigned keep, int *base, int (*cnt)[32], int turn)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int mine = __popc(keep);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) cnt[turn & 1][wid] = incl;
    __syncthreads();
    int w = cnt[turn & 1][lane];   // 32 warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += n;
    }
    const int before = wid ? __shfl_sync(0xffffffffu, w, wid ? wid - 1 : 0) : 0;
    const int pos = *base + before + incl - mine;
    *base += __shfl_sync(0xffffffffu, w, 31);
    return pos;
}

// One block of 1024 threads, four voxels per thread and round: stream
// compaction in loop order, then (order or tile_xy != NULL) the same voxels
// once more in tiles of 8 x 4 voxels: order[i] is the loop-order number of the
// i-th voxel in tile order, tile_xy[i] its packed coordinates.  Thirty-two neighbours in tile order lie within 8 x 4 voxels,
// in loop order within a strip 32 long: the lanes of a warp that takes them see
// more even scattering angles and distances.  rank: [nx*ny] scratch.
__global__ void __launch_bounds__(1024)
k_compact_voxels(int nx, int ny, int n_mat, const int32_t *__restrict__ seg, int *__restrict__ vox_xy,
                 int *__restrict__ vox_mat, int *__restrict__ counters, int *__restrict__ order, int *rank,
                 int *__restrict__ tile_xy)
{
    __shared__ int cnt[2][32];
    int bad = 0, base = 0, turn = 0;
    const int64_t total = (int64_t)nx * ny;
    for (int64_t L0 = 0; L0 < total; L0 += 4096, turn++) {
        int s[4], x[4], y[4];
        unsigned keep = 0;
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const int64_t L = L0 + 4 * (int)threadIdx.x + r;
            s[r] = 0;
            x[r] = y[r] = 0;
            if (L < total) {
                x[r] = (int)(L / ny);
                y[r] = (int)(L - (int64_t)x[r] * ny);
                s[r] = seg[(int64_t)x[r] + (int64_t)y[r] * nx];
            }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) {
            bad |= (s[r] > n_mat);
            if (s[r] > 0 && s[r] <= n_mat) keep |= 1u << r;
        }
        int pos = block_positions(keep, &base, cnt, turn);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const bool k = keep >> r & 1u;
            if (k) {
                vox_xy[pos] = x[r] | (y[r] << 16);
                vox_mat[pos] = s[r] - 1;
            }
            if (rank && L0 + 4 * (int)threadIdx.x + r < total) rank[(int64_t)x[r] + (int64_t)y[r] * nx] = k ? pos : -1;
            pos += k;
        }
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        counters[0] = base;
        counters[1] = bad;
    }
    if (!rank) return;
    const int nty = (ny + 3) >> 2;
    const int64_t quads = 8 * (int64_t)((nx + 7) >> 3) * nty;   // columns of four voxels
    base = 0;
    for (int64_t Q0 = 0; Q0 < quads; Q0 += 1024, turn++) {
        const int64_t q = Q0 + threadIdx.x;
        int v[4] = {-1, -1, -1, -1};
        unsigned keep = 0;
        if (q < quads) {
            const int64_t tile = q >> 3;
            const int tx = (int)(tile / nty), ty = (int)(tile - (int64_t)tx * nty);
            const int x = 8 * tx + (int)(q & 7);
#pragma unroll
            for (int r = 0; r < 4; r++)
                if (x < nx && 4 * ty + r < ny) v[r] = rank[(int64_t)x + (int64_t)(4 * ty + r) * nx];
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
            if (v[r] >= 0) keep |= 1u << r;
        int pos = block_positions(keep, &base, cnt, turn);
#pragma unroll
        for (int r = 0; r < 4; r++)
            if (v[r] >= 0) {
                if (order) order[pos] = v[r];
                if (tile_xy) tile_xy[pos] = vox_xy[v[r]];
                pos++;
            }
    }
}

__global__ void k_voxel_compton(DevProblem P, const float *__restrict__ a1, const float *__restrict__ a2,
                                const int *__restrict__ vox_xy, const int *__restrict__ counters,
                                int *__restrict__ vox_na, float *__restrict__ vox_a2, float *__restrict__ vox_ta)
{
    allow_dependents();
    const int nv = counters[0];
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x) {
        double sx = 0.0, sy = 0.0;  // stale coordinates start at (0,0)
        int use = P.quirk_stale ? v - 1 : v;
        if (use >= 0) {
            const int xy = vox_xy[use];
            sx = ((double)(xy & 0xffff) + 0.5) * P.vox;
            sy = ((double)(xy >> 16) + 0.5) * P.vox;
        }
        double a1now, a2now;
        bilinear_f64(a1, a2, P.nx, P.ny, sx, sy, &a1now, &a2now);
        const double l2a = log2(fabs(a1now / a2now));
        int na = floor_to_int((l2a - P.a_min) / P.da_tab);
        vox_na[v] = na < 0 ? 0 : (na >= P.na ? P.na - 1 : na);
        vox_a2[v] = (float)a2now;
        if (vox_ta) vox_ta[v] = (float)((l2a - P.a_min) / P.da_grid);   // clamped where it is used
    }
}

// 2^lg_split lanes per (source, voxel): attenuator(Rsrc, Rvox) of
// integrate_diffraction.cu:260, decided as the detector side's (walk_decide)
// and walked cell by cell from the voxel (walk_cells), each lane its share of the
// samples.  A warp takes neighbouring voxels of one source.
template <bool FINE>
__global__ void k_src_atten(DevProblem P, F32Consts c, const SrcGeom *__restrict__ sg, const int *__restrict__ vox_xy,
                            int nv, const float4 *__restrict__ cells, float2 *__restrict__ out, int lg_split)
{
    allow_dependents();
    const int64_t nwork = (int64_t)P.n_src * nv;
    const unsigned ncell_m1 = (unsigned)((P.nx + 1) * (P.ny + 1) - 1);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int split = 1 << lg_split, sub = threadIdx.x & (split - 1);
    // (the loop runs by whole warps: lanes past the end repeat the last walk)
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; (t & ~31) < nwork << lg_split; t += stride) {
        const int64_t w = min(t >> lg_split, nwork - 1);
        const int src = (int)(w / nv), v = (int)(w % nv);
        const int xy = vox_xy[v];
        const float vx = ((float)(xy & 0xffff) + 0.5f) * c.vox;
        const float vy = ((float)(xy >> 16) + 0.5f) * c.vox;
        const SrcGeom *g = sg + src;
        WalkSetup ws;
        walk_decide(P, c, ff_from_double(g->Rsrc_x), ff_from_double(g->Rsrc_y), &g->Rsrc_x, &g->Rsrc_y, vx, vy, &ws);
        const int per = (ws.n + split - 1) >> lg_split;
        ws.n = min(ws.n, (sub + 1) * per);
        float2 A = walk_cells<false, FINE>(cells, 1, P.nx + 1, ncell_m1, ws, vx, vy, c, make_float2(0.f, 0.f), (float)(sub * per));
        for (int o = split >> 1; o > 0; o >>= 1) {
            A.x += __shfl_xor_sync(0xffffffffu, A.x, o);
            A.y += __shfl_xor_sync(0xffffffffu, A.y, o);
        }
        if (sub == 0 && t >> lg_split < nwork) out[(int64_t)src * nv + v] = A;
    }
}

} // namespace

cudaError_t launch_prep_map(const DevProblem &P, const float *a1, const float *a2, const float *S2,
                            PrepBuffers &B, cudaStream_t s, int64_t *launches, const float *S1, const float *spec,
                            const int *win_lo, float *rf_win, bool early)
{
    // one block of 1024 threads per tile of 32 x 32 cells, and up to eight for
    // the tables
    const int tiles = ((P.nx + 1 + 31) / 32) * ((P.ny + 1 + 31) / 32);
    const int ns2 = S2 ? P.nq * P.na : 0, W = 2 * P.dnrg + 1, nrf = rf_win ? P.nrg_det * W : 0;
    const int more = std::min(8, (std::max(ns2, nrf) + 1023) / 1024);
    if (launches) (*launches)++;
    return launch_after(k_build_cells, tiles + more, 1024, 0, s, early, P.nx, P.ny, a1, a2, B.cells, S2, B.s2u8, ns2,
                        B.s1u8 ? S1 : nullptr, B.s1u8, spec, win_lo, rf_win, P.nrg_src, nrf, W, tiles);
}

cudaError_t launch_list_voxels(const DevProblem &P, const int32_t *seg, PrepBuffers &B, cudaStream_t s,
                               int64_t *launches)
{
    k_compact_voxels<<<1, 1024, 0, s>>>(P.nx, P.ny, P.n_mat, seg, B.vox_xy, B.vox_mat, B.counters, B.vox_order,
                                        B.vox_rank, nullptr);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_voxel_compton(const DevProblem &P, const float *a1, const float *a2, PrepBuffers &B, cudaStream_t s,
                                 int64_t *launches)
{
    // blocks of a warp: an FP64 logarithm per voxel, spread over the SMs (in
    // blocks of 256 a 45x33 map took 10.9 us on six of them, now 7)
    const int64_t nvox = (int64_t)P.nx * P.ny;
    int blocks = (int)std::min<int64_t>((nvox + 31) / 32, 16384);
    k_voxel_compton<<<blocks, 32, 0, s>>>(P, a1, a2, B.vox_xy, B.counters, B.vox_na, B.vox_a2, B.vox_ta);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

cudaError_t launch_prep_voxels(const DevProblem &P, const int32_t *seg, const float *a1,
                               const float *a2, PrepBuffers &B, cudaStream_t s, int64_t *launches)
{
    cudaError_t e = launch_list_voxels(P, seg, B, s, launches);
    return e == cudaSuccess ? launch_voxel_compton(P, a1, a2, B, s, launches) : e;
}

cudaError_t launch_compact_voxels(const DevProblem &P, const int32_t *seg, PrepBuffers &B, cudaStream_t s,
                                  int64_t *launches)
{
    k_compact_voxels<<<1, 1024, 0, s>>>(P.nx, P.ny, P.n_mat, seg, B.vox_order, B.vox_mat, B.counters, nullptr,
                                        B.vox_rank, B.vox_xy);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

int current_sm_count()
{
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();   // a failed query leaves no error behind for the next launch check
        return 152;
    }
    if (cached[dev] > 0) return cached[dev];
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
        cudaGetLastError();
        return 152;
    }
    cached[dev] = sms;
    return sms;
}

cudaError_t launch_src_atten(const DevProblem &P, const SrcGeom *d_src, int nv, PrepBuffers &B,
                             cudaStream_t s, int64_t *launches)
{
    if (nv == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    // lanes per walk: up to 8, as far as 32 warps per SM have them
    const int64_t items = (int64_t)P.n_src * nv;
    int lg_split = 0;
    while (lg_split < 3 && items << (lg_split + 1) <= 1024LL * sms) lg_split++;
    int64_t blocks = ((items << lg_split) + 127) / 128;
    if (blocks > (int64_t)sms * 16) blocks = (int64_t)sms * 16;
    const F32Consts c = make_f32_consts(P);
    auto *kernel = c.grain > 1.f ? k_src_atten<true> : k_src_atten<false>;
    kernel<<<(int)blocks, 128, 0, s>>>(P, c, d_src, B.vox_xy, nv, B.cells, B.atten_src, lg_split);
    if (launches) (*launches)++;
    return cudaGetLastError();
}

} // namespace xrdt
