// k_mlem.cu -- MLEM with an explicit model matrix (main.m:154-176).
//
//   x <- x .* (A' * (y ./ (A*x + c + 1e-20))) ./ (sum(A,1)' + 1e-7)
//   x(~isfinite(x)) = 0;  x(x < 0) = 0
//
// A is the model matrix of Forward_XRD in its own layout: row r (a ray,
// src + det*SRC + nrg*SRC*DET) is the K = NWT*MAT contiguous floats
// Amatrix[:, :, ray] (main.m:140 reshapes it to [K, rays] and transposes).
//
// One iteration reads A once: L lanes take a ray, form t = A(r,:).x with a
// shuffle reduction, the ratio y_r / (t + c_r + 1e-20), and add ratio*A(r,:)
// into their register accumulators -- the same row, still in registers.  The
// first iteration adds up sum(A,1) on the same reading.  The pass is
// HBM-bound (2 flops per 4 bytes).  Each block writes its column sums to a
// partial row; the update kernel adds the partial rows in FP64, divides by
// the sensitivity sum(A,1) (also FP64) and applies the fix-ups.
//
// What keeps HBM busy:
//  * every lane has its own ring of 16-byte asynchronous copies in shared
//    memory (112 to 160 KB in flight per SM by the row's length, 128 at K = 256),
//    refilled as it is used, so no load waits for the arithmetic before it;
//  * the kernels of a call overlap (programmatic dependent launch): a pass
//    fills its ring, which needs A alone, while the update before it runs;
//  * passes go over a warp's rows forwards and backwards in turn, so that what
//    a pass read last, still in L2, is what the next one reads first (131072 x
//    256: 500 -> 440 us for ten iterations, with the loop as it then was).
// 131072 x 256, ten iterations: 220 us, against 198 for ten readings of A from
// HBM; with loads into registers, 11 passes and separate launches 344.
// 100000 x 64: 202 -> 90, 500 x 32: 99 -> 51 (the launches), 300000 x 256, five
// iterations: 353 -> 239, 40000 x 1024, ten: 322 -> 265.  A row per warp with
// its own division and reductions, and 64-bit addresses formed per row, issued
// twice the instructions: 425 us on the first.
#include <algorithm>

#include "xrdt_device.cuh"
#include "ff.cuh"

namespace xrdt {

namespace {

constexpr int kRingBytes = 192 * 1024;

// A row is L lanes x KC chunks of 16 bytes: lane l of the L holds columns
// 4l..4l+3 of every 4L-column chunk.  L < 32 (K <= 64) has one chunk and
// 32 / L rows in a warp.  A step of a warp's ring holds kRows visits (a visit
// is a row, or 32 / L rows): their sums are reduced together, so that a step
// takes one division and L / kRows lanes share it.
template <int L, int KC> struct MlemShape {
    static constexpr int kWarps = KC <= 4 ? 16 : 8;   // the first pass holds up to 20 KC registers
    static constexpr int kRows = KC >= 3 ? 2 : (L < 4 ? L : 4);
    static constexpr int kStepBytes = kWarps * kRows * KC * 512;   // of a block
    static constexpr int kSteps = kRingBytes / kStepBytes < 8 ? kRingBytes / kStepBytes : 8;
    static constexpr int kSmem = kSteps * kStepBytes;
};

// Sums over L lanes of P values each: lane l of the L gets the sum of value
// l / (L / P) (halves of the set are exchanged first: L = 32, P = 4 takes 6
// shuffles instead of 20).
template <int L, int P> __device__ __forceinline__ float sum_lanes(const float (&t)[P], int lane)
{
    float v;
    if constexpr (P == 4) {
        const bool up = lane & (L / 2), up2 = lane & (L / 4);
        float a = up ? t[2] : t[0], b = up ? t[3] : t[1];
        a += __shfl_xor_sync(0xffffffffu, up ? t[0] : t[2], L / 2);
        b += __shfl_xor_sync(0xffffffffu, up ? t[1] : t[3], L / 2);
        v = up2 ? b : a;
        v += __shfl_xor_sync(0xffffffffu, up2 ? a : b, L / 4);
    } else if constexpr (P == 2) {
        const bool up = lane & (L / 2);
        v = up ? t[1] : t[0];
        v += __shfl_xor_sync(0xffffffffu, up ? t[0] : t[1], L / 2);
    } else {
        v = t[0];
    }
#pragma unroll
    for (int o = L / P / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void copy16(uint32_t dst, const void *src, bool valid)
{
    const int n = valid ? 16 : 0;   // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

__device__ __forceinline__ void add4(float4 &s, float w, const float4 &a)
{
    s.x = fmaf(w, a.x, s.x);
    s.y = fmaf(w, a.y, s.y);
    s.z = fmaf(w, a.z, s.z);
    s.w = fmaf(w, a.w, s.w);
}

// FIRST: also the column sums of A, into partial rows gridDim.x ... 2 gridDim.x - 1.
template <int L, int KC, bool FIRST>
__global__ void __launch_bounds__(MlemShape<L, KC>::kWarps * 32)
k_mlem_pass(const float *__restrict__ A, long long rays, int K, const float *__restrict__ y,
            const float *__restrict__ c, const float *x, float *partial, int reverse)
{
    using S = MlemShape<L, KC>;
    constexpr int G = 32 / L, P = S::kRows;
    extern __shared__ __align__(16) float4 ring[];   // [kSteps][kWarps][P][KC][32]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int K4 = K >> 2, ql = lane & (L - 1);
    const long long gw = (long long)blockIdx.x * S::kWarps + wid;
    const long long nw = (long long)gridDim.x * S::kWarps;
    const long long visits = (rays + G - 1) / G;
    const int mine = gw < visits ? (int)((visits - 1 - gw) / nw + 1) : 0;   // visits of this warp
    const int steps = (mine + P - 1) / P;
    allow_dependents();

    float4 *const slot0 = ring + wid * P * KC * 32 + lane;
    constexpr int kStride = S::kWarps * P * KC * 32;
    // rows of visit 0, and from one visit to the next
    const long long row0 = (gw + (reverse ? mine - 1 : 0) * nw) * G + lane / L;
    const long long drow = (reverse ? -nw : nw) * G;
    // the copies, visit by visit; the last chunk of a row may be narrower
    // than the lanes
    const int q_last = min(ql + L * (KC - 1), K4 - 1);
    const bool in_last = ql + L * (KC - 1) < K4;
    const char *src = reinterpret_cast<const char *>(A + row0 * K + 4 * ql);
    const long long dsrc = drow * K * 4;
    const int last_off = 16 * (q_last - ql);
    long long crow = row0;
    int copied = 0;
    auto issue = [&](int slot) {
        if (copied < mine) {
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(slot0 + slot * kStride);
#pragma unroll
            for (int p = 0; p < P; p++) {
                const bool in = copied + p < mine && (G == 1 || crow < rays);
                const char *from = in ? src : reinterpret_cast<const char *>(A);
#pragma unroll
                for (int i = 0; i < KC; i++)
                    copy16(dst + (p * KC + i) * 512, from + (!in ? 0 : i == KC - 1 ? last_off : 16 * L * i),
                           in && (i < KC - 1 || in_last));
                src += dsrc;
                if (G > 1) crow += drow;
            }
            copied += P;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // y and c of this lane's visit of a step, one step ahead in registers
    const int own = ql / (L / P);
    long long yrow = row0 + own * drow;
    int yvisit = own;
    float yn, cn;
    bool on;
    auto load_yc = [&]() {
        on = yvisit < mine && (G == 1 || yrow < rays);
        yn = on ? __ldcg(y + yrow) : 0.f;
        cn = on ? __ldcg(c + yrow) : 0.f;
        yrow += P * drow;
        yvisit += P;
    };
    for (int s = 0; s < S::kSteps - 1; s++) issue(s);
    load_yc();
    // x and the partial rows belong to the update before until here
    await_predecessor();
    float4 xv[KC], g[KC], h[FIRST ? KC : 1];
#pragma unroll
    for (int i = 0; i < KC; i++) {
        const int q = ql + L * i;
        xv[i] = q < K4 ? __ldcg(reinterpret_cast<const float4 *>(x) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
        g[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (FIRST) h[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    int slot = 0, free_slot = S::kSteps - 1;
    for (int step = 0; step < steps; step++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::kSteps - 2) : "memory");
        float4 a[P][KC];
#pragma unroll
        for (int p = 0; p < P; p++)
#pragma unroll
            for (int i = 0; i < KC; i++) a[p][i] = slot0[slot * kStride + (p * KC + i) * 32];
        const float yc = yn, cc = cn;
        const bool oc = on;
        __syncwarp();
        issue(free_slot);   // the slot that the step before used up
        load_yc();
        float t[P];
#pragma unroll
        for (int p = 0; p < P; p++) {
            t[p] = 0.f;
#pragma unroll
            for (int i = 0; i < KC; i++)
                t[p] = fmaf(a[p][i].x, xv[i].x,
                            fmaf(a[p][i].y, xv[i].y, fmaf(a[p][i].z, xv[i].z, fmaf(a[p][i].w, xv[i].w, t[p]))));
        }
        const float sum = sum_lanes<L, P>(t, lane);
        const float own_ratio = oc ? yc / (sum + cc + 1e-20f) : 0.f;
        // a step's rows add up among themselves first: the long sums then round
        // once per step
        float4 add[KC], ones[FIRST ? KC : 1];
#pragma unroll
        for (int p = 0; p < P; p++) {
            const float ratio = L == 1 ? own_ratio : __shfl_sync(0xffffffffu, own_ratio, (lane & ~(L - 1)) + p * (L / P));
#pragma unroll
            for (int i = 0; i < KC; i++) {
                if (p == 0) {
                    add[i] = make_float4(ratio * a[0][i].x, ratio * a[0][i].y, ratio * a[0][i].z, ratio * a[0][i].w);
                    if (FIRST) ones[i] = a[0][i];
                } else {
                    add4(add[i], ratio, a[p][i]);
                    if (FIRST) add4(ones[i], 1.f, a[p][i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < KC; i++) {
            add4(g[i], 1.f, add[i]);
            if (FIRST) add4(h[i], 1.f, ones[i]);
        }
        free_slot = slot;
        slot = slot == S::kSteps - 1 ? 0 : slot + 1;
    }
    // the block's sums: rows of a warp, then the warps through shared memory
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < KC; i++) {
        auto fold = [&](float4 v, int at) {
#pragma unroll
            for (int o = L; o < 32; o <<= 1) {
                v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
                v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
                v.z += __shfl_xor_sync(0xffffffffu, v.z, o);
                v.w += __shfl_xor_sync(0xffffffffu, v.w, o);
            }
            ring[((at * S::kWarps + wid) * KC + i) * 32 + lane] = v;
        };
        fold(g[i], 0);
        if (FIRST) fold(h[i], 1);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < (FIRST ? 2 : 1) * KC * L; j += S::kWarps * 32) {
        const int at = j / (KC * L), q = j - at * KC * L;   // chunk q of the row
        if (q >= K4) continue;
        // (as float pairs: a partial row is rounded once)
        ff s[4] = {};
        for (int w = 0; w < S::kWarps; w++) {
            const float4 v = ring[((at * S::kWarps + w) * KC + q / L) * 32 + (q & (L - 1))];
            const float t[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const ff u = two_sum(s[i].hi, t[i]);
                s[i] = ff{u.hi, s[i].lo + u.lo};
            }
        }
        const float4 sum = make_float4(s[0].hi + s[0].lo, s[1].hi + s[1].lo, s[2].hi + s[2].lo, s[3].hi + s[3].lo);
        reinterpret_cast<float4 *>(partial + ((size_t)at * gridDim.x + blockIdx.x) * K)[q] = sum;
    }
}

// Sums over a warp of four doubles: lane l gets the sum of v[l / 8] (the
// halves of the set are exchanged first, so six additions instead of 20: FP64
// is what this kernel waits for).
__device__ __forceinline__ double warp_sum4(const double (&v)[4], int lane)
{
    const bool up = lane & 16;
    double a = up ? v[2] : v[0], b = up ? v[3] : v[1];
    a += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
    b += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
    const bool up8 = lane & 8;
    double s = up8 ? b : a;
    s += __shfl_xor_sync(0xffffffffu, up8 ? a : b, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}

constexpr int kUpdateThreads = 128;

// Four columns per block: the FP64 sums of their partial rows, then the
// multiplicative update.  `first`: the sensitivity from the second set of
// partial rows.
__global__ void __launch_bounds__(kUpdateThreads)
k_mlem_update(const float *partial, int nparts, int K, double *sens, float *x, int first)
{
    __shared__ double part[2][kUpdateThreads / 32][4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    allow_dependents();
    await_predecessor();
    for (int at = 0; at <= first; at++) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        for (int p = threadIdx.x; p < nparts; p += kUpdateThreads) {
            const float4 f = __ldcg(reinterpret_cast<const float4 *>(partial + ((size_t)at * nparts + p) * K) + blockIdx.x);
            v[0] += (double)f.x;
            v[1] += (double)f.y;
            v[2] += (double)f.z;
            v[3] += (double)f.w;
        }
        const double s = warp_sum4(v, lane);
        if ((lane & 7) == 0) part[at][wid][lane >> 3] = s;
    }
    __syncthreads();
    if (threadIdx.x >= 4) return;
    const int k = 4 * blockIdx.x + threadIdx.x;
    double s = 0.0, n = 0.0;
    for (int w = 0; w < kUpdateThreads / 32; w++) s += part[0][w][threadIdx.x];
    if (first) {
        for (int w = 0; w < kUpdateThreads / 32; w++) n += part[1][w][threadIdx.x];
        sens[k] = n;
    } else {
        n = __ldcg(sens + k);
    }
    float v = (float)((double)__ldcg(x + k) * s / (n + 1e-7));
    if (!isfinite(v)) v = 0.f;   // main.m:163
    if (v < 0.f) v = 0.f;        // main.m:176
    x[k] = v;
}

template <int L, int KC>
cudaError_t run_iterations(const float *A, long long rays, int K, const float *y, const float *c, float *x, int iters,
                           float *partial, int nparts, double *sens, cudaStream_t s)
{
    using S = MlemShape<L, KC>;
    static_assert(S::kSteps >= 2, "the block's sums take two steps of the ring");
    cudaError_t e =
        cudaFuncSetAttribute(k_mlem_pass<L, KC, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_mlem_pass<L, KC, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
    for (int it = 0; it < iters && e == cudaSuccess; it++) {
        // the first pass waits for whatever wrote its inputs
        e = launch_after(it ? k_mlem_pass<L, KC, false> : k_mlem_pass<L, KC, true>, nparts, S::kWarps * 32, S::kSmem, s,
                         it > 0, A, rays, K, y, c, (const float *)x, partial, it & 1);
        if (e == cudaSuccess)
            e = launch_after(k_mlem_update, K / 4, kUpdateThreads, 0, s, true, (const float *)partial, nparts, K, sens,
                             x, it == 0 ? 1 : 0);
    }
    return e;
}

} // namespace

int mlem_pass_blocks(int sm_count, long long rays, int K)
{
    // one block per SM; fewer when its warps would have no rows
    int lanes = 1;
    while (lanes < 32 && lanes * 4 < K) lanes *= 2;
    const long long visits = (rays * lanes + 31) / 32;
    const int warps = K <= 512 ? 16 : 8;
    return (int)std::min<long long>(sm_count, (visits + warps - 1) / warps);
}

cudaError_t launch_mlem_matrix(const float *A, long long rays, int K, const float *y, const float *c, float *x,
                               int iters, float *partial, int nparts, double *sens, cudaStream_t s, int64_t *launches)
{
    cudaError_t e = cudaErrorInvalidValue;
#define XRDT_RUN(l, kc) e = run_iterations<l, kc>(A, rays, K, y, c, x, iters, partial, nparts, sens, s)
    if (K <= 4) XRDT_RUN(1, 1);
    else if (K <= 8) XRDT_RUN(2, 1);
    else if (K <= 16) XRDT_RUN(4, 1);
    else if (K <= 32) XRDT_RUN(8, 1);
    else if (K <= 64) XRDT_RUN(16, 1);
    else if (K <= 128) XRDT_RUN(32, 1);
    else if (K <= 256) XRDT_RUN(32, 2);
    else if (K <= 384) XRDT_RUN(32, 3);
    else if (K <= 512) XRDT_RUN(32, 4);
    else if (K <= 640) XRDT_RUN(32, 5);
    else if (K <= 768) XRDT_RUN(32, 6);
    else if (K <= 896) XRDT_RUN(32, 7);
    else if (K <= 1024) XRDT_RUN(32, 8);
#undef XRDT_RUN
    if (launches) (*launches) += 2 * (int64_t)iters;
    return e;
}

} // namespace xrdt
