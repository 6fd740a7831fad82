// direct.cu - softened O(n^2) direct sums.
//
// k_direct_fp64_pairs restates CpuParallelBackend.ComputeForces
// (src/CelestialMechanics.Physics/Solvers/CpuParallelBackend.cs:99-142) with
// GravityKernel.AccelerationCoeffFromSource (GravityKernel.cs:9-33): every
// FP64 operation rounded exactly as the C# code rounds it (no FMA
// contraction) and every target's terms summed in source-row order, so its
// output is bit-identical to that backend's.  It also
// replaces the reference GPU gravity_kernel (engine/src/cuda/gravity_kernel.cu:
// 20-95), which loads inactive sources with their real mass.
//
// The throughput kernels, k_direct_fp32 and k_direct_fp32_rows: Morton-sorted
// targets, sources in chunks, one persistent launch over a work queue of
// (targets, chunk) items so the grid ends evenly; sources arrive raw by
// cp.async in one of two shared-memory buffers while the previous ones are
// evaluated, and are converted to FP32 coordinates differenced in FP64 against
// the centre of mass of the 2560 targets around; several targets per thread so
// every broadcast shared-memory read feeds several pair evaluations; a Kahan
// fold of the FP32 partial sum of each j-tile (1024 sources).  The chunk
// partials are written in FP64 and k_direct_reduce adds them in chunk order, so
// the result depends neither on scheduling nor on which kernel ran.
//   * k_direct_fp32: 2560 targets per item, ten per thread, which keeps five
//     independent packed chains per source in flight and feeds the FMA pipe
//     best (measured against 4, 6 and 8), one block per SM.
//   * k_direct_fp32_rows: 256 targets per item, two per thread, five blocks of
//     128 threads per SM, sources staged 256 at a time: the queue ends evenly
//     and few bodies spread over all SMs.
#include <algorithm>

#include "direct.cuh"
#include "tree.cuh"

namespace nb {

constexpr int kD32Tile = 1024;  // sources per FP32 partial sum (a j-tile)
constexpr int kD32Threads = 256, kD32Per = 10;
constexpr int kD32Ref = kD32Threads * kD32Per;      // targets that share a reference point
constexpr int kD32Stage = kD32Tile / kD32Threads;   // sources staged per thread per j-tile
constexpr size_t kD32Smem = 2 * kD32Tile * sizeof(double4) + 2 * kD32Tile * sizeof(float4);
constexpr int kRowThreads = 128, kRowPer = 2, kRowBlocks = 5;
constexpr int kRowSub = 256;                        // sources staged at a time
constexpr int kRowTargets = kRowThreads * kRowPer;
static_assert(kD32Per % 2 == 0 && kRowPer % 2 == 0, "targets are packed two per f32x2 register");
static_assert(kD32Ref % kRowTargets == 0 && kD32Tile % kRowSub == 0, "rows lie inside one tile");

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
constexpr int kD32Unroll = 8;  // source loop unroll

__device__ __forceinline__ void kahan32(float& s, float& c, float x) {
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
}

// Targets and sources are the n sorted bodies (all active).  Item it covers
// target tile it / chunks and source chunk it % chunks; its partial sums go
// to part[(chunk * 3 + axis) * n + target].  The self pair has
// dx = dy = dz = 0 and contributes 0 when eps > 0; GUARD (used when
// eps == 0) zeroes 1/r at r = 0 instead of evaluating 0 * inf.
template <bool GUARD>
__global__ void __launch_bounds__(kD32Threads)
k_direct_fp32(int n, const double4* __restrict__ sbody, float eps2, int n_items, int chunks, int chunk_len, unsigned* __restrict__ ctr,
              double* __restrict__ part, unsigned long long* __restrict__ counter) {
    extern __shared__ __align__(16) unsigned char s_d32[];
    double4* raw = (double4*)s_d32;                       // [2][kD32Tile]
    float4* sj = (float4*)(raw + 2 * kD32Tile);
    float4* sj2 = sj + kD32Tile;
    __shared__ double s_box[4][kD32Threads / 32];
    __shared__ int s_item;
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(ctr, 1u);
        __syncthreads();
        const int it = s_item;
        __syncthreads();  // every thread has the item before thread 0 fetches the next
        if (it >= n_items) break;
        const int tile = it / chunks, chunk = it - tile * chunks;
        const int t0 = tile * (kD32Threads * kD32Per);
        const int j0 = chunk * chunk_len, j1 = min(n, j0 + chunk_len);
        // reference point: the target tile's centre of mass (the FP32
        // coordinates are most precise where the mass is)
        double acc[4] = {0.0, 0.0, 0.0, 0.0};  // m, m x, m y, m z
#pragma unroll
        for (int u = 0; u < kD32Per; u++) {
            const int i = t0 + u * kD32Threads + threadIdx.x;
            if (i < n) {
                const double4 b = sbody[i];
                acc[0] += b.w;
                acc[1] += b.w * b.x;
                acc[2] += b.w * b.y;
                acc[3] += b.w * b.z;
            }
        }
        for (int k = 0; k < 4; k++)
            for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xFFFFFFFFu, acc[k], o);
        if ((threadIdx.x & 31) == 0)
            for (int k = 0; k < 4; k++) s_box[k][threadIdx.x >> 5] = acc[k];
        __syncthreads();
        double4 ref;
        {
            double m = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
            for (int w = 0; w < kD32Threads / 32; w++) {
                m += s_box[0][w];
                mx += s_box[1][w];
                my += s_box[2][w];
                mz += s_box[3][w];
            }
            ref = m > 0.0 ? make_double4(mx / m, my / m, mz / m, 0.0) : sbody[t0];
        }
        float bx[kD32Per], by[kD32Per], bz[kD32Per];
        float sx[kD32Per], sy[kD32Per], sz[kD32Per], cx[kD32Per], cy[kD32Per], cz[kD32Per];
#pragma unroll
        for (int u = 0; u < kD32Per; u++) {
            const int i = t0 + u * kD32Threads + threadIdx.x;
            const double4 b = sbody[i < n ? i : n - 1];
            bx[u] = (float)(b.x - ref.x);
            by[u] = (float)(b.y - ref.y);
            bz[u] = (float)(b.z - ref.z);
            sx[u] = sy[u] = sz[u] = cx[u] = cy[u] = cz[u] = 0.f;
        }
        // the next j-tile's raw sources arrive by cp.async while the current
        // one is evaluated (two raw buffers)
        auto issue = [&](int b0, int buf) {
#pragma unroll
            for (int u = 0; u < kD32Stage; u++) {
                const int k = u * kD32Threads + threadIdx.x;
                if (b0 + k < j1) {
                    double4* dst = raw + buf * kD32Tile + k;
                    cp_async16(dst, &sbody[b0 + k]);
                    cp_async16((char*)dst + 16, (const char*)&sbody[b0 + k] + 16);
                }
            }
            cp_async_commit();
        };
        issue(j0, 0);
        int buf = 0;
        for (int base = j0; base < j1; base += kD32Tile, buf ^= 1) {
            if (base + kD32Tile < j1) {
                issue(base + kD32Tile, buf ^ 1);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();  // every thread's copies of this tile have landed
#pragma unroll
            for (int u = 0; u < kD32Stage; u++) {
                const int k = u * kD32Threads + threadIdx.x;
                const int j = base + k;
                float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j < j1) {
                    const double4 qn = raw[buf * kD32Tile + k];
                    q4 = make_float4((float)(qn.x - ref.x), (float)(qn.y - ref.y),
                                     (float)(qn.z - ref.z), (float)qn.w);
                }
                // each source duplicated into both halves of the packed pairs
                sj[k] = make_float4(q4.x, q4.x, q4.y, q4.y);
                sj2[k] = make_float4(q4.z, q4.z, q4.w, q4.w);
            }
            __syncthreads();
            const int cnt = min(kD32Tile, j1 - base);
            float tx[kD32Per], ty[kD32Per], tz[kD32Per];
#pragma unroll
            for (int u = 0; u < kD32Per; u++) tx[u] = ty[u] = tz[u] = 0.f;
            {
                // two targets per packed instruction; d = q - b, so each half
                // rounds exactly as fmaf(-f, b - q, t) and fmaf(b - q, b - q, .)
                constexpr int P = kD32Per / 2;
                f32x2 BX[P], BY[P], BZ[P], AX[P], AY[P], AZ[P];
#pragma unroll
                for (int p = 0; p < P; p++) {
                    BX[p] = pk2(bx[2 * p], bx[2 * p + 1]);
                    BY[p] = pk2(by[2 * p], by[2 * p + 1]);
                    BZ[p] = pk2(bz[2 * p], bz[2 * p + 1]);
                    AX[p] = AY[p] = AZ[p] = 0ull;
                }
                const f32x2 E2 = pk2(eps2, eps2);
#pragma unroll kD32Unroll
                for (int k = 0; k < cnt; k++) {
                    const float4 qa = sj[k], qb = sj2[k];
                    const f32x2 qx = pk2(qa.x, qa.y), qy = pk2(qa.z, qa.w);
                    const f32x2 qz = pk2(qb.x, qb.y), qm = pk2(qb.z, qb.w);
#pragma unroll
                    for (int p = 0; p < P; p++) {
                        const f32x2 dx = sub2(qx, BX[p]), dy = sub2(qy, BY[p]), dz = sub2(qz, BZ[p]);
                        const f32x2 r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, E2)));
                        float ra, rb;
                        upk2(r2, ra, rb);
                        float ia = rsqrt_ftz(ra), ib = rsqrt_ftz(rb);
                        if (GUARD) {
                            ia = ra > 0.f ? ia : 0.f;
                            ib = rb > 0.f ? ib : 0.f;
                        }
                        const f32x2 inv = pk2(ia, ib);
                        const f32x2 f = mul2(mul2(mul2(inv, inv), inv), qm);
                        AX[p] = fma2(f, dx, AX[p]);
                        AY[p] = fma2(f, dy, AY[p]);
                        AZ[p] = fma2(f, dz, AZ[p]);
                    }
                }
#pragma unroll
                for (int p = 0; p < P; p++) {
                    upk2(AX[p], tx[2 * p], tx[2 * p + 1]);
                    upk2(AY[p], ty[2 * p], ty[2 * p + 1]);
                    upk2(AZ[p], tz[2 * p], tz[2 * p + 1]);
                }
            }
#pragma unroll
            for (int u = 0; u < kD32Per; u++) {
                kahan32(sx[u], cx[u], tx[u]);
                kahan32(sy[u], cy[u], ty[u]);
                kahan32(sz[u], cz[u], tz[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kD32Per; u++) {
            const int i = t0 + u * kD32Threads + threadIdx.x;
            if (i < n) {
                part[(size_t)(chunk * 3 + 0) * n + i] = (double)sx[u] - (double)cx[u];
                part[(size_t)(chunk * 3 + 1) * n + i] = (double)sy[u] - (double)cy[u];
                part[(size_t)(chunk * 3 + 2) * n + i] = (double)sz[u] - (double)cz[u];
            }
        }
        if (threadIdx.x == 0 && counter) {
            const int nt = min(kD32Threads * kD32Per, n - t0);
            atomicAdd(counter, (unsigned long long)nt * (unsigned long long)(j1 - j0));
        }
    }
}

// The reference points of the rows: the same sums as above.
__global__ void __launch_bounds__(kD32Threads)
k_direct_ref(int n, const double4* __restrict__ sbody, double4* __restrict__ ref) {
    __shared__ double s_box[4][kD32Threads / 32];
    const int t0 = blockIdx.x * kD32Ref;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};  // m, m x, m y, m z
#pragma unroll
    for (int u = 0; u < kD32Per; u++) {
        const int i = t0 + u * kD32Threads + threadIdx.x;
        if (i < n) {
            const double4 b = sbody[i];
            acc[0] += b.w;
            acc[1] += b.w * b.x;
            acc[2] += b.w * b.y;
            acc[3] += b.w * b.z;
        }
    }
    for (int k = 0; k < 4; k++)
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xFFFFFFFFu, acc[k], o);
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 4; k++) s_box[k][threadIdx.x >> 5] = acc[k];
    __syncthreads();
    if (threadIdx.x != 0) return;
    double m = 0.0, mx = 0.0, my = 0.0, mz = 0.0;
    for (int w = 0; w < kD32Threads / 32; w++) {
        m += s_box[0][w];
        mx += s_box[1][w];
        my += s_box[2][w];
        mz += s_box[3][w];
    }
    ref[blockIdx.x] = m > 0.0 ? make_double4(mx / m, my / m, mz / m, 0.0) : sbody[t0];
}

// As k_direct_fp32 over rows of kRowTargets, with the shell theorem too (a
// source of radius R pulls as a softened shell inside it).
template <bool SHELL, bool GUARD>
__global__ void __launch_bounds__(kRowThreads, kRowBlocks)
k_direct_fp32_rows(int n, const double4* __restrict__ sbody, const float* __restrict__ srad,
              float eps2, const double4* __restrict__ refs, int n_items, int chunks,
              int chunk_len, unsigned* __restrict__ ctr, double* __restrict__ part,
              unsigned long long* __restrict__ counter) {
    constexpr int PER = kRowPer, kThreads = kRowThreads, kSub = kRowSub;
    constexpr int kStage = kSub / kThreads;  // sources staged per thread
    // static shared memory: its constant addresses make the kernel 2 % faster
    constexpr size_t kBytes = kSub * (2 * sizeof(double4) + 2 * sizeof(float4) +
                                      (SHELL ? 2 * sizeof(float) + sizeof(float2) : 0));
    __shared__ __align__(16) unsigned char s_own[kBytes];
    double4* raw = (double4*)s_own;      // [2][kSub]
    float4* sj = (float4*)(raw + 2 * kSub);
    float4* sj2 = sj + kSub;
    float2* ss = (float2*)(sj2 + kSub);  // shell theorem only, as rawR
    float* rawR = (float*)(ss + kSub);   // [2][kSub]
    __shared__ int s_item;
    if (blockIdx.x == 0 && threadIdx.x == 0 && counter)
        atomicAdd(counter, (unsigned long long)n * (unsigned long long)n);
    for (;;) {
        if (threadIdx.x == 0) s_item = (int)atomicAdd(ctr, 1u);
        __syncthreads();
        const int it = s_item;
        __syncthreads();  // every thread has the item before thread 0 fetches the next
        if (it >= n_items) break;
        const int row = it / chunks, chunk = it - row * chunks;
        const int t0 = row * (kThreads * PER);
        const int j0 = chunk * chunk_len, j1 = min(n, j0 + chunk_len);
        const double4 ref = refs[t0 / kD32Ref];
        float bx[PER], by[PER], bz[PER];
        float sx[PER], sy[PER], sz[PER], cx[PER], cy[PER], cz[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = t0 + u * kThreads + threadIdx.x;
            const double4 b = sbody[i < n ? i : n - 1];
            bx[u] = (float)(b.x - ref.x);
            by[u] = (float)(b.y - ref.y);
            bz[u] = (float)(b.z - ref.z);
            sx[u] = sy[u] = sz[u] = cx[u] = cy[u] = cz[u] = 0.f;
        }
        // the next j-tile's raw sources arrive by cp.async while the current
        // one is evaluated (two raw buffers)
        auto issue = [&](int b0, int buf) {
#pragma unroll
            for (int u = 0; u < kStage; u++) {
                const int k = u * kThreads + threadIdx.x;
                if (b0 + k < j1) {
                    double4* dst = raw + buf * kSub + k;
                    cp_async16(dst, &sbody[b0 + k]);
                    cp_async16((char*)dst + 16, (const char*)&sbody[b0 + k] + 16);
                    if (SHELL) cp_async4(rawR + buf * kSub + k, &srad[b0 + k]);
                }
            }
            cp_async_commit();
        };
        issue(j0, 0);
        int buf = 0;
        for (int tile = j0; tile < j1; tile += kD32Tile) {
            float tx[PER], ty[PER], tz[PER];
            constexpr int P = PER / 2;
            f32x2 BX[P], BY[P], BZ[P], AX[P], AY[P], AZ[P];
#pragma unroll
            for (int p = 0; p < P; p++) {
                BX[p] = pk2(bx[2 * p], bx[2 * p + 1]);
                BY[p] = pk2(by[2 * p], by[2 * p + 1]);
                BZ[p] = pk2(bz[2 * p], bz[2 * p + 1]);
                AX[p] = AY[p] = AZ[p] = 0ull;
            }
            const int tile_end = min(tile + kD32Tile, j1);
            for (int base = tile; base < tile_end; base += kSub, buf ^= 1) {
                if (base + kSub < j1) {
                    issue(base + kSub, buf ^ 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncthreads();  // every thread's copies of these sources have landed
#pragma unroll
                for (int u = 0; u < kStage; u++) {
                    const int k = u * kThreads + threadIdx.x;
                    const int j = base + k;
                    float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f);
                    float R = 0.f;
                    if (j < j1) {
                        const double4 qn = raw[buf * kSub + k];
                        q4 = make_float4((float)(qn.x - ref.x), (float)(qn.y - ref.y),
                                         (float)(qn.z - ref.z), (float)qn.w);
                        if (SHELL) R = rawR[buf * kSub + k];
                    }
                    // each source duplicated into both halves of the packed pairs
                    sj[k] = make_float4(q4.x, q4.x, q4.y, q4.y);
                    sj2[k] = make_float4(q4.z, q4.z, q4.w, q4.w);
                    if (SHELL) {
                        const float id = rsqrtf(R * R + eps2);
                        ss[k] = j < j1 ? make_float2(R > 0.f ? R * R : 0.f, q4.w * id * id * id)
                                       : make_float2(0.f, 0.f);
                    }
                }
                __syncthreads();
                const int cnt = min(kSub, j1 - base);
                // two targets per packed instruction; d = q - b, so each half
                // rounds exactly as fmaf(-f, b - q, t) and fmaf(b - q, b - q, .)
                const f32x2 E2 = pk2(eps2, eps2);
#pragma unroll kD32Unroll
                for (int k = 0; k < cnt; k++) {
                    const float4 qa = sj[k], qb = sj2[k];
                    const f32x2 qx = pk2(qa.x, qa.y), qy = pk2(qa.z, qa.w);
                    const f32x2 qz = pk2(qb.x, qb.y), qm = pk2(qb.z, qb.w);
                    const float2 sh = SHELL ? ss[k] : make_float2(0.f, 0.f);
#pragma unroll
                    for (int p = 0; p < P; p++) {
                        const f32x2 dx = sub2(qx, BX[p]), dy = sub2(qy, BY[p]), dz = sub2(qz, BZ[p]);
                        f32x2 r2, raw2 = 0ull;
                        if constexpr (SHELL) {
                            raw2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
                            r2 = add2(raw2, E2);
                        } else {
                            r2 = fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, E2)));
                        }
                        float ra, rb;
                        upk2(r2, ra, rb);
                        float ia = rsqrt_ftz(ra), ib = rsqrt_ftz(rb);
                        if (GUARD) {
                            ia = ra > 0.f ? ia : 0.f;
                            ib = rb > 0.f ? ib : 0.f;
                        }
                        const f32x2 inv = pk2(ia, ib);
                        f32x2 f = mul2(mul2(mul2(inv, inv), inv), qm);
                        if constexpr (SHELL) {
                            float wa, wb, fa, fb;
                            upk2(raw2, wa, wb);
                            upk2(f, fa, fb);
                            f = pk2(wa < sh.x ? sh.y : fa, wb < sh.x ? sh.y : fb);
                        }
                        AX[p] = fma2(f, dx, AX[p]);
                        AY[p] = fma2(f, dy, AY[p]);
                        AZ[p] = fma2(f, dz, AZ[p]);
                    }
                }
            }
            // the j-tile's FP32 sums go into the compensated ones
#pragma unroll
            for (int p = 0; p < P; p++) {
                upk2(AX[p], tx[2 * p], tx[2 * p + 1]);
                upk2(AY[p], ty[2 * p], ty[2 * p + 1]);
                upk2(AZ[p], tz[2 * p], tz[2 * p + 1]);
            }
#pragma unroll
            for (int u = 0; u < PER; u++) {
                kahan32(sx[u], cx[u], tx[u]);
                kahan32(sy[u], cy[u], ty[u]);
                kahan32(sz[u], cz[u], tz[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = t0 + u * kThreads + threadIdx.x;
            if (i < n) {
                part[(size_t)(chunk * 3 + 0) * n + i] = (double)sx[u] - (double)cx[u];
                part[(size_t)(chunk * 3 + 1) * n + i] = (double)sy[u] - (double)cy[u];
                part[(size_t)(chunk * 3 + 2) * n + i] = (double)sz[u] - (double)cz[u];
            }
        }
    }
}

// Sum of the chunk partials in chunk order, written by body row.
__global__ void k_direct_reduce(int n, int chunks, const double* __restrict__ part,
                                const uint32_t* __restrict__ sidx, double* __restrict__ ax,
                                double* __restrict__ ay, double* __restrict__ az) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s[3] = {0.0, 0.0, 0.0};
    for (int c = 0; c < chunks; c++)
        for (int k = 0; k < 3; k++) s[k] += part[(size_t)(c * 3 + k) * n + i];
    const uint32_t row = sidx[i];
    ax[row] = s[0];
    ay[row] = s[1];
    az[row] = s[2];
}

// The FP64 pair sum.  Every target's terms have to be subtracted one by one
// in source order (that order is what makes the result bit-identical to
// CpuParallelBackend's), so a target component is one chain of n dependent
// additions; the costly part of a term (a correctly rounded square root and
// division) is not part of the chain.  A block therefore has producer warps,
// which compute the TI x kPTj pair terms of a source tile (each rounded
// exactly as the CPU code rounds it) into one of two shared-memory buffers,
// and one accumulator warp, whose lane (target, component) walks the other
// buffer meanwhile: one barrier a tile, and the chain and the term arithmetic
// overlap.  A term that is not added (the body itself, an inactive source) is
// stored as +0, whose subtraction changes no bit.  The chain bounds a small
// system (1000 dependent additions), the square root and division a large
// one; the two buffers are 2 x 25 KB at TI = 8, and three blocks share an SM.
// Two phases of a tile behind one another, 256 threads for both, took 51.2 us
// for 1,000 bodies, 731 us for 8,192 and 3.47 ms for 20,000; now 21.5, 273 and
// 1,424 us (call times on the stream; 10, 53 and 60 % of the FP64 rate by some
// 40 operations a pair).  Half the tile (64 sources) was 17 to 28 % slower.
//
// A step of the integrator needs nothing else: the accumulator lane that ends
// with component c of a body's acceleration closes the step (v += dt/2 a) and
// opens the next one (v += dt'/2 a, x' = x + dt' v, in the order and rounding
// of SoAVerletIntegrator.Step), writing x' to the other position buffer, since
// other blocks may still read x.  One launch a step, each started while its
// predecessor ends, instead of three and four memsets: 1,000 bodies 43.3 ->
// 11.0 us a step, 200 bodies 20.7 -> 4.9, 3,000 bodies 117 -> 43.8.
//
// ORDER selects the rounding and summation order of another CPU backend of
// the desktop app (without the shell theorem; with it every backend runs
// CpuParallelBackend's arithmetic):
//   kOrderParallel  CpuParallelBackend: c = ((m*inv)*inv)*inv, one running sum;
//   kOrderSimd      SimdSingleThreadBackend (SimdSingleThreadBackend.cs:43-165)
//                   and the native engine's CPU brute force (engine/src/sim/
//                   engine.cpp:649-674): c = m*((inv*inv)*inv), sources in
//                   row order (the vector lanes are summed in lane order);
//   kOrderPairwise  CpuSingleThreadBackend's Newton's-third-law loop
//                   (CpuSingleThreadBackend.cs:50-159): the same c, and a
//                   body's sum is (its running sum over lower rows, which the
//                   loop adds into ax[j] as +c*(x_lower - x_j), i.e. minus
//                   the term) + (its running sum over higher rows).
constexpr int kPTj = 128;        // sources per tile
constexpr int kPRow = kPTj + 2;  // padded row: the lanes' 16-byte reads meet no bank twice

template <int TI, bool MANY>
struct Fp64Shape {
    // producer threads: one block per SM (not MANY) hides the term's latency
    // with threads, several blocks with independent terms per thread
    static constexpr int most = MANY ? 256 : 512;
    static constexpr int producers = TI * kPTj < most ? TI * kPTj : most;
    static constexpr int threads = 32 + producers;
    static constexpr int blocks = MANY ? 3 : 1;
    static constexpr size_t smem = sizeof(double) * 2 * 3 * TI * kPRow;
};

template <bool SHELL, int ORDER, int TI, bool MANY>
__global__ void __launch_bounds__(Fp64Shape<TI, MANY>::threads, Fp64Shape<TI, MANY>::blocks)
k_direct_fp64_pairs(Fp64Args a) {
    constexpr int kProd = Fp64Shape<TI, MANY>::producers;
    constexpr int kPer = TI * kPTj / kProd;  // terms per producer thread and tile
    static_assert(kProd % kPTj == 0 && kPer * kProd == TI * kPTj && 3 * TI <= 32, "block shape");
    extern __shared__ __align__(16) double s_t[];  // [2][3 TI][kPRow]
    __shared__ double s_i[TI][3];
    __shared__ uint8_t s_iact[TI];
    // the previous step's kernel has ended, and its stores are visible (a
    // launch without the overlap attribute passes at once)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int n = a.n;
    const int i0 = blockIdx.x * TI;
    if (threadIdx.x < TI) {
        const int i = i0 + threadIdx.x;
        const bool me = i < n && a.act[i];
        const double x = me ? a.px[i] : 0.0, y = me ? a.py[i] : 0.0, z = me ? a.pz[i] : 0.0;
        s_iact[threadIdx.x] = me;
        s_i[threadIdx.x][0] = x;
        s_i[threadIdx.x][1] = y;
        s_i[threadIdx.x][2] = z;
        if (me && !(isfinite(x) && isfinite(y) && isfinite(z) && isfinite(a.m[i])))
            dev_flag(a.err, kErrNonFinite);
    }
    __syncthreads();
    const int tiles = (n + kPTj - 1) / kPTj;
    constexpr bool kSplit = !SHELL && ORDER == kOrderPairwise;
    if (threadIdx.x >= 32) {
        // producer: source column tj of every tile, targets ti0, ti0 + kProd / kPTj, ...
        const int p = threadIdx.x - 32;
        const int tj = p % kPTj, ti0 = p / kPTj;
        double xj = 0.0, yj = 0.0, zj = 0.0, mj = 0.0, R = 0.0;
        bool aj = false;
        auto load = [&](int j) {
            aj = j < n && a.act[j];
            if (aj) {
                xj = a.px[j];
                yj = a.py[j];
                zj = a.pz[j];
                mj = a.m[j];
                if (SHELL) R = a.rad[j];
            }
        };
        load(tj);
        for (int t = 0; t <= tiles; t++) {
            if (t < tiles) {
                const int j = t * kPTj + tj;
                const double cx = xj, cy = yj, cz = zj, cm = mj, cR = R;
                const bool ca = aj;
                load(j + kPTj);  // the next tile's words travel while this one is computed
                double* out = s_t + (t & 1) * (3 * TI * kPRow) + tj;
#pragma unroll
                for (int k = 0; k < kPer; k++) {
                    const int ti = ti0 + k * (kProd / kPTj);
                    double tx = 0.0, ty = 0.0, tz = 0.0;
                    if (ca && j != i0 + ti) {
                        const double dx = __dsub_rn(s_i[ti][0], cx);
                        const double dy = __dsub_rn(s_i[ti][1], cy);
                        const double dz = __dsub_rn(s_i[ti][2], cz);
                        const double raw = __dadd_rn(
                            __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                        double c;
                        if (SHELL && cR > 0.0 && sqrt(raw) < cR) {
                            const double den = __dadd_rn(__dmul_rn(cR, cR), a.eps2);
                            const double ids = 1.0 / sqrt(den);
                            c = __dmul_rn(cm, ids) / den;
                        } else {
                            const double inv = 1.0 / sqrt(__dadd_rn(raw, a.eps2));
                            c = !SHELL && ORDER != kOrderParallel
                                    ? __dmul_rn(cm, __dmul_rn(__dmul_rn(inv, inv), inv))
                                    : __dmul_rn(__dmul_rn(__dmul_rn(cm, inv), inv), inv);
                        }
                        tx = __dmul_rn(c, dx);
                        ty = __dmul_rn(c, dy);
                        tz = __dmul_rn(c, dz);
                    }
                    out[(3 * ti + 0) * kPRow] = tx;
                    out[(3 * ti + 1) * kPRow] = ty;
                    out[(3 * ti + 2) * kPRow] = tz;
                }
            }
            __syncthreads();
        }
        return;
    }
    // accumulator lane: (target, component)
    const int lane = threadIdx.x < 3 * TI ? threadIdx.x : 0;
    const int acc_t = lane / 3, acc_c = lane % 3;
    const int i = i0 + acc_t;
    double sum = 0.0;
    double hi = 0.0;  // kSplit: the sum over higher rows (sum holds the lower rows')
    for (int t = 0; t <= tiles; t++) {
        if (t > 0) {
            const int base = (t - 1) * kPTj;
            const double2* row =
                (const double2*)(s_t + ((t - 1) & 1) * (3 * TI * kPRow) + lane * kPRow);
            const int cnt = min(kPTj, n - base);
            if (kSplit) {
                const int split = i - base;  // first tj with j > i (the body's own term is 0)
                const double* r = (const double*)row;
                for (int tj = 0; tj < cnt; tj++) {
                    if (tj < split) sum = __dsub_rn(sum, r[tj]);
                    else hi = __dsub_rn(hi, r[tj]);
                }
            } else {
                // rows past n were stored as 0
                const int blocks = (cnt + 15) / 16;
                for (int k = 0; k < blocks; k++) {
                    double2 v[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) v[u] = row[8 * k + u];
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        sum = __dsub_rn(sum, v[u].x);
                        sum = __dsub_rn(sum, v[u].y);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x >= 3 * TI || i >= n) return;
    const bool me = s_iact[acc_t];
    if (kSplit) sum = __dadd_rn(sum, hi);
    if (!me) sum = 0.0;
    a.acc[acc_c][i] = sum;
    if (!a.close && !a.open) return;
    double v = 0.0;
    if (me) {
        v = a.vel[acc_c][i];
        if (a.close) v = __dadd_rn(v, __dmul_rn(0.5 * a.dt_close, sum));
        if (a.open) v = __dadd_rn(v, __dmul_rn(0.5 * a.dt_open, sum));
        a.vel[acc_c][i] = v;
    }
    if (a.open) {
        const double x = acc_c == 0 ? a.px[i] : acc_c == 1 ? a.py[i] : a.pz[i];
        a.next[acc_c][i] = me ? __dadd_rn(x, __dmul_rn(a.dt_open, v)) : x;
    }
}

// Opens the first of a run of steps: v += dt/2 a, x' = x + dt v for active
// rows, every row's position to `next` (which may be the position arrays).
__global__ void k_fp64_open(Fp64Args a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const bool me = a.act[i];
    const double* const pos[3] = {a.px, a.py, a.pz};
#pragma unroll
    for (int c = 0; c < 3; c++) {
        double x = pos[c][i];
        if (me) {
            const double v = __dadd_rn(a.vel[c][i], __dmul_rn(0.5 * a.dt_open, a.acc[c][i]));
            a.vel[c][i] = v;
            x = __dadd_rn(x, __dmul_rn(a.dt_open, v));
        }
        a.next[c][i] = x;
    }
}

namespace {

template <bool SHELL, int ORDER, int TI, bool MANY>
cudaError_t launch_fp64(cudaStream_t st, const Fp64Args& a) {
    using Shape = Fp64Shape<TI, MANY>;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(a.n, TI));
    cfg.blockDim = dim3(Shape::threads);
    cfg.dynamicSmemBytes = Shape::smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_direct_fp64_pairs<SHELL, ORDER, TI, MANY>, a);
}

template <bool SHELL, int ORDER, bool MANY>
void init_fp64() {
    cudaFuncSetAttribute((const void*)k_direct_fp64_pairs<SHELL, ORDER, 8, MANY>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)Fp64Shape<8, MANY>::smem);
}

template <int TI, bool MANY>
cudaError_t launch_fp64_order(cudaStream_t st, const Fp64Args& a, bool shell, int order) {
    if (shell) return launch_fp64<true, kOrderParallel, TI, MANY>(st, a);
    if (order == kOrderSimd) return launch_fp64<false, kOrderSimd, TI, MANY>(st, a);
    if (order == kOrderPairwise) return launch_fp64<false, kOrderPairwise, TI, MANY>(st, a);
    return launch_fp64<false, kOrderParallel, TI, MANY>(st, a);
}

template <bool MANY>
void init_fp64_orders() {
    init_fp64<true, kOrderParallel, MANY>();
    init_fp64<false, kOrderParallel, MANY>();
    init_fp64<false, kOrderSimd, MANY>();
    init_fp64<false, kOrderPairwise, MANY>();
}

}  // namespace

void direct_init() {
    init_fp64_orders<false>();
    init_fp64_orders<true>();
}

// Targets per block: the fewest of 2, 4, 8 that still gives every block an SM
// of its own (a block's chain takes as long for 2 targets as for 8, and its
// terms take less); beyond that 8 targets, which share the source loads, in
// smaller blocks with more independent terms per thread, several to an SM.
// Measured at 8,192 bodies: 512 producers 460 us, 256 273, 128 276; at 1,000
// bodies (8 targets, one block per SM) 512 producers 11.4 us a step, 256 12.2.
cudaError_t direct_fp64(cudaStream_t st, const Fp64Args& a, bool shell, int order, int sms) {
    if (a.n <= 0) return cudaSuccess;
    if (ceil_div(a.n, 2) <= sms) return launch_fp64_order<2, false>(st, a, shell, order);
    if (ceil_div(a.n, 4) <= sms) return launch_fp64_order<4, false>(st, a, shell, order);
    if (ceil_div(a.n, 8) <= sms) return launch_fp64_order<8, false>(st, a, shell, order);
    return launch_fp64_order<8, true>(st, a, shell, order);
}

// The opening kick-drift writes positions to the buffer from which the
// alternation ends in pos[0], so the caller's arrays hold the final state.
cudaError_t direct_fp64_steps(cudaStream_t st, Fp64Args a, bool shell, int order, int sms,
                              double* const pos[2][3], const double* dts, int n_dt, int steps) {
    if (a.n <= 0 || steps <= 0) return cudaSuccess;
    int buf = (steps - 1) & 1;
    auto use = [&](int from, int to) {
        a.px = pos[from][0];
        a.py = pos[from][1];
        a.pz = pos[from][2];
        for (int c = 0; c < 3; c++) a.next[c] = pos[to][c];
    };
    use(0, buf);
    a.dt_open = dts[0];
    k_fp64_open<<<ceil_div(a.n, 256), 256, 0, st>>>(a);
    cudaError_t e = cudaPeekAtLastError();
    for (int k = 0; k < steps && e == cudaSuccess; k++, buf ^= 1) {
        use(buf, buf ^ 1);
        a.close = true;
        a.open = k + 1 < steps;
        a.dt_close = dts[k % n_dt];
        a.dt_open = dts[(k + 1) % n_dt];
        e = direct_fp64(st, a, shell, order, sms);
    }
    return e;
}

// Fullness of the tiles' waves (items over the slots of their whole waves) from
// which k_direct_fp32 is the faster one: its items run 2.5 % faster than the
// rows', which end evenly whatever their number.  tile / row kernel, ms: 50,000
// bodies (0.88 full) 1.13 / 1.07, 100,003 0.81 full 4.80 / 3.98 and 0.99 full
// (a roomier handle: more chunks) 3.95 / 3.97, 150,000 0.96 full 8.98 / 8.87 and
// 0.997 full 8.64 / 8.85, 262,144 (0.994) 26.3 / 27.0, 350,000 0.93 full 50.0 /
// 48.4 and 0.997 full 46.5 / 47.8.
constexpr double kD32TileFill = 0.975;

void direct_fp32(cudaStream_t st, int n, const double4* sbody, const float* srad,
                 const uint32_t* sidx, double eps, bool shell, double* ax, double* ay,
                 double* az, unsigned long long* counter, double* part, double4* ref, int capacity,
                 unsigned* ctr, int sms) {
    if (n <= 0) return;
    const float eps2 = (float)(eps * eps);
    // Chunks: from each chunk on the j-tiles start anew, so the chunk length
    // decides how the FP32 sums round, and it keeps to this rule: items of
    // kD32Ref targets make at least 4 waves on one block per SM where 4096
    // sources per chunk and some 290 bytes of `part` per body allow it, and among
    // those counts the fewest chunks within 0.5 % of the fullest last wave.  (The
    // byte count keeps the chunks where they were when the tree's memory, which
    // `part` is, had that size; it never exceeds what is there.)
    const int tiles = ceil_div(n, kD32Ref);
    const long long room = std::min<long long>(
        290LL * capacity + (capacity / 1024 + 2) * 4 + 1328, (long long)tree_bytes(capacity));
    const long long cmax =
        std::max<long long>(1, std::min<long long>(std::max(1, ceil_div(n, 4096)), room / (24LL * n)));
    const long long cmin = std::min<long long>(cmax, std::max(1, ceil_div(4LL * sms, tiles)));
    auto fill = [&](long long c) {
        const long long nc = ceil_div(n, ceil_div(n, (int)c));  // chunks actually formed
        const long long it = (long long)tiles * nc;
        return (double)it / (double)(((it + sms - 1) / sms) * sms);
    };
    double best = 0.0;
    for (long long c = cmin; c <= cmax; c++) best = std::max(best, fill(c));
    long long chunks = cmin;
    while (chunks < cmax && fill(chunks) < best - 0.005) chunks++;
    const int chunk_len = ceil_div(n, (int)chunks);
    const int nchunks = ceil_div(n, chunk_len);
    auto grid = [&](auto kernel, int threads, size_t smem, int items) {
        if (smem)
            cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        return std::min(items, sms * std::max(1, per_sm));
    };
    // shells have the row kernel only (262,144: 38.4 by tiles / 34.6 ms)
    if (!shell && fill(chunks) >= kD32TileFill) {
        const auto k = eps2 > 0.f ? k_direct_fp32<false> : k_direct_fp32<true>;
        const int items = tiles * nchunks;
        k<<<grid(k, kD32Threads, kD32Smem, items), kD32Threads, kD32Smem, st>>>(
            n, sbody, eps2, items, nchunks, chunk_len, ctr, part, counter);
    } else {
        const auto k = eps2 > 0.f
                           ? (shell ? k_direct_fp32_rows<true, false> : k_direct_fp32_rows<false, false>)
                           : (shell ? k_direct_fp32_rows<true, true> : k_direct_fp32_rows<false, true>);
        const int items = ceil_div(n, kRowTargets) * nchunks;
        k_direct_ref<<<tiles, kD32Threads, 0, st>>>(n, sbody, ref);
        k<<<grid(k, kRowThreads, 0, items), kRowThreads, 0, st>>>(
            n, sbody, srad, eps2, ref, items, nchunks, chunk_len, ctr, part, counter);
    }
    k_direct_reduce<<<ceil_div(n, 256), 256, 0, st>>>(n, nchunks, part, sidx, ax, ay, az);
}

}  // namespace nb
