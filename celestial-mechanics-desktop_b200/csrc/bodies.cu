// bodies.cu - per-body kernels of the step.
#include "bodies.cuh"

#include <algorithm>

namespace nb {

// One row's half kick and drift, SoAVerletIntegrator.Step phases 1-2
// (SoAVerletIntegrator.cs:70-88): FP64, explicit round-to-nearest operations,
// v += (dt/2) a, x += dt v, exactly as the reference rounds them.
__device__ __forceinline__ void kick_drift_row(const State& s, int i, double dt, double& x,
                                               double& y, double& z) {
    const double half = 0.5 * dt;
    const double vx = __dadd_rn(s.vx[i], __dmul_rn(half, s.ax[i]));
    const double vy = __dadd_rn(s.vy[i], __dmul_rn(half, s.ay[i]));
    const double vz = __dadd_rn(s.vz[i], __dmul_rn(half, s.az[i]));
    x = __dadd_rn(x, __dmul_rn(dt, vx));
    y = __dadd_rn(y, __dmul_rn(dt, vy));
    z = __dadd_rn(z, __dmul_rn(dt, vz));
    s.vx[i] = vx; s.vy[i] = vy; s.vz[i] = vz;
    s.px[i] = x; s.py[i] = y; s.pz[i] = z;
}

__global__ void k_kick_drift(int n, State s, double dt, int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !s.active[i]) return;
    double x = s.px[i], y = s.py[i], z = s.pz[i];
    kick_drift_row(s, i, dt, x, y, z);
    if (!isfinite(x) || !isfinite(y) || !isfinite(z) || !isfinite(s.mass[i]))
        dev_flag(err, kErrNonFinite);
}

// The cube around the box of the words `ord` (gpu_tree.cu:163-167 /
// octree_builder.cpp:29-35).
__device__ void cube_of_box(const unsigned long long* ord, double* cube) {
    double mn[3], mx[3];
    for (int k = 0; k < 3; k++) {
        mn[k] = ord_to_dbl(ord[k]);
        mx[k] = ord_to_dbl(ord[3 + k]);
    }
    double cx = __dmul_rn(__dadd_rn(mn[0], mx[0]), 0.5);
    double cy = __dmul_rn(__dadd_rn(mn[1], mx[1]), 0.5);
    double cz = __dmul_rn(__dadd_rn(mn[2], mx[2]), 0.5);
    double e = fmax(fmax(__dsub_rn(mx[0], mn[0]), __dsub_rn(mx[1], mn[1])), __dsub_rn(mx[2], mn[2]));
    double h = fmax(__dmul_rn(e, 0.5), 1e-10);
    h = __dmul_rn(h, 1.001);
    cube[0] = cx; cube[1] = cy; cube[2] = cz; cube[3] = h;
}

constexpr int kBoxThreads = 256;
constexpr int kBoxBlocks = kSMs * 8;
constexpr int kBoxVals = 8;  // min xyz, max xyz, active rows, 0

// Half kick + drift fused with the bounding box of the active bodies
// (BarnesHutBackend.cs:150-170; replaces reduction_kernel.cu:68-132 + the host
// finish of gpu_tree.cu:207-259, so no host sync): a grid-stride pass over a
// few resident waves of blocks; each leaves its box and count in `part`, and
// the last block to end folds them and derives the cube, so the pass needs no
// word initialised and no kernel behind it for the cube.  It also zeroes the
// words that the sort, the tree and the walk count in, which were ten memsets
// of some 2 us each in front of their kernels.
__global__ void __launch_bounds__(kBoxThreads)
k_kick_drift_bbox(int n, State s, int kick, double dt, BoxBufs box, ZeroWords zero, int* err,
                  const int* dn) {
    __shared__ double sh[kBoxVals][kBoxThreads / 32];
    __shared__ bool s_last;
    pdl_enter();
    n = dev_rows(n, dn);
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < zero.words;
         t += (size_t)gridDim.x * blockDim.x)
        zero.range[t] = 0;
    if (blockIdx.x == 0 && threadIdx.x < 12 && zero.w[threadIdx.x]) *zero.w[threadIdx.x] = 0;
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    double lo[3] = {inf, inf, inf}, hi[3] = {-inf, -inf, -inf}, act = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (!s.active[i]) continue;
        double x = s.px[i], y = s.py[i], z = s.pz[i];
        if (kick) kick_drift_row(s, i, dt, x, y, z);
        if (!isfinite(x) || !isfinite(y) || !isfinite(z) || !isfinite(s.mass[i]))
            dev_flag(err, kErrNonFinite);
        lo[0] = fmin(lo[0], x); hi[0] = fmax(hi[0], x);
        lo[1] = fmin(lo[1], y); hi[1] = fmax(hi[1], y);
        lo[2] = fmin(lo[2], z); hi[2] = fmax(hi[2], z);
        act += 1.0;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // value k of the block's 8: lane 0 of every warp, then thread k over the warps
    auto fold = [&]() -> double {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            lo[k] = warp_min(lo[k]);
            hi[k] = warp_max(hi[k]);
        }
        act = warp_sum(act);
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                sh[k][warp] = lo[k];
                sh[3 + k][warp] = hi[k];
            }
            sh[6][warp] = act;
            sh[7][warp] = 0.0;
        }
        __syncthreads();
        double v = 0.0;
        if (threadIdx.x < kBoxVals) {
            const int k = threadIdx.x;
            v = sh[k][0];
            for (int w = 1; w < kBoxThreads / 32; w++)
                v = k < 3 ? fmin(v, sh[k][w]) : k < 6 ? fmax(v, sh[k][w]) : v + sh[k][w];
        }
        return v;
    };
    const double mine = fold();
    if (threadIdx.x < kBoxVals) {
        box.part[blockIdx.x * kBoxVals + threadIdx.x] = mine;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(box.ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int k = 0; k < 3; k++) {
        lo[k] = inf;
        hi[k] = -inf;
    }
    act = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kBoxThreads) {
        const double* p = box.part + b * kBoxVals;
        for (int k = 0; k < 3; k++) {
            lo[k] = fmin(lo[k], __ldcg(p + k));
            hi[k] = fmax(hi[k], __ldcg(p + 3 + k));
        }
        act += __ldcg(p + 6);
    }
    const double all = fold();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x;
        // no active row (or a value out of range): the empty box's words
        const bool some = k < 3 ? all < 1.0e308 : all > -1.0e308;
        box.ord[k] = some ? dbl_to_ord(all) : (k < 3 ? ~0ull : 0ull);
    }
    if (threadIdx.x == 6) *box.n_active = (int)all;
    __syncthreads();
    if (threadIdx.x == 0 && box.cube) cube_of_box(box.ord, box.cube);
}

// Phases 4-5 (SoAVerletIntegrator.cs:95-116): v += (dt/2) a for active rows;
// the acceleration buffer itself is the next step's "old" acceleration.
__global__ void k_kick(int n, State s, double dt, const int* dn) {
    pdl_enter();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= dev_rows(n, dn) || !s.active[i]) return;
    const double half = 0.5 * dt;
    s.vx[i] = __dadd_rn(s.vx[i], __dmul_rn(half, s.ax[i]));
    s.vy[i] = __dadd_rn(s.vy[i], __dmul_rn(half, s.ay[i]));
    s.vz[i] = __dadd_rn(s.vz[i], __dmul_rn(half, s.az[i]));
}

__global__ void k_cube(const double* given, double* cube) {
    if (threadIdx.x < 4) cube[threadIdx.x] = given[threadIdx.x];
}

__device__ __forceinline__ uint64_t quant_cube(double p, double lo, double inv2h) {
    double u = __dmul_rn(__dsub_rn(p, lo), inv2h);
    u = fmax(0.0, fmin(1.0, u));
    uint64_t q = (uint64_t)__dmul_rn(u, 2097152.0);
    return q > 2097151ull ? 2097151ull : q;
}

constexpr int kKeyThreads = 256;

// Cube-mode keys of ITEMS keys per thread, plus the digit histograms of
// all 8 sort passes; a block folds its keys into shared bins and adds the
// non-zero bins to the global counts.  8 keys per thread (2048 per block)
// make the fewest global atomics per key; with fewer bodies than make a block
// per SM that way the kernel is latency, and 2 or 1 keys per thread spread it
// (262,144 bodies: the call's sort stage 124 us with 8, 119 with 2).
// With `rows`, every row's (x, y, z, m) is also written there in row order,
// and with `amag` its |a| (the acceleration buffer still holds the previous
// step's), so the gather after the sort reads one 32-byte record and one
// word per body instead of seven scattered 8-byte fields.
template <int ITEMS>
__global__ void __launch_bounds__(kKeyThreads)
k_keys_cube(int n, State s, const double* __restrict__ cube, uint64_t* __restrict__ keys,
            uint32_t* __restrict__ vals, uint32_t* __restrict__ hist, double4* __restrict__ rows,
            float* __restrict__ amag, int zero_acc, const int* dn) {
    __shared__ uint32_t sh[8][256];
    pdl_enter();
    n = dev_rows(n, dn);
    for (int t = threadIdx.x; t < 8 * 256; t += blockDim.x) (&sh[0][0])[t] = 0;
    __syncthreads();
    const double h = cube[3];
    const double inv2h = 1.0 / __dmul_rn(2.0, h);
    const double lx = __dsub_rn(cube[0], h), ly = __dsub_rn(cube[1], h), lz = __dsub_rn(cube[2], h);
#pragma unroll 1
    for (int k = 0; k < ITEMS; k++) {
        const int i = (blockIdx.x * ITEMS + k) * kKeyThreads + threadIdx.x;
        uint64_t key = kInactiveKey;
        if (i < n) {
            const double x = s.px[i], y = s.py[i], z = s.pz[i];
            const bool active = s.active[i];
            if (active)
                key = (spread21(quant_cube(x, lx, inv2h)) << 2) |
                      (spread21(quant_cube(y, ly, inv2h)) << 1) | spread21(quant_cube(z, lz, inv2h));
            keys[i] = key;
            vals[i] = (uint32_t)i;
            if (rows) rows[i] = make_double4(x, y, z, s.mass[i]);
            if (amag) {
                const double ax = s.ax[i], ay = s.ay[i], az = s.az[i];
                amag[i] = (float)sqrt(ax * ax + ay * ay + az * az);
            }
            if (zero_acc && !active) s.ax[i] = s.ay[i] = s.az[i] = 0.0;
        }
        // plain shared atomics: measured faster than warp-aggregating the
        // digits with match_any (whose issue cost exceeds the serialisation
        // of the few same-bin lanes of a clustered system's high digits)
        if (i < n) {
#pragma unroll
            for (int p = 0; p < 8; p++) atomicAdd(&sh[p][(uint32_t)(key >> (8 * p)) & 0xFF], 1u);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 8 * 256; t += blockDim.x) {
        uint32_t v = (&sh[0][0])[t];
        if (v) atomicAdd(&hist[t], v);
    }
}

// morton_code_kernel semantics (morton_kernel.cu:11-45 with the inverse
// ranges of launch_morton_codes, :57-64) and morton_from_unit
// (morton.hpp:29-35).
__global__ void k_keys_aabb(int n, State s, const unsigned long long* __restrict__ bbox_ord,
                            uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    vals[i] = (uint32_t)i;
    if (!s.active[i]) {
        keys[i] = kInactiveKey;
        return;
    }
    double mn[3], r[3], inv[3];
    for (int k = 0; k < 3; k++) {
        mn[k] = ord_to_dbl(bbox_ord[k]);
        r[k] = __dsub_rn(ord_to_dbl(bbox_ord[3 + k]), mn[k]);
        inv[k] = (r[k] > 1e-30) ? 1.0 / r[k] : 0.0;
    }
    const double p[3] = {s.px[i], s.py[i], s.pz[i]};
    uint64_t q[3];
    for (int k = 0; k < 3; k++) {
        double u = __dmul_rn(__dsub_rn(p[k], mn[k]), inv[k]);
        u = fmax(0.0, fmin(1.0, u));
        q[k] = (uint64_t)__dmul_rn(u, 2097151.0);
    }
    keys[i] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
}

__global__ void k_gather(int n, State s, const uint32_t* __restrict__ sidx,
                         double4* __restrict__ sbody, float* __restrict__ srad,
                         float* __restrict__ samag, const double4* __restrict__ rows,
                         const float* __restrict__ amag, const int* dn) {
    pdl_enter();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= dev_rows(n, dn)) return;
    const uint32_t i = sidx[k];
    if (rows) {
        sbody[k] = rows[i];
        if (srad) srad[k] = s.radius ? (float)s.radius[i] : 0.f;
        if (samag) samag[k] = amag[i];
        return;
    }
    sbody[k] = make_double4(s.px[i], s.py[i], s.pz[i], s.mass[i]);
    if (srad) srad[k] = s.radius ? (float)s.radius[i] : 0.f;
    if (samag) {  // |a| of the previous step (acceleration buffer before it is overwritten)
        const double ax = s.ax[i], ay = s.ay[i], az = s.az[i];
        samag[k] = (float)sqrt(ax * ax + ay * ay + az * az);
    }
}

size_t box_part_bytes() { return sizeof(double) * kBoxVals * kBoxBlocks; }

void launch_kick_drift_bbox(cudaStream_t st, int n, State s, bool kick, double dt,
                            const BoxBufs& box, const ZeroWords& zero, int* err, const int* dn) {
    launch_pdl(n, k_kick_drift_bbox, std::max(1, std::min(ceil_div(n, kBoxThreads), kBoxBlocks)),
               kBoxThreads, 0, st, n, s, kick ? 1 : 0, dt, box, zero, err, dn);
}

void launch_kick_drift(cudaStream_t st, int n, State s, double dt, int* err) {
    if (n > 0) k_kick_drift<<<ceil_div(n, 256), 256, 0, st>>>(n, s, dt, err);
}

void launch_kick(cudaStream_t st, int n, State s, double dt, const int* dn) {
    if (n > 0) launch_pdl(n, k_kick, ceil_div(n, 256), 256, 0, st, n, s, dt, dn);
}

void launch_cube(cudaStream_t st, const double* given, double* cube) {
    k_cube<<<1, 32, 0, st>>>(given, cube);
}

void launch_keys_cube(cudaStream_t st, int n, const State& s, const double* cube,
                      uint64_t* keys, uint32_t* vals, uint32_t* hist, double4* rows,
                      float* amag, bool zero_acc, const int* dn) {
    if (n <= 0) return;
    auto go = [&](auto kernel, int items) {
        launch_pdl(n, kernel, ceil_div(n, kKeyThreads * items), kKeyThreads, 0, st, n, s, cube, keys,
                   vals, hist, rows, amag, zero_acc ? 1 : 0, dn);
    };
    if (n > 8 * kSMs * kKeyThreads) go(k_keys_cube<8>, 8);
    else if (n > kSMs * kKeyThreads) go(k_keys_cube<2>, 2);
    else go(k_keys_cube<1>, 1);
}

void launch_keys_aabb(cudaStream_t st, int n, const State& s,
                      const unsigned long long* bbox_ord, uint64_t* keys, uint32_t* vals) {
    if (n > 0) k_keys_aabb<<<ceil_div(n, 256), 256, 0, st>>>(n, s, bbox_ord, keys, vals);
}

void launch_gather(cudaStream_t st, int n, const State& s, const uint32_t* sidx,
                   double4* sbody, float* srad, float* samag, const double4* rows,
                   const float* amag, const int* dn) {
    if (n > 0)
        launch_pdl(n, k_gather, ceil_div(n, 256), 256, 0, st, n, s, sidx, sbody, srad, samag, rows,
                   amag, dn);
}

}  // namespace nb
