// direct.cuh - softened O(n^2) direct sums.
#pragma once
#include "common.cuh"

namespace nb {

// Rounding and summation orders of the desktop app's CPU backends.
enum DirectOrder { kOrderParallel = 0, kOrderSimd = 1, kOrderPairwise = 2 };

// Kernel attributes, once per device before the first call.
void direct_init();
// Rows in caller order; acc[c] receives every row's acceleration (0 for an
// inactive row).  close: v += dt_close/2 a follows, and open: v += dt_open/2 a,
// x' = x + dt_open v after it, x' of every row to `next`, which must not be
// the arrays px, py, pz then.  err: a non-finite active position or mass sets
// kErrNonFinite.
struct Fp64Args {
    int n;
    const double *px, *py, *pz, *m, *rad;  // rad: with the shell theorem only
    const uint8_t* act;
    double eps2;
    double* acc[3];
    int* err;
    bool close, open;
    double dt_close, dt_open;
    double* vel[3];
    double* next[3];
};
// FP64 sums, bit-identical to the CPU backend `order` names
// (CpuParallelBackend, SimdSingleThreadBackend / the native engine's CPU
// brute force, CpuSingleThreadBackend).  Returns the launch's status.
cudaError_t direct_fp64(cudaStream_t st, const Fp64Args& a, bool shell, int order, int sms);
// `steps` velocity-Verlet steps, step k with dts[k % n_dt], on the position
// arrays pos[0] with pos[1] as the other buffer; one kernel per step.  The
// state ends in pos[0], vel and acc, which must hold the accelerations at the
// start.
cudaError_t direct_fp64_steps(cudaStream_t st, Fp64Args a, bool shell, int order, int sms,
                              double* const pos[2][3], const double* dts, int n_dt, int steps);
// FP32 pair math over the n sorted (active) bodies; writes rows sidx[k].
// part: device memory of tree_bytes(capacity) for the chunks' FP64 partial
// sums; ref: n / 2560 + 1 reference points; ctr: a work-queue counter, 0 before
// the call.
void direct_fp32(cudaStream_t st, int n, const double4* sbody, const float* srad,
                 const uint32_t* sidx, double eps, bool shell, double* ax, double* ay,
                 double* az, unsigned long long* counter, double* part, double4* ref, int capacity,
                 unsigned* ctr, int sms);

}  // namespace nb
