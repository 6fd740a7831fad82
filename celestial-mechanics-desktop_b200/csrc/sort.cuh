// sort.cuh - stable one-sweep LSD radix sort of (uint64, uint32) pairs.
#pragma once
#include "common.cuh"

namespace nb {

void sort_init();
size_t sort_workspace_bytes(int capacity);
// Leading words of the workspace that a sort of n pairs counts in.
size_t sort_zero_words(int n, int sms);
// hist_ready: those words were zeroed and the 8x256 histograms at their head
// then filled by the kernel that made the keys.
// Returns the first failing status of the call's own memsets and launches.
// dn: optional device count replacing n when smaller (launches sized for n).
cudaError_t sort_pairs(cudaStream_t st, int n, uint64_t* k0, uint32_t* v0, uint64_t* k1,
                       uint32_t* v1, void* ws, bool hist_ready, int* err, int sms,
                       const int* dn = nullptr);

}  // namespace nb
