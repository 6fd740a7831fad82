// hostio.cuh - copies between the caller's pageable arrays and the device.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace nb {

// One array of a transfer; `dst` / `src` is host or device memory by direction.
struct CopySeg {
    void* dst;
    const void* src;
    size_t bytes;
};

struct CopyPool;

// A handle's side of the transfers: a pinned buffer of its own for small ones
// (two halves, up and down, so a call may fill one while the other is read,
// and kHostExtra bytes for the handle's own use) and its share of the device's
// copy pool for large ones.
constexpr size_t kHostExtra = 4096;
struct HostIO {
    char* pin = nullptr;
    size_t half = 0;
    CopyPool* pool = nullptr;
    char* extra() const { return pin + 2 * half; }
};

// A handle's pinned half, at most; a small handle's holds its largest transfer.
// The forces of 20,011 bodies (0.66 MB up, 0.48 MB down) take 0.48 ms a call,
// with 256 KB 0.52 and with 1 MB 0.50.
constexpr size_t kHalfBytes = 512 << 10;
// For transfers of up to `rows` arrays of row_bytes each (rows 0: no pinned
// half).  Without pinned memory (half 0) every array takes the plain copy.
// False: no memory at all.
bool hostio_init(HostIO& io, int device, int rows, size_t row_bytes);
void hostio_free(HostIO& io);

// Host arrays to the device in stream order.  Pageable arrays may be changed on
// return, pinned ones when the stream has been synchronised.  An earlier upload through the same handle has to have ended.
cudaError_t copy_up(HostIO& io, cudaStream_t st, const CopySeg* seg, int n);

// Device arrays to the host.  start_down enqueues what fits the pinned half
// (adjacent rows in one copy) and reports in *queued whether everything did;
// after the stream has been synchronised finish_down puts the data into the
// host arrays, by the pool where start_down queued nothing.
cudaError_t start_down(HostIO& io, cudaStream_t st, const CopySeg* seg, int n, bool* queued);
cudaError_t finish_down(HostIO& io, cudaStream_t st, const CopySeg* seg, int n, bool queued);

}  // namespace nb
