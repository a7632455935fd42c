// rms_reduce.cu -- ordered sum of the per-warp accumulator rows.
//
// Each warp of a walk launch owns one FP64 row block (rms_walk_*.cu); the
// job's totals are their sum.  Column i is summed by one thread over a chunk of
// rows in slot order with eight interleaved partial sums (slot k goes to
// partial k % 8), then the partials are added in order, and the chunks' sums the
// same way: a fixed association, so a rerun with the same launch shape
// reproduces every bit.
// Replaces the contended FP64 CAS atomics of hpc_code/lib/main.cu:40-56.
//
// Bound by HBM (a gigabyte of rows).  One thread per column over all rows is
// 250 blocks for 1000 records of 64 columns, too few loads in flight (1.9 TB/s:
// 0.85 ms for 3125 rows); with the rows cut into chunks, eight blocks' worth
// per SM, 0.29 ms.  A chunk's sum goes where its first row lay (only its own
// thread reads that column there), so no second buffer is needed.
#include <cuda_runtime.h>

#include <algorithm>

#include "rms_internal.h"

namespace rms {
namespace {

// rows k * stride (k = blockIdx.y * per .. + per), summed into out + blockIdx.y * out_stride
__global__ void reduce_slots_kernel(const double* slots, int nslots, size_t stride, int per, size_t row, double* out,
                                    size_t out_stride) {
    const int s0 = blockIdx.y * per, s1 = min(nslots, s0 + per);
    out += (size_t)blockIdx.y * out_stride;
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < row; i += step) {
        double p[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        int k = s0;
        for (; k + 8 <= s1; k += 8) {
#pragma unroll
            for (int u = 0; u < 8; ++u) p[u] += __ldcs(slots + (size_t)(k + u) * stride + i);
        }
        for (int u = 0; k < s1; ++k, ++u) p[u] += __ldcs(slots + (size_t)k * stride + i);
        out[i] = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
    }
}

}  // namespace

int launch_reduce_slots(double* slots, int nslots, size_t row, double* out, void* stream) {
    if (row == 0) return 0;
    const int block = 256;
    const size_t gx = std::min<size_t>((row + block - 1) / block, 4096);
    // chunks of at least 16 rows, about eight blocks per SM in all
    const int chunks = (int)std::max<size_t>(1, std::min<size_t>(nslots / 16, (148 * 8 + gx - 1) / gx));
    const int per = (nslots + chunks - 1) / chunks, n = (nslots + per - 1) / per;
    if (n > 1) {
        const size_t first = (size_t)per * row;   // doubles from one chunk's first row to the next
        reduce_slots_kernel<<<dim3((unsigned)gx, (unsigned)n), block, 0, (cudaStream_t)stream>>>(slots, nslots, row, per,
                                                                                               row, slots, first);
        reduce_slots_kernel<<<(unsigned)gx, block, 0, (cudaStream_t)stream>>>(slots, n, first, n, row, out, 0);
    } else {
        reduce_slots_kernel<<<(unsigned)gx, block, 0, (cudaStream_t)stream>>>(slots, nslots, row, nslots, row, out, 0);
    }
    return (int)cudaGetLastError();
}

const char* cuda_error_string(int code) { return cudaGetErrorString((cudaError_t)code); }

}  // namespace rms
