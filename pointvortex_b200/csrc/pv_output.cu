// pv_output.cu — the reference's text output at GPU rates: trajectory rows
// (TrajectoryWriter::write, src/print.cpp:29-40) and the vortex block of a checkpoint
// (writeCheckpoint, src/checkpoint.cpp:86-88), byte for byte as the reference's
// `std::ostream << std::setprecision(17)` writes them.
//
// Three launches per frame:
//   1. format_rows_kernel: one thread per vortex formats its row (pv_format.cuh: exact 17-digit %g
//      conversion) into shared memory, at a stride of an odd number of words, so that a warp's
//      byte stores meet no bank twice; the block scans its rows' lengths and writes its text
//      without gaps, neighbouring lanes on neighbouring bytes, into its slot of the staging;
//   2. scan_blocks_kernel: one block turns the blocks' lengths into exclusive offsets and the
//      frame's total;
//   3. gather_rows_kernel: each block moves its text to its place, by words: a word of the output is
//      cut from two of the staging.
// The frame then crosses to the host in one copy of exactly its size.
#include "pv_format.cuh"
#include "pv_internal.h"
#include "pvb200.h"

namespace pvb {

namespace {

constexpr int kRowThreads = kFormatRows;
constexpr int kRowWords = PV_TRAJECTORY_ROW_MAX / 4 | 1;  // shared memory per row
static_assert(PV_CHECKPOINT_ROW_MAX <= PV_TRAJECTORY_ROW_MAX && PV_CHECKPOINT_ROW_MAX % 4 == 0 &&
                  kRowThreads % 32 == 0,
              "a block's slot of the staging is whole words");

__device__ __forceinline__ int put(char *o, const char *s, int n) {
    for (int i = 0; i < n; ++i)
        o[i] = s[i];
    return n;
}

__device__ __forceinline__ int put_value(char *o, double v, char end) {
    const int n = fmt::format_g17(v, o);
    o[n] = end;
    return n + 1;
}

__global__ void __launch_bounds__(kRowThreads)
    format_rows_kernel(RowFormat f, char *__restrict__ staging,
                       unsigned long long *__restrict__ block_sums) {
    __shared__ uint32_t rows[kRowThreads * kRowWords];
    __shared__ uint32_t starts[kRowThreads];
    __shared__ uint32_t warp_sums[kRowThreads / 32];
    const size_t i = static_cast<size_t>(blockIdx.x) * kRowThreads + threadIdx.x;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t len = 0;
    if (i < f.n) {
        char *o = reinterpret_cast<char *>(rows + threadIdx.x * kRowWords);
        const bool trajectory = f.kind == ROWS_TRAJECTORY;
        const char sep = trajectory ? ',' : ' ';
        int p = 0;
        if (trajectory) {  // time,frame,index,x,y,circulation,u,v
            p = put(o, f.prefix, f.prefix_len);
            p += fmt::format_u64(i, o + p);
            o[p++] = ',';
        }
        // x y circulation, and the trajectory's u v: one copy of the conversion's code
        const double *columns[5] = {f.x, f.y, f.g, f.u, f.v};
        const int count = trajectory ? 5 : 3;
#pragma unroll 1
        for (int c = 0; c < count; ++c)
            p += put_value(o + p, columns[c][i], c + 1 < count ? sep : '\n');
        len = static_cast<uint32_t>(p);
    }
    uint32_t at = len;  // inclusive scan of the lengths
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t below = __shfl_up_sync(0xffffffffu, at, d);
        at += lane >= static_cast<unsigned>(d) ? below : 0;
    }
    if (lane == 31)
        warp_sums[warp] = at;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (unsigned w = 0; w < kRowThreads / 32; ++w) {
        before += w < warp ? warp_sums[w] : 0;
        total += warp_sums[w];
    }
    starts[threadIdx.x] = before + at - len;
    if (threadIdx.x == 0)
        block_sums[blockIdx.x] = total;
    __syncwarp();
    char *dst = staging + static_cast<size_t>(blockIdx.x) * kRowThreads * f.stride;
    for (unsigned r = 0; r < 32; ++r) {
        const uint32_t n = __shfl_sync(0xffffffffu, len, r);
        const unsigned row = warp * 32 + r;
        const char *o = reinterpret_cast<const char *>(rows + row * kRowWords);
        for (uint32_t b = lane; b < n; b += 32)
            dst[starts[row] + b] = o[b];
    }
}

// Exclusive scan of the block sums in place (one block, chunks of 1024 with a running carry);
// block_sums[blocks] receives the total.
__global__ void __launch_bounds__(1024)
    scan_blocks_kernel(unsigned long long *block_sums, size_t blocks) {
    __shared__ unsigned long long buf[1024];
    __shared__ unsigned long long carry;
    if (threadIdx.x == 0)
        carry = 0;
    __syncthreads();
    for (size_t base = 0; base < blocks; base += 1024) {
        const size_t j = base + threadIdx.x;
        const unsigned long long v = j < blocks ? block_sums[j] : 0;
        buf[threadIdx.x] = v;
        __syncthreads();
        for (int d = 1; d < 1024; d <<= 1) {  // Hillis-Steele inclusive scan
            const unsigned long long add = threadIdx.x >= d ? buf[threadIdx.x - d] : 0;
            __syncthreads();
            buf[threadIdx.x] += add;
            __syncthreads();
        }
        if (j < blocks)
            block_sums[j] = carry + buf[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 1023)
            carry += buf[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        block_sums[blocks] = carry;
}

__global__ void __launch_bounds__(256)
    gather_rows_kernel(const char *__restrict__ staging,
                       const unsigned long long *__restrict__ block_offsets, int stride,
                       char *__restrict__ out) {
    const unsigned long long from = block_offsets[blockIdx.x];
    const uint32_t total = static_cast<uint32_t>(block_offsets[blockIdx.x + 1] - from);
    const char *text = staging + static_cast<size_t>(blockIdx.x) * kRowThreads * stride;
    const uint32_t *words = reinterpret_cast<const uint32_t *>(text);
    char *dst = out + from;
    const uint32_t head = min(static_cast<uint32_t>(-from & 3), total);  // bytes before a whole word
    const uint32_t count = (total - head) / 4;
    uint32_t *whole = reinterpret_cast<uint32_t *>(dst + head);
    for (uint32_t w = threadIdx.x; w < count; w += blockDim.x) {
        const uint32_t low = words[w];  // bytes 4w + head ... lie in words w and w + 1
        const uint32_t high = head ? words[w + 1] : 0;
        whole[w] = __funnelshift_r(low, high, 8 * head);
    }
    const uint32_t tail = head + 4 * count;
    if (threadIdx.x < head)
        dst[threadIdx.x] = text[threadIdx.x];
    if (threadIdx.x < total - tail)
        dst[tail + threadIdx.x] = text[tail + threadIdx.x];
}

}  // namespace

int format_prefix(double time, uint64_t frame, char *out) {
    int p = fmt::format_g17(time, out);
    out[p++] = ',';
    p += fmt::format_u64(frame, out + p);
    out[p++] = ',';
    return p;
}

cudaError_t launch_format_rows(const RowFormat &f, char *staging, unsigned long long *block_sums,
                               char *out, cudaStream_t stream) {
    const size_t blocks = (f.n + kRowThreads - 1) / kRowThreads;
    if (blocks == 0) {
        return cudaMemsetAsync(block_sums, 0, sizeof(unsigned long long), stream);
    }
    format_rows_kernel<<<static_cast<unsigned>(blocks), kRowThreads, 0, stream>>>(
        f, staging, block_sums);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    scan_blocks_kernel<<<1, 1024, 0, stream>>>(block_sums, blocks);
    if ((e = cudaGetLastError()) != cudaSuccess)
        return e;
    gather_rows_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(staging, block_sums, f.stride,
                                                                          out);
    return cudaGetLastError();
}

}  // namespace pvb
