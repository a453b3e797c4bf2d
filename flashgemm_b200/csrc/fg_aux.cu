// Bandwidth-bound helper kernels around the GEMM stages: the FP32 -> TF32
// hi/lo split that feeds 3xTF32 stages, and the INT8 weight preparation that
// carries the reference's tail-row behaviour into the tensor-core path.
#include <cuda_runtime.h>

#include "fg_kernels.h"

namespace fg {

__device__ __forceinline__ float tf32_rne(float f)
{
    uint32_t u = __float_as_uint(f);
    if ((u & 0x7f800000u) == 0x7f800000u) return f;
    u += 0xfffu + ((u >> 13) & 1u);
    return __uint_as_float(u & 0xffffe000u);
}

// Whether a matrix is split by 16-byte accesses; one of dense rows is one long row.
__host__ __device__ __forceinline__ bool split_flat(const SplitJob &j) { return j.ld_in == j.cols && j.ld_out == j.cols; }
__host__ __device__ __forceinline__ bool split_vec(const SplitJob &j)
{
    return (split_flat(j) ? (j.rows * j.cols) % 4 == 0 : ((j.cols | j.ld_in | j.ld_out) & 3) == 0) &&
           (((uintptr_t)j.in | (uintptr_t)j.hi | (uintptr_t)j.lo) & 15) == 0;
}

// x = hi + lo + r with hi = rne_tf32(x), lo = rne_tf32(x - hi), |r| <= 2^-22 |x|.
// Block `part` of `parts` of one matrix. Bound by memory (4 bytes in, 8 out): four accesses
// in flight per thread, of 16 bytes where rows and pointers allow it. Measured (B200): the
// weights and B of 24 grouped FP32 chains, two launches, 73 -> 44 us against one value and one
// 64-bit division per thread and step; a GEMM of 17789 x 252 x 1429 (4-byte accesses) 203 ->
// 168 against one of them in flight. MIXED: some matrix of the launch needs 4-byte accesses
// (together the two loops take more registers, and 3 % of the time, than the one).
template <bool MIXED>
__device__ __forceinline__ void split_rows(const SplitJob &j, long part, long parts)
{
    const bool flat = split_flat(j);
    const long cols = flat ? j.rows * j.cols : j.cols;
    constexpr int U = 4;  // accesses in flight
    if (MIXED && !split_vec(j)) {
        const long total = j.rows * j.cols, step = parts * blockDim.x * U;
        for (long i0 = part * blockDim.x * U + threadIdx.x; i0 < total; i0 += step) {
            float x[U];
            long to[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const long i = i0 + u * (long)blockDim.x;
                to[u] = -1;
                if (i < total) {
                    const long r = total >> 32 ? i / j.cols : (uint32_t)i / (uint32_t)j.cols;
                    const long c = i - r * j.cols;
                    to[u] = r * j.ld_out + c;
                    x[u] = j.in[r * j.ld_in + c];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (to[u] < 0) continue;
                const float h = tf32_rne(x[u]);
                j.hi[to[u]] = h;
                j.lo[to[u]] = tf32_rne(x[u] - h);
            }
        }
        return;
    }
    const long row_quads = cols / 4, total = flat ? row_quads : row_quads * j.rows;
    const long step = parts * blockDim.x * U;
    for (long i0 = part * blockDim.x * U + threadIdx.x; i0 < total; i0 += step) {
        float4 x[U];
        long to[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const long i = i0 + u * (long)blockDim.x;
            to[u] = -1;
            if (i < total) {
                long from = i * 4;
                to[u] = from;
                if (!flat) {
                    const long r = total >> 32 ? i / row_quads : (uint32_t)i / (uint32_t)row_quads;
                    const long c = (i - r * row_quads) * 4;
                    from = r * j.ld_in + c;
                    to[u] = r * j.ld_out + c;
                }
                x[u] = *reinterpret_cast<const float4 *>(j.in + from);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (to[u] < 0) continue;
            float4 h, l;
            h.x = tf32_rne(x[u].x); l.x = tf32_rne(x[u].x - h.x);
            h.y = tf32_rne(x[u].y); l.y = tf32_rne(x[u].y - h.y);
            h.z = tf32_rne(x[u].z); l.z = tf32_rne(x[u].z - h.z);
            h.w = tf32_rne(x[u].w); l.w = tf32_rne(x[u].w - h.w);
            *reinterpret_cast<float4 *>(j.hi + to[u]) = h;
            *reinterpret_cast<float4 *>(j.lo + to[u]) = l;
        }
    }
}

// A few matrices in one launch, blockIdx.y = job, the jobs in the parameters or in
// device memory.
template <bool MIXED>
__global__ void __launch_bounds__(256) split_tf32_kernel(const __grid_constant__ SplitBatch b)
{
    overlap_next();
    overlap_wait();
    split_rows<MIXED>(b.job[blockIdx.y], blockIdx.x, gridDim.x);
}
template <bool MIXED>
__global__ void __launch_bounds__(256) split_tf32_jobs_kernel(const SplitJob *__restrict__ jobs)
{
    const SplitJob j = jobs[blockIdx.y];
    split_rows<MIXED>(j, blockIdx.x, gridDim.x);
}

void SplitSize::add(const SplitJob &j)
{
    const bool vec = split_vec(j);
    const long per_block = vec ? 4096 : 1024;
    const long n = (j.rows * j.cols + per_block - 1) / per_block;
    blocks = n > blocks ? n : blocks;
    mixed = mixed || !vec;
}

// Blocks per matrix of a launch: what the largest takes, at most 8 per SM.
static unsigned split_grid(const SplitSize &z) { return (unsigned)(z.blocks < 148 * 8 ? z.blocks : 148 * 8); }

cudaError_t launch_split_tf32(const SplitBatch &b, cudaStream_t s)
{
    SplitSize z;
    for (int i = 0; i < b.n; ++i) z.add(b.job[i]);
    if (z.blocks < 1) return cudaSuccess;
    return launch_overlapped(z.mixed ? split_tf32_kernel<true> : split_tf32_kernel<false>,
                             dim3(split_grid(z), (unsigned)b.n), 256, 0, s, b);
}

cudaError_t launch_split_tf32_jobs(const SplitJob *jobs_dev, int njobs, const SplitSize &z, cudaStream_t s)
{
    if (njobs < 1 || z.blocks < 1) return cudaSuccess;
    if (njobs > 65535) return cudaErrorInvalidValue;
    const dim3 grid(split_grid(z), (unsigned)njobs);
    if (z.mixed)
        split_tf32_jobs_kernel<true><<<grid, 256, 0, s>>>(jobs_dev);
    else
        split_tf32_jobs_kernel<false><<<grid, 256, 0, s>>>(jobs_dev);
    return cudaGetLastError();
}

// Rows m in [tail_lo, tail_hi) of the reference's INT8 chain meet activation
// k-quad max(s-1, 0) with weight k-quad s (multigemm/src/kernel_int8.h:405 vs
// :427, :590 vs :608). The prepared copy shifts those rows left by one quad,
// so a plain MMA yields sum_{s>=1} A_q(s) X_q(s-1); the missing A_q(0) X_q(0)
// term is added by the GEMM epilogue from the first quad kept at [K, K + 4).
// Other rows are copied unchanged; columns [K, ld_out) of them are zero.
// One thread writes 16 bytes (ld_out is a multiple of 16).
__global__ void prep_int8_weights_kernel(const int8_t *__restrict__ src, long ld_in,
                                         uint8_t *__restrict__ dst, long ld_out, long M, long K,
                                         long tail_lo, long tail_hi)
{
    const long per_row = ld_out / 16;
    const long total = M * per_row;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        const long m = i / per_row, k0 = (i - m * per_row) * 16;
        const uint8_t *row = reinterpret_cast<const uint8_t *>(src) + m * ld_in;
        const bool tail = (m >= tail_lo && m < tail_hi);
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t word = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const long k = k0 + 4 * q + b;
                uint8_t v = 0;
                if (tail) {
                    if (k < K - 4)
                        v = row[k + 4];
                    else if (k >= K && k < K + 4)
                        v = row[k - K];
                } else if (k < K) {
                    v = row[k];
                }
                word |= (uint32_t)v << (8 * b);
            }
            w[q] = word;
        }
        *reinterpret_cast<uint4 *>(dst + m * ld_out + k0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

cudaError_t launch_prep_int8_weights(const int8_t *src, long ld_in, uint8_t *dst, long ld_out,
                                     long M, long K, long tail_lo, long tail_hi, cudaStream_t s)
{
    if (M <= 0) return cudaSuccess;
    if (ld_out % 16) return cudaErrorInvalidValue;
    const long total = M * (ld_out / 16);
    long blocks = (total + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    prep_int8_weights_kernel<<<(unsigned)blocks, 256, 0, s>>>(src, ld_in, dst, ld_out, M, K,
                                                               tail_lo, tail_hi);
    return cudaGetLastError();
}

// Several preparations in one launch (blockIdx.y = job).
__global__ void prep_int8_jobs_kernel(const __grid_constant__ PrepJobs jobs)
{
    overlap_next();
    overlap_wait();
    const PrepJob &j = jobs.job[blockIdx.y];
    const long per_row = j.ld_out / 16;
    const long total = j.M * per_row;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total;
         i += (long)gridDim.x * blockDim.x) {
        const long m = i / per_row, k0 = (i - m * per_row) * 16;
        const uint8_t *row = reinterpret_cast<const uint8_t *>(j.src) + m * j.ld_in;
        const bool tail = (m >= j.tail_lo && m < j.tail_hi);
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t word = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const long k = k0 + 4 * q + b;
                uint8_t v = 0;
                if (tail) {
                    if (k < j.K - 4)
                        v = row[k + 4];
                    else if (k >= j.K && k < j.K + 4)
                        v = row[k - j.K];
                } else if (k < j.K) {
                    v = row[k];
                }
                word |= (uint32_t)v << (8 * b);
            }
            w[q] = word;
        }
        *reinterpret_cast<uint4 *>(j.dst + m * j.ld_out + k0) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

cudaError_t launch_prep_int8_jobs(const PrepJobs &jobs, cudaStream_t s)
{
    if (jobs.n <= 0) return cudaSuccess;
    long most = 0;
    for (int i = 0; i < jobs.n; ++i) {
        if (jobs.job[i].ld_out % 16) return cudaErrorInvalidValue;
        const long t = jobs.job[i].M * (jobs.job[i].ld_out / 16);
        most = t > most ? t : most;
    }
    long blocks = (most + 255) / 256;
    if (blocks > 148 * 4) blocks = 148 * 4;
    if (blocks < 1) blocks = 1;
    return launch_overlapped(prep_int8_jobs_kernel, dim3((unsigned)blocks, jobs.n), 256, 0, s, jobs);
}

__global__ void fill_u32_kernel(uint32_t *dst, size_t count, uint32_t value)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count;
         i += (size_t)gridDim.x * blockDim.x)
        dst[i] = value;
}

cudaError_t launch_fill_u32(uint32_t *dst, size_t count, uint32_t value, cudaStream_t s)
{
    if (count == 0) return cudaSuccess;
    size_t blocks = (count + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    fill_u32_kernel<<<(unsigned)blocks, 256, 0, s>>>(dst, count, value);
    return cudaGetLastError();
}

}  // namespace fg
