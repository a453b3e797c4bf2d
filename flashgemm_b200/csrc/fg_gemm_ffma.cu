// Plain FP32 SGEMM on the CUDA cores: C = A * B, row-major.
//
// Each output is one FP32 fused multiply-add per k in increasing k, the
// arithmetic of the reference's vfmadd231ps register tiles
// (singlegemm/src/kernel.h:8, multigemm/src/kernel_f32.h:3), so results are
// bit-identical to the reference's. With kblock > 0 and K > kblock, K is cut
// into blocks of kblock: each block is summed from zero and then added into
// the result, as singlegemm's GEMM_K = 2048 blocking does
// (singlegemm/src/NN_mp.h:13 and its ADD_C step, singlegemm/src/kernel.h:384-400).
//
// One tile, in several shapes (the table kShapes says what each is for):
//
// * BM x BN outputs per CTA, TM x TN per thread. A thread's rows are ty + i * TY
//   and its columns tx * 4 + j * 4 * TX + {0..3}. The multiply-adds go in pairs
//   along n (fma.rn.f32x2: two IEEE round-to-nearest FMAs per instruction, each
//   exactly an fmaf), the A value of a pair duplicated in registers.
// * A stays row by row in shared memory (k contiguous), so a thread reads four k
//   of a row with one 16-byte load, any TM fits and no transpose is needed; B is
//   read four columns at a time. A's 16-byte chunks are swizzled over the rows:
//   the two or four consecutive rows that a warp reads fall on distinct banks.
// * k slices of BK come in through a ring of ST buffers filled by cp.async, one
//   barrier per slice; the fragments of k + 1 load while k computes.
//
// What bounds it is the FMA pipe and the instructions around it: on B200 a loop
// of nothing but f32x2 FMAs on registers issues 114 of the 128 FMA per clock and
// SM, and one that also reads its fragments from shared memory 83 (one warp per
// scheduler) to 100 (two). Measured alternatives that lost: A duplicated in shared
// memory instead of in registers (1.2-1.4x slower: twice the shared-memory
// reads), pairs along the diagonal (no faster), scalar FMAs (0.9x), registers
// between global and shared memory instead of cp.async (the kernel before this
// one). Before and now, us a call (B200): 1024^3 80 -> 58 (27 -> 37 TFLOP/s),
// 1632 x 36548 x 1024 2694 -> 2402 (51 TFLOP/s), 35 x 8457 x 2560 142 -> 77,
// 512 x 289 x 1024 66 -> 29, 4096^3 3580 -> 2566.
#include <cuda_runtime.h>

#include <cstdlib>
#include <mutex>

#include "fg_kernels.h"

namespace fg {

namespace {

__device__ __forceinline__ unsigned long long pack2(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}

__device__ __forceinline__ void unpack2(unsigned long long v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// d (two lanes) = a * b + d, each lane one round-to-nearest FMA
__device__ __forceinline__ void ffma2(unsigned long long &d, unsigned long long a,
                                      unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// E floats (4: one 16-byte copy, 1: one of 4 bytes) global -> shared, the last
// 4 * E - bytes of them zero
template <int E>
__device__ __forceinline__ void copy_async(uint32_t dst, const float *src, int bytes)
{
    if constexpr (E == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                     : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int BM_, int BN_, int BK_, int TM_, int TN_, int ST_, int OCC_>
struct Shape {
    static constexpr int BM = BM_, BN = BN_, BK = BK_, TM = TM_, TN = TN_, ST = ST_;
    static constexpr int OCC = OCC_;  // CTAs per SM: what the registers have to allow
    static constexpr int TX = BN / TN, TY = BM / TM, NT = TX * TY;
    static constexpr int STAGE = (BM + BN) * BK;  // floats per ring buffer
    static constexpr int SMEM = ST * STAGE * 4;
    static_assert(BM % TM == 0 && BN % TN == 0 && TN % 4 == 0, "whole fragments");
    static_assert(BK == 32, "a row of A's tile is one 128-byte line, its 8 chunks swizzled");
    static_assert(TX == 8 || TX == 16, "a warp holds 4 or 2 rows of column groups");
    static_assert(NT % BK == 0 && NT % (BN / 4) == 0, "copies: a thread's k chunk and column are its own");
};

// Where the 16-byte chunk c of row r lies in A's tile.
__device__ __forceinline__ int a_chunk(int r, int c) { return c ^ (r & 7); }

// One BM x BN output tile at (m0, n0). VA / VB: A / B has 16-byte-aligned rows and
// pointer, and comes in 16-byte copies; else in 4-byte ones. Rows past M read
// row M - 1 and columns past N read zeros (neither is stored).
template <class S, bool VA, bool VB>
__device__ __forceinline__ void ffma_tile(const FfmaArgs &p, int m0, int n0, float *sm)
{
    constexpr int BM = S::BM, BN = S::BN, BK = S::BK, TM = S::TM, TN = S::TN, ST = S::ST;
    constexpr int TX = S::TX, TY = S::TY, NT = S::NT;
    const int tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    const int M = p.M, N = p.N, K = p.K;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);

    // copies: A_C of EA floats per row of A, A_R rows per pass of the CTA; B alike
    // (a B row may take several passes: B_P copies per thread and row group)
    constexpr int EA = VA ? 4 : 1, EB = VB ? 4 : 1;
    constexpr int A_C = BK / EA, A_R = NT / A_C, A_V = (BM + A_R - 1) / A_R;
    constexpr int B_C = BN / EB, B_P = B_C > NT ? B_C / NT : 1, B_R = B_C > NT ? 1 : NT / B_C;
    constexpr int B_V = (BK + B_R - 1) / B_R;
    static_assert(NT % A_C == 0 && (NT % B_C == 0 || B_C % NT == 0), "whole passes");
    const int a_r = tid / A_C, a_c = tid % A_C;
    const int b_r = B_C > NT ? 0 : tid / B_C, b_c = tid % B_C;
    auto a_dst = [&](int r) {
        return sbase + (r * BK + a_chunk(r, a_c * EA / 4) * 4 + (EA == 4 ? 0 : a_c % 4)) * 4;
    };
    const uint32_t a_dst0 = a_dst(a_r);
    int b_bytes[B_P];
    const float *b_src[B_P];
    uint32_t b_dst[B_P];
#pragma unroll
    for (int q = 0; q < B_P; ++q) {
        const int c = (b_c + q * NT) * EB, gn = n0 + c;
        b_bytes[q] = 4 * min(max(N - gn, 0), EB);  // clamped first: 4 N may not fit in an int
        b_src[q] = p.B + (b_bytes[q] ? gn : 0) + (long)b_r * p.ldb;
        b_dst[q] = sbase + (BM * BK + b_r * BN + c) * 4;
    }
    auto load = [&](int slice, int buf) {
        const int k0 = slice * BK;
        const uint32_t off = buf * S::STAGE * 4;
        if (k0 + BK <= K) {
#pragma unroll
            for (int v = 0; v < A_V; ++v) {
                const int r = a_r + v * A_R;
                if (BM % A_R && r >= BM) break;
                // the swizzle repeats every 8 rows
                const uint32_t d = A_R % 8 == 0 ? a_dst0 + v * A_R * BK * 4 : a_dst(r);
                copy_async<EA>(d + off, p.A + (long)min(m0 + r, M - 1) * p.lda + k0 + a_c * EA, 4 * EA);
            }
#pragma unroll
            for (int q = 0; q < B_P; ++q) {
                const float *s = b_src[q] + (long)k0 * p.ldb;
#pragma unroll
                for (int v = 0; v < B_V; ++v) {
                    if (BK % B_R && b_r + v * B_R >= BK) break;
                    copy_async<EB>(b_dst[q] + off + v * B_R * BN * 4, s + (long)(v * B_R) * p.ldb,
                                   b_bytes[q]);
                }
            }
        } else {  // the last slice of a K that is no multiple of BK: zeros past K
#pragma unroll
            for (int v = 0; v < A_V; ++v) {
                const int r = a_r + v * A_R;
                if (BM % A_R && r >= BM) break;
                const int gk = k0 + a_c * EA;
                const int n = 4 * min(max(K - gk, 0), EA);
                copy_async<EA>(a_dst(r) + off, p.A + (long)min(m0 + r, M - 1) * p.lda + (n ? gk : 0), n);
            }
#pragma unroll
            for (int q = 0; q < B_P; ++q)
#pragma unroll
                for (int v = 0; v < B_V; ++v) {
                    const int r = b_r + v * B_R;
                    if (BK % B_R && r >= BK) break;
                    const bool in = k0 + r < K;
                    copy_async<EB>(b_dst[q] + off + v * B_R * BN * 4,
                                   in ? b_src[q] + (long)(k0 + v * B_R) * p.ldb : p.B,
                                   in ? b_bytes[q] : 0);
                }
        }
    };

    unsigned long long acc[TM][TN / 2];
    auto clear = [&] {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    };
    // the block's sums into C: stored, or added to the blocks before it
    const bool vec_c = p.ldc % 4 == 0 && ((uintptr_t)p.C & 15) == 0;
    auto flush = [&](bool add) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int gm = m0 + ty + i * TY;
            if (gm >= M) continue;
            float *c = p.C + (size_t)gm * p.ldc;
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) {
                const int gn = n0 + tx * 4 + j * 4 * TX;
                float r[4];
                unpack2(acc[i][2 * j], r[0], r[1]);
                unpack2(acc[i][2 * j + 1], r[2], r[3]);
                if (vec_c && gn + 3 < N) {
                    float4 *c4 = reinterpret_cast<float4 *>(c + gn);
                    if (add) {
                        const float4 o = *c4;
                        r[0] = o.x + r[0]; r[1] = o.y + r[1]; r[2] = o.z + r[2]; r[3] = o.w + r[3];
                    }
                    const float4 v = make_float4(r[0], r[1], r[2], r[3]);
                    if constexpr (TN == 8)  // past L1 (18720 x 30480 x 48 1401 -> 1335)
                        __stcg(c4, v);
                    else
                        *c4 = v;
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (gn + u < N) c[gn + u] = add ? c[gn + u] + r[u] : r[u];
                }
            }
        }
    };

    const int slices = (K + BK - 1) / BK;
    const int per_block = p.kblock > 0 && p.kblock < K ? p.kblock / BK : slices;
    clear();
    if (slices == 0) flush(false);  // an empty sum
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < slices) load(s, s);
        copy_commit();
    }
    int buf = 0, in_block = 0;
#pragma unroll 1
    for (int s = 0; s < slices; ++s) {
        copy_wait<ST - 2>();
        __syncthreads();  // slice s has landed; every thread has read slice s - 1
        if (s + ST - 1 < slices) load(s + ST - 1, buf == 0 ? ST - 1 : buf - 1);
        copy_commit();
        const float *As = sm + buf * S::STAGE, *Bs = As + BM * BK;
        auto a_quad = [&](int i, int q) {
            const int r = ty + i * TY;
            return *reinterpret_cast<const float4 *>(&As[r * BK + a_chunk(r, q) * 4]);
        };
        auto b_quad = [&](int k, int j) {
            return *reinterpret_cast<const float4 *>(&Bs[k * BN + tx * 4 + j * 4 * TX]);
        };
        if ((s + 1) * BK <= K) {
            float4 a[2][TM], b[2][TN / 4];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[0][i] = a_quad(i, 0);
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) b[0][j] = b_quad(0, j);
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                if (k + 1 < BK)
#pragma unroll
                    for (int j = 0; j < TN / 4; ++j) b[(k + 1) & 1][j] = b_quad(k + 1, j);
                if (k % 4 == 0 && k + 4 < BK)
#pragma unroll
                    for (int i = 0; i < TM; ++i) a[(k / 4 + 1) & 1][i] = a_quad(i, k / 4 + 1);
                unsigned long long bp[TN / 2];
#pragma unroll
                for (int j = 0; j < TN / 4; ++j) {
                    bp[2 * j] = pack2(b[k & 1][j].x, b[k & 1][j].y);
                    bp[2 * j + 1] = pack2(b[k & 1][j].z, b[k & 1][j].w);
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float4 v = a[(k / 4) & 1][i];
                    const float x = k % 4 == 0 ? v.x : k % 4 == 1 ? v.y : k % 4 == 2 ? v.z : v.w;
                    const unsigned long long ap = pack2(x, x);
                    // back and forth: neighbouring FMAs share an operand
#pragma unroll
                    for (int t = 0; t < TN / 2; ++t) {
                        const int j = (i & 1) ? TN / 2 - 1 - t : t;
                        ffma2(acc[i][j], ap, bp[j]);
                    }
                }
            }
        } else {
            // the k past K hold zeros for both operands; they are skipped, so that no
            // extra rounding step (or 0 x infinity) touches the sums. Whole quads of k first
            // (18720 x 30480 x 48, 64 x 64 1429 -> 1401); the 64 x 128 tile has no registers for
            // it, and in the 16 x 64 one it costs the whole slices 10 %.
            const int rest = K - s * BK, quads = TM * TN < 64 && TM > 2 ? rest / 4 : 0;
            auto step = [&](int k, const float (&x)[TM]) {
                unsigned long long bp[TN / 2];
#pragma unroll
                for (int j = 0; j < TN / 4; ++j) {
                    const float4 t = b_quad(k, j);
                    bp[2 * j] = pack2(t.x, t.y);
                    bp[2 * j + 1] = pack2(t.z, t.w);
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const unsigned long long ap = pack2(x[i], x[i]);
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) ffma2(acc[i][j], ap, bp[j]);
                }
            };
#pragma unroll 1
            for (int q = 0; q < quads; ++q) {
                float4 v[TM];
#pragma unroll
                for (int i = 0; i < TM; ++i) v[i] = a_quad(i, q);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float x[TM];
#pragma unroll
                    for (int i = 0; i < TM; ++i)
                        x[i] = u == 0 ? v[i].x : u == 1 ? v[i].y : u == 2 ? v[i].z : v[i].w;
                    step(q * 4 + u, x);
                }
            }
#pragma unroll 1
            for (int k = quads * 4; k < rest; ++k) {
                float x[TM];
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const int r = ty + i * TY;
                    x[i] = As[r * BK + a_chunk(r, k / 4) * 4 + (k & 3)];
                }
                step(k, x);
            }
        }
        buf = buf + 1 == ST ? 0 : buf + 1;
        if (++in_block == per_block || s + 1 == slices) {
            flush(s >= per_block);
            clear();
            in_block = 0;
        }
    }
}

// m_fast: neighbouring CTAs share columns of B rather than rows of A. APART (p.part is
// set): blockIdx.z is a K block of its own; block 0 writes C, block z part z - 1, for
// ffma_add_blocks_kernel. (A kernel of its own: arguments that change live in registers,
// which costs the other one 5 %.)
template <class S, bool VA, bool VB, bool APART>
__global__ void __launch_bounds__(S::NT, S::OCC) ffma_sgemm_kernel(FfmaArgs p, int tiles_m, int tiles_n,
                                                           int m_fast)
{
    extern __shared__ __align__(128) float sm[];
    const int t = blockIdx.x;
    const int tm = m_fast ? t % tiles_m : t / tiles_n, tn = m_fast ? t / tiles_m : t % tiles_n;
    if constexpr (APART) {
        const int z = blockIdx.z, k0 = z * p.kblock;
        p.A += k0;
        p.B += (size_t)k0 * p.ldb;
        p.K = min(p.kblock, p.K - k0);
        if (z > 0) {
            p.C = p.part + (size_t)(z - 1) * p.M * p.ld_part;
            p.ldc = p.ld_part;
        }
        p.kblock = 0;
    }
    ffma_tile<S, VA, VB>(p, tm * S::BM, tn * S::BN, sm);
}

// C = (C + part 0) + part 1 ...: the K blocks' sums, each added in turn as one CTA that
// runs all blocks of its tile adds them. Four columns of a row per thread; VEC: C's
// rows are 16-byte aligned (the parts' always are).
template <bool VEC>
__global__ void __launch_bounds__(256) ffma_add_blocks_kernel(const FfmaArgs p, int parts)
{
    overlap_next();
    overlap_wait();
    const long quads = (p.N + 3) / 4, total = quads * p.M;
    const size_t step = (size_t)p.M * p.ld_part;
    for (long i = blockIdx.x * 256l + threadIdx.x; i < total; i += gridDim.x * 256l) {
        const long m = i / quads, n = (i - m * quads) * 4;
        float *c = p.C + m * p.ldc + n;
        const float *q = p.part + m * p.ld_part + n;
        float r[4];
        if (VEC && n + 3 < p.N) {
            const float4 v = *reinterpret_cast<const float4 *>(c);
            r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u) r[u] = n + u < p.N ? c[u] : 0.f;
        }
#pragma unroll 4
        for (int z = 0; z < parts; ++z) {
            const float4 v = *reinterpret_cast<const float4 *>(q + z * step);
            r[0] = r[0] + v.x; r[1] = r[1] + v.y; r[2] = r[2] + v.z; r[3] = r[3] + v.w;
        }
        if (VEC && n + 3 < p.N) {
            *reinterpret_cast<float4 *>(c) = make_float4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (n + u < p.N) c[u] = r[u];
        }
    }
}

// Many independent SGEMMs: CTA b works on job j with tile0[j] <= b < tile0[j + 1].
template <class S>
__global__ void __launch_bounds__(S::NT, S::OCC) ffma_group_kernel(const FfmaJob *__restrict__ jobs, int njobs)
{
    extern __shared__ __align__(128) float sm[];
    const int b = blockIdx.x;
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (jobs[mid].tile0 <= b)
            lo = mid;
        else
            hi = mid - 1;
    }
    const FfmaJob &j = jobs[lo];
    const int t = b - j.tile0;
    FfmaArgs p;
    p.M = j.M; p.N = j.N; p.K = j.K;
    p.A = j.A; p.lda = j.lda;
    p.B = j.B; p.ldb = j.ldb;
    p.C = j.C; p.ldc = j.ldc;
    p.kblock = 0;
    const int m0 = (t / j.tiles_n) * S::BM, n0 = (t % j.tiles_n) * S::BN;
    if (j.vec)
        ffma_tile<S, true, true>(p, m0, n0, sm);
    else
        ffma_tile<S, false, false>(p, m0, n0, sm);
}

using Wide = Shape<64, 128, 32, 8, 8, 3, 3>;
using Square = Shape<64, 64, 32, 4, 8, 3, 4>;
using Low = Shape<40, 64, 32, 5, 4, 3, 4>;
using Small = Shape<32, 64, 32, 4, 4, 3, 4>;
using Tiny = Shape<16, 64, 32, 2, 4, 3, 5>;

// The tile shapes: CTAs resident per SM, and FMA per clock that an SM reaches with
// one CTA and with all of them (B200; from 256 x 256 x 2048, which gives every shape
// at most one CTA per SM, and from 1632 x 36548 x 1024).
// rest: what a k past the last whole slice of 32 costs, in k of a whole one (18720 x 30480 x
// 40, 48, 64: Wide 1333, 1637, 1589, Square 1160, 1335, 1597).
struct ShapeInfo {
    int bm, bn, occ;
    double one, full, rest;
};
constexpr ShapeInfo kShapes[] = {
    {64, 128, Wide::OCC, 78.5, 87.9, 2.0},   // Wide: the best rate; 128 x 128 (8 x 16 per thread) gains nothing on
                                // it and leaves the SMs idle at both ends of a short K
    {64, 64, Square::OCC, 61.0, 83.9, 1.0},    // Square: two or three per SM where Wide leaves SMs idle
    {40, 64, Low::OCC, 48.0, 79.8, 1.0},    // Low: few rows, and dimensions that 64 pads
    {32, 64, Small::OCC, 43.5, 72.7, 1.0},    // Small: more CTAs where outputs are few
    {16, 64, Tiny::OCC, 28.8, 40.0, 1.0},    // Tiny: few outputs, so many CTAs
};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);

// Clocks per k that the busiest SM needs for `tiles` tiles of a shape: full waves at
// the full rate, then the last wave's CTAs per SM, each as fast as alone until the
// SM saturates. (Occupancy as if every shape's waves were in step; the measured
// order of the shapes at 14 sizes between 256 x 256 x 2048 and 4096 x 4096 x 2048 is the
// model's, but for ties.)
double shape_cost(const ShapeInfo &s, long tiles, int num_sms)
{
    const double area = (double)s.bm * s.bn;
    const long wave = (long)num_sms * s.occ;
    const long rem = tiles % wave;
    double t = (double)(tiles / wave) * s.occ * area / s.full;
    if (rem) {
        const double c = (double)((rem + num_sms - 1) / num_sms);
        t += c * area / (c * s.one < s.full ? c * s.one : s.full);
    }
    return t;
}

// The cheapest shape for `blocks` K blocks side by side (1: none apart), and its cost.
int pick_shape(long M, long N, long K, double blocks, int num_sms, double &cost)
{
    int best = 0;
    const double rest = K > 16 ? (double)(K % 32) / K : 0.0;  // fewer: a tile's fixed cost counts more
    for (int i = 0; i < kNumShapes; ++i) {
        const ShapeInfo &s = kShapes[i];
        const double tiles = (double)((M + s.bm - 1) / s.bm) * ((N + s.bn - 1) / s.bn);
        const double c = shape_cost(s, (long)(tiles * blocks + 0.999), num_sms) * (1.0 + (s.rest - 1.0) * rest);
        if (i == 0 || c < cost) {
            best = i;
            cost = c;
        }
    }
    return best;
}

// FG_FFMA_CFG forces one row of kShapes
int forced_shape()
{
    static const int forced = [] {
        const char *v = getenv("FG_FFMA_CFG");
        const int i = v ? atoi(v) : -1;
        return i < kNumShapes ? i : -1;
    }();
    return forced;
}

// Dynamic shared memory above 48 KB is granted per function and device, once.
template <class F>
cudaError_t allow_smem(F *f, int smem, unsigned long long &done, std::mutex &mu)
{
    if (smem <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    if (done >> (dev & 63) & 1) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) done |= 1ull << (dev & 63);
    return e;
}

template <class S, bool VA, bool VB, bool APART>
cudaError_t launch_tiles(const FfmaArgs &a, cudaStream_t s)
{
    static unsigned long long done;
    static std::mutex mu;
    const cudaError_t e = allow_smem(ffma_sgemm_kernel<S, VA, VB, APART>, S::SMEM, done, mu);
    if (e != cudaSuccess) return e;
    const long tm = (a.M + S::BM - 1) / S::BM, tn = (a.N + S::BN - 1) / S::BN;
    if (tm * tn > 0x7fffffffl) return cudaErrorInvalidConfiguration;
    const unsigned blocks = APART ? (unsigned)((a.K + a.kblock - 1) / a.kblock) : 1u;
    ffma_sgemm_kernel<S, VA, VB, APART>
        <<<dim3((unsigned)(tm * tn), 1, blocks), S::NT, S::SMEM, s>>>(a, (int)tm, (int)tn, tm <= tn);
    return cudaGetLastError();
}

template <class S, bool VA, bool VB>
cudaError_t launch_apart(const FfmaArgs &a, cudaStream_t s)
{
    return a.part ? launch_tiles<S, VA, VB, true>(a, s) : launch_tiles<S, VA, VB, false>(a, s);
}

template <class S>
cudaError_t launch_shape(const FfmaArgs &a, cudaStream_t s)
{
    const bool va = a.lda % 4 == 0 && ((uintptr_t)a.A & 15) == 0;
    const bool vb = a.ldb % 4 == 0 && ((uintptr_t)a.B & 15) == 0;
    if (va) return vb ? launch_apart<S, true, true>(a, s) : launch_apart<S, true, false>(a, s);
    return vb ? launch_apart<S, false, true>(a, s) : launch_apart<S, false, false>(a, s);
}

}  // namespace

void ffma_group_tile(int big, int &tile_m, int &tile_n)
{
    tile_m = big ? Wide::BM : Square::BM;
    tile_n = big ? Wide::BN : Square::BN;
}

cudaError_t launch_ffma_group(const FfmaJob *jobs_dev, int njobs, int total_tiles, int big,
                              cudaStream_t s)
{
    if (njobs < 1 || total_tiles < 1) return cudaSuccess;
    static unsigned long long done[2];
    static std::mutex mu;
    if (big) {
        const cudaError_t e = allow_smem(ffma_group_kernel<Wide>, Wide::SMEM, done[0], mu);
        if (e != cudaSuccess) return e;
        ffma_group_kernel<Wide><<<total_tiles, Wide::NT, Wide::SMEM, s>>>(jobs_dev, njobs);
    } else {
        const cudaError_t e = allow_smem(ffma_group_kernel<Square>, Square::SMEM, done[1], mu);
        if (e != cudaSuccess) return e;
        ffma_group_kernel<Square><<<total_tiles, Square::NT, Square::SMEM, s>>>(jobs_dev, njobs);
    }
    return cudaGetLastError();
}

// K blocks are independent sums until they are added, so where the tiles alone leave
// SMs idle they run side by side, the sums of all but the first in a workspace, and
// a second kernel adds them in order: the same bits. That costs the launch (about
// 3 us) and the parts' traffic; it is taken where the tiles' cost falls by more.
// Measured (B200, us a call; first figure: the kernel before this tile, which could not):
// 128 x 2048 x 4096 277 -> 70, 84 x 1024 x 4096 304 -> 47, 35 x 8457 x 2560 142 -> 77,
// 1024 x 16 x 500000 38100 -> 1435.
size_t ffma_sgemm_workspace(long M, long N, long K, int kblock, int num_sms)
{
    if (M <= 0 || N <= 0 || kblock <= 0 || K <= kblock) return 0;
    const long blocks = (K + kblock - 1) / kblock;
    if (blocks > 65535) return 0;
    const long ld = (N + 3) / 4 * 4;
    const double part_bytes = (double)(blocks - 1) * M * ld * 4;
    if (part_bytes > (double)(1l << 30)) return 0;  // such results fill the SMs anyhow
    double whole = 0.0, apart = 0.0;
    pick_shape(M, N, K, 1.0, num_sms, whole);
    pick_shape(M, N, K, (double)K / kblock, num_sms, apart);
    // clocks: 6000 for the launch, the parts written and read once at 3000 bytes a clock
    return apart * kblock + 6000.0 + 2.0 * part_bytes / 3000.0 < whole * K ? (size_t)part_bytes : 0;
}

cudaError_t launch_ffma_sgemm(const FfmaArgs &a, int num_sms, cudaStream_t s)
{
    if (a.M <= 0 || a.N <= 0) return cudaSuccess;
    if (a.kblock > 0 && a.kblock % 32) return cudaErrorInvalidValue;  // K blocks end on slices
    double cost = 0.0;
    const int shape = forced_shape() >= 0 ? forced_shape()
                                          : pick_shape(a.M, a.N, a.K, a.part ? (double)a.K / a.kblock : 1.0,
                                                       num_sms, cost);
    cudaError_t e;
    switch (shape) {
    case 0: e = launch_shape<Wide>(a, s); break;
    case 1: e = launch_shape<Square>(a, s); break;
    case 2: e = launch_shape<Low>(a, s); break;
    case 3: e = launch_shape<Small>(a, s); break;
    default: e = launch_shape<Tiny>(a, s); break;
    }
    if (e != cudaSuccess || !a.part) return e;
    const int parts = (a.K + a.kblock - 1) / a.kblock - 1;
    const long ctas = ((a.N + 3) / 4 * (long)a.M + 255) / 256;
    const unsigned grid = (unsigned)(ctas < num_sms * 8l ? ctas : num_sms * 8l);
    return launch_overlapped(a.ldc % 4 == 0 && ((uintptr_t)a.C & 15) == 0 ? ffma_add_blocks_kernel<true>
                                                                          : ffma_add_blocks_kernel<false>,
                             dim3(grid), 256, 0, s, a, parts);
}

}  // namespace fg
