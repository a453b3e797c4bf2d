// BF16 / INT8 chains with narrow intermediates, kept in tensor memory.
//
// What the column chain (fg_column.cu) does for FP32, for chains whose intermediates have
// at most 256 rows: one CTA runs a 128-column block of the chain from B to C, every
// stage as the transposed product D^T = X^T W^T. The block's 128 columns are the MMA's M,
// the stage's rows, padded to 16, its N, so that a stage of 24 or 144 rows costs 24 / 128 or
// 144 / 128 of a full tile, not one or two whole ones. D and, from the second stage on, the A
// operand lie in tensor memory (lane = column): an epilogue thread narrows its column's
// sums exactly as the reference does (BF16 round-to-nearest-even, int8 saturation;
// multigemm/src/kernel_bf16.h:356-391, kernel_int8.h:329-385), two or four rows to a TMEM
// word, and writes them back as the next A. The reference's panel permutation moves values
// between the 32 columns of a panel, which are a warp's lanes: shuffles.
//
// What bounds it: shared memory. A 128 x 128 tile with both operands there reads 8 KB per
// 64-clock MMA, all that shared memory delivers, beside what TMA writes; here an MMA reads 4
// KB of activations (later stages: none, A is in TMEM) and 32 bytes per real row.
// Measured (B200, us a call, before -> now; before, the rows were the MMA's M and the
// intermediates lay in shared memory): BF16 16384 x 1296, 144, 32, 192 24.1 -> 16.9, INT8
// 4096 x 4800, 192, 56, 336 37.0 -> 25.0; 65536 x 288, 32, 24, 144, registered, 36 -> 22
// (BF16), 33 -> 18 (INT8); 20000 x 64, 128, 1024 37 -> 30 (BF16), 43 -> 29 (INT8). What is left:
// the first stage's k-blocks come from L2 at 13 TB/s (BF16 table chain), or 32 blocks leave
// 116 SMs idle (INT8; its k-blocks shared by a cluster of four CTAs, sums exchanged over
// distributed shared memory, took 26.8 us: the exchange costs what the split saves).
// Eight epilogue warps, not four: 65536 x 256, 256, 256 44.3 -> 39.4 (BF16), 43.2 -> 35.4 (INT8).
//
// INT8 reference tail rows (multigemm/src/kernel_int8.h:771-1057): their weights come
// pre-shifted by one k-quad, and the epilogue adds weight quad 0 x input quad 0 (one
// mixed-sign dp4a); the stage before puts each column's first quad aside.
//
// Warp 0 is the TMA producer, warp 1 allocates TMEM and issues MMAs, warps 2-9 run the
// epilogues (two per TMEM lane quarter). TMEM: A of the stages after the first, then the
// accumulators (two row tiles of the last stage). A warp stores 32 columns of a row of
// the result at once, a whole line. Every wait is bounded (fg_ptx.cuh); no CTA
// waits on another.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "fg_tc_common.cuh"

namespace fg {

namespace {

constexpr int kNBN = 128;                  // columns per block (MMA M)
constexpr int kNXBytes = kNBN * 128;       // a k-block of B: 128 bytes of k per column
constexpr int kNThreads = 320;
constexpr int kNFixed = 2048 + 1024;       // barriers, alignment
constexpr int kNMaxSmem = 232448, kNHalfSmem = 113 * 1024;

template <int OP>
struct NarrowGeo {
    static constexpr int elt = OP == OP_BF16 ? 2 : 1;
    static constexpr int BK = 128 / elt;                // k per k-block
    static constexpr int KS = 32 / elt;                 // k per MMA
    static constexpr int BOX_N = 128 / elt;             // MN-major box of B: 128-byte rows
    static constexpr int NBOX = kNBN / BOX_N;
    static constexpr int BOX_BYTES = BOX_N * BK * elt;
    static constexpr int X_KSTEP = KS * 128;            // bytes per MMA k-step (MN-major)
    // D F32 / S32; A activations (BF16 / S8), B weights (BF16 / U8, as the reference reads
    // them); a_mn: A as TMA lands it (else in TMEM, k along the columns)
    __host__ __device__ static constexpr uint32_t idesc(bool a_mn, int rows)
    {
        return OP == OP_BF16 ? make_idesc(1, 1, 1, a_mn, 0, kNBN, rows)
                             : make_idesc(2, 1, 0, a_mn, 0, kNBN, rows);
    }
};

struct __align__(8) NarrowBars {
    uint64_t full[kNarrowMaxRing], empty[kNarrowMaxRing];  // ring (TMA bytes / MMAs retired)
    uint64_t dfull[2], dempty[2];                // accumulators (MMAs retired / 8 epilogue warps)
    uint64_t xready;                             // the next stage's A is in place (8 warps)
    uint64_t mma_done;
    uint32_t tmem_base;
    int abort;
    NarrowStage st[kNarrowMaxStages];            // the launch's, read from here (a first read of a
                                                 // parameter line costs some 400 ns, per stage and role)
    uint32_t quad[2][kNBN];                      // INT8: a column's first quad of the next stage's A
};
static_assert(sizeof(NarrowBars) <= 2048, "barrier block");

__device__ __forceinline__ void n_set_abort(NarrowBars *b) { *reinterpret_cast<volatile int *>(&b->abort) = 1; }
__device__ __forceinline__ bool n_aborted(NarrowBars *b) { return *reinterpret_cast<volatile int *>(&b->abort) != 0; }

// Timeline of a tile (FG_TRACE_DIR): its description, then the roles' stamps.
enum { NT_DESC, NT_PROD_START, NT_PROD_END, NT_MMA_WAIT, NT_MMA_START, NT_MMA_END, NT_EPI_START,
       NT_EPI_END };
__device__ __forceinline__ void ntrace(const NarrowArgs &g, int u, int f, unsigned long long v)
{
    if (g.trace && u < g.trace_units)
        g.trace[((size_t)blockIdx.x * g.trace_units + u) * kNarrowTraceFields + f] = v;
}

}  // namespace

template <int OP>
__global__ void __launch_bounds__(kNThreads, 2) tc_narrow_kernel(const __grid_constant__ NarrowArgs g)
{
    using G = NarrowGeo<OP>;
    constexpr MmaKind KIND = OP == OP_BF16 ? MmaKind::F16 : MmaKind::I8;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    NarrowBars *bars = reinterpret_cast<NarrowBars *>(smem + g.ring * g.slot_bytes);
    int *status = g.status;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // What a tile's k-blocks are loaded with: the weights' map and row, the boxes of B that
    // start inside N (stage 0).
    struct Tile {
        const CUtensorMap *w;
        uint32_t bytes;
        int wy, nvb, n0;
    };
    auto tile_of = [&](const NarrowStage &cs, int st, int blk, int t) {
        Tile q;
        const int m0 = t * cs.rows;
        const bool tail = cs.tail_hi > cs.tail_lo && m0 < cs.tail_hi && m0 + cs.rows > cs.tail_lo;
        q.n0 = blk * kNBN;
        q.nvb = st == 0 ? min(G::NBOX, (g.N - q.n0 + G::BOX_N - 1) / G::BOX_N) : 0;
        q.w = tail ? &g.tm_wt[st] : &g.tm_w[st];
        q.wy = tail ? m0 - cs.tail_row0 : m0;
        q.bytes = (uint32_t)(cs.rows * 128 + q.nvb * G::BOX_BYTES);
        return q;
    };
    // k-block kb of a tile into ring slot i
    auto load = [&](const Tile &q, int kb, int i) {
        uint8_t *p = smem + i * g.slot_bytes;
        mbar_arrive_expect_tx(&bars->full[i], q.bytes);
        if (q.nvb > 0) tma_load_2d(p, &g.tm_x, &bars->full[i], q.n0, kb * G::BK);
        if (G::NBOX > 1 && q.nvb > 1)
            tma_load_2d(p + G::BOX_BYTES, &g.tm_x, &bars->full[i], q.n0 + G::BOX_N, kb * G::BK);
        tma_load_2d(p + kNXBytes, q.w, &bars->full[i], kb * G::BK, q.wy);
    };
    const int first_loads = min(g.ring, (g.st[0].K + G::BK - 1) / G::BK);

    if (threadIdx.x == 0) {
        for (int r = 0; r < kNarrowMaxRing; ++r) {
            mbar_init(&bars->full[r], 1);
            mbar_init(&bars->empty[r], 1);
        }
        for (int d = 0; d < 2; ++d) {
            mbar_init(&bars->dfull[d], 1);
            mbar_init(&bars->dempty[d], 8);
        }
        mbar_init(&bars->xready, 8);
        mbar_init(&bars->mma_done, 1);
        bars->abort = 0;
        fence_mbar_init();
        // the ring's first round needs no wait: under way before the CTA meets
        overlap_wait();
        const Tile q0 = tile_of(g.st[0], 0, blockIdx.x, 0);
        for (int kb = 0; kb < first_loads; ++kb) load(q0, kb, kb);
        for (int i = 1; i < g.n; ++i) {
            tma_prefetch_desc(&g.tm_w[i]);
            if (g.st[i].tail_hi > g.st[i].tail_lo) tma_prefetch_desc(&g.tm_wt[i]);
        }
    }
    if (warp == 1) tmem_alloc(&bars->tmem_base, g.tmem_cols);
    if (threadIdx.x >= 64 && threadIdx.x < 64 + g.n) bars->st[threadIdx.x - 64] = g.st[threadIdx.x - 64];
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    overlap_next();
    overlap_wait();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            int s = 0, skip = first_loads, u = 0;
            uint32_t ph = 0, pending = (1u << first_loads) - 1, pending_ph = 0;
            for (int blk = blockIdx.x; blk < g.nblocks; blk += gridDim.x) {
                for (int st = 0; st < g.n; ++st) {
                    const NarrowStage cs = bars->st[st];  // in registers
                    const int nkb = (cs.K + G::BK - 1) / G::BK;
                    for (int t = 0; t < cs.tiles; ++t, ++u) {
                        if (g.trace) {
                            unsigned sm;
                            asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
                            ntrace(g, u, NT_DESC,
                                   (unsigned long long)st | (unsigned long long)(blk / gridDim.x) << 8 |
                                       (unsigned long long)t << 24 | 1ull << 32 | (unsigned long long)sm << 40);
                            ntrace(g, u, NT_PROD_START, globaltimer_ns());
                        }
                        const Tile q = tile_of(cs, st, blk, t);
                        bool ready = false;
                        for (int kb = 0; kb < nkb; ++kb) {
                            if (skip > 0) {  // loaded above
                                --skip;
                            } else {
                                if (!ready && !mbar_wait(&bars->empty[s], ph ^ 1, status, KERR_WAIT_EMPTY)) {
                                    n_set_abort(bars);
                                    goto producer_done;
                                }
                                // the next slot, asked now and looked at after these loads are issued
                                const int s1 = s + 1 == g.ring ? 0 : s + 1;
                                ready = mbar_test(&bars->empty[s1], s1 ? ph ^ 1 : ph);
                                load(q, kb, s);
                                pending |= 1u << s;
                                pending_ph = (pending_ph & ~(1u << s)) | (ph << s);
                            }
                            if (++s == g.ring) {
                                s = 0;
                                ph ^= 1;
                            }
                        }
                        if (g.trace) ntrace(g, u, NT_PROD_END, globaltimer_ns());
                    }
                }
                if (n_aborted(bars)) break;
            }
        producer_done:
            // never leave with copies in flight into this CTA's shared memory
            for (int i = 0; i < g.ring; ++i)
                if (pending & (1u << i))
                    mbar_wait(&bars->full[i], (pending_ph >> i) & 1u, status, KERR_WAIT_FULL);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 0, tiles = 0, xr = 0;
            const uint64_t x_desc0 = smem_desc(smem_u32(smem), G::BOX_BYTES, 1024, SMEM_SW128);
            const uint64_t w_desc0 = smem_desc(smem_u32(smem) + kNXBytes, 16, 1024, SMEM_SW128);
            bool ok = true;
            for (int blk = blockIdx.x; ok && blk < g.nblocks; blk += gridDim.x) {
                for (int st = 0; ok && st < g.n; ++st) {
                    const NarrowStage cs = bars->st[st];  // in registers
                    const int K = cs.K, ntiles = cs.tiles;
                    const int nkb = (K + G::BK - 1) / G::BK;
                    const uint32_t idesc = G::idesc(st == 0, cs.rows);
                    if (g.trace) ntrace(g, tiles, NT_MMA_WAIT, globaltimer_ns());
                    if (st > 0) {
                        ok = mbar_wait(&bars->xready, xr & 1u, status, KERR_WAIT_FULL);
                        ++xr;
                    }
                    for (int t = 0; ok && t < ntiles; ++t, ++tiles) {
                        // accumulator t & 1; the tile before is read first where this is a new stage
                        // (its accumulators may overlie; past the first, xready came after that
                        // read), else only the one before that
                        if (t == 0 && st == 0 && tiles > 0)
                            ok = mbar_wait(&bars->dempty[(tiles - 1) & 1u], ((tiles - 1) >> 1) & 1u, status,
                                           KERR_WAIT_ACC_EMPTY);
                        else if (t > 1)
                            ok = mbar_wait(&bars->dempty[tiles & 1u], ((tiles - 2) >> 1) & 1u, status,
                                           KERR_WAIT_ACC_EMPTY);
                        if (!ok) break;
                        if (g.trace) {
                            if (t > 0) ntrace(g, tiles, NT_MMA_WAIT, globaltimer_ns());
                            ntrace(g, tiles, NT_MMA_START, globaltimer_ns());
                        }
                        const uint32_t d_tmem = tmem_base + g.acc + (t & 1) * g.acc_step;
                        uint32_t more = 0;
                        bool ready = false;
                        for (int kb = 0; kb < nkb; ++kb) {
                            if (!ready && !(ok = mbar_wait(&bars->full[s], ph, status, KERR_WAIT_FULL))) break;
                            tc_fence_after();
                            // the next slot, asked now and looked at after these MMAs are issued
                            const int s1 = s + 1 == g.ring ? 0 : s + 1;
                            ready = mbar_test(&bars->full[s1], s1 ? ph : ph ^ 1);
                            const uint64_t off = (uint64_t)((s * g.slot_bytes) >> 4);
                            const uint64_t w = w_desc0 + off, x = x_desc0 + off;
                            const int steps = min(4, (K - kb * G::BK + G::KS - 1) / G::KS);
                            if (st == 0) {
                                if (steps == 4) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k) {
                                        tc_mma<KIND>(d_tmem, x + k * (G::X_KSTEP >> 4), w + k * 2, idesc, more);
                                        more = 1;
                                    }
                                } else {
                                    for (int k = 0; k < steps; ++k) {
                                        tc_mma<KIND>(d_tmem, x + k * (G::X_KSTEP >> 4), w + k * 2, idesc, more);
                                        more = 1;
                                    }
                                }
                            } else {
                                const uint32_t a = tmem_base + kb * 32;
                                if (steps == 4) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k) {
                                        tc_mma_ts<KIND>(d_tmem, a + k * 8, w + k * 2, idesc, more);
                                        more = 1;
                                    }
                                } else {
                                    for (int k = 0; k < steps; ++k) {
                                        tc_mma_ts<KIND>(d_tmem, a + k * 8, w + k * 2, idesc, more);
                                        more = 1;
                                    }
                                }
                            }
                            tc_commit(&bars->empty[s]);
                            if (++s == g.ring) {
                                s = 0;
                                ph ^= 1;
                            }
                        }
                        if (!ok) break;
                        tc_commit(&bars->dfull[tiles & 1u]);
                        if (g.trace) ntrace(g, tiles, NT_MMA_END, globaltimer_ns());
                    }
                }
                if (n_aborted(bars)) break;
            }
            if (!ok) n_set_abort(bars);
            tc_commit(&bars->mma_done);
            mbar_wait(&bars->mma_done, 0, status, KERR_WAIT_FULL);
        }
    } else {
        // ------------------------------------------------------------ epilogues
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        uint32_t(*quad)[kNBN] = bars->quad;
        uint32_t xr = 0;
        const uint32_t t_lane = (uint32_t)(quarter * 32) << 16;
        uint32_t tiles = 0;
        bool ok = true;
        for (int blk = blockIdx.x; ok && blk < g.nblocks; blk += gridDim.x) {
            const int c0 = blk * kNBN + quarter * 32, col = c0 + lane;
            const bool panel = c0 + 32 <= g.N;  // a whole panel: permuted
            for (int st = 0; ok && st < g.n; ++st) {
                const NarrowStage cs = bars->st[st];  // in registers
                const bool last = st + 1 == g.n;
                const bool tails = OP == OP_I8 && cs.tail_hi > cs.tail_lo;
                // INT8 tails: the first quad of this column's input; of B it is fetched while
                // the MMAs run, later ones were put aside by the stage before
                uint32_t xq = 0;
                if (OP == OP_I8 && st > 0) {
                    if (!(ok = mbar_wait(&bars->xready, xr & 1u, status, KERR_WAIT_FULL))) break;
                    ++xr;
                    xq = quad[st & 1][quarter * 32 + lane];
                }
                if (tails && st == 0 && col < g.N)
                    for (int q = 0; q < 4 && q < cs.K; ++q)
                        xq |= (uint32_t)g.b[(size_t)q * g.ldb + col] << (8 * q);
                // and lane j's weight quad 0 of tail row tail_lo + j (at most 8 rows)
                uint32_t wq = 0;
                if (tails && lane < cs.tail_hi - cs.tail_lo)
                    wq = *reinterpret_cast<const uint32_t *>(
                        cs.w_tail + (size_t)(cs.tail_lo + lane - cs.tail_row0) * cs.ld_w_tail + cs.K);
                for (int t = 0; ok && t < cs.tiles; ++t, ++tiles) {
                    if (!(ok = mbar_wait(&bars->dfull[tiles & 1u], (tiles >> 1) & 1u, status, KERR_WAIT_ACC_FULL)))
                        break;
                    tc_fence_after();
                    if (g.trace && warp == 2 && lane == 0) ntrace(g, tiles, NT_EPI_START, globaltimer_ns());
                    const uint32_t d = tmem_base + g.acc + (t & 1) * g.acc_step + t_lane;
                    // the two warps of a quarter share the rows
                    const int m0 = t * cs.rows, g2 = (cs.rows / 16 + 1) / 2;
                    const int first = half * g2, groups = half ? cs.rows / 16 : g2;
                    // 16 rows from the stage's row r0 on
                    auto rows16 = [&](uint32_t (&v)[16], int c) {
                        const int r0 = m0 + c * 16;
                        if (tails && r0 < cs.tail_hi && r0 + 16 > cs.tail_lo) {
// tail_lo and tail_hi are whole quads of rows: warp-uniform tests per quad
#pragma unroll
                            for (int q = 0; q < 16; q += 4)
                                if (r0 + q >= cs.tail_lo && r0 + q < cs.tail_hi) {
#pragma unroll
                                    for (int j = q; j < q + 4; ++j) {
                                        const uint32_t w = __shfl_sync(0xffffffffu, wq, r0 + j - cs.tail_lo);
                                        int r;
                                        asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(xq), "r"((int)v[j]));
                                        v[j] = (uint32_t)r;
                                    }
                                }
                        }
                        if (last) {
                            // a row's 32 columns of this warp are one 128-byte line
                            if (col < g.N) {
                                uint32_t *o = g.out + (size_t)r0 * g.ldo + col;
                                if (r0 + 16 <= g.out_rows) {
#pragma unroll
                                    for (int j = 0; j < 16; ++j) o[(size_t)j * g.ldo] = v[j];
                                } else {
#pragma unroll
                                    for (int j = 0; j < 16; ++j)
                                        if (r0 + j < g.out_rows) o[(size_t)j * g.ldo] = v[j];
                                }
                            }
                        } else if constexpr (OP == OP_BF16) {
                            // row pairs to words; (2q + h, c) -> (2q + (c & 1), 16h + c / 2) of a panel
                            // (kernel_bf16.h:6-32): column 16h + t takes row 2q + h of columns
                            // 2t and 2t + 1
                            uint32_t w[8];
#pragma unroll
                            for (int q = 0; q < 8; ++q) w[q] = pack_bf16x2(v[2 * q], v[2 * q + 1]);
                            // rows past M are zeros for the next stage (0 x NaN would not be);
                            // its MMAs read no row past these 16
                            if (r0 + 16 > cs.M) {
#pragma unroll
                                for (int q = 0; q < 8; ++q) {
                                    const int left = cs.M - (r0 + 2 * q);
                                    w[q] &= left >= 2 ? 0xffffffffu : left == 1 ? 0xffffu : 0u;
                                }
                            }
                            if (cs.permute && panel) {
                                const int from = 2 * (lane & 15);
                                const uint32_t pick = lane & 16 ? 0x7632u : 0x5410u;
#pragma unroll
                                for (int q = 0; q < 8; ++q) {
                                    const uint32_t a = __shfl_sync(0xffffffffu, w[q], from);
                                    const uint32_t b = __shfl_sync(0xffffffffu, w[q], from + 1);
                                    // an odd last row stays where it is
                                    if (r0 + 2 * q + 1 < cs.M) w[q] = __byte_perm(a, b, pick);
                                }
                            }
                            tmem_st_32x32b_x8(tmem_base + t_lane + c * 8, w);
                        } else {
                            // row quads to words; (4q + h, c) -> (4q + (c & 3), 8h + c / 4) of a panel
                            // (kernel_int8.h:6-50): column 8h + t takes row 4q + h of columns
                            // 4t .. 4t + 3
                            uint32_t w[4];
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                w[q] = pack_s8x4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                            if (cs.permute && panel) {
                                const int from = 4 * (lane & 7);
                                const uint32_t h = lane >> 3, pick = h | (h + 4) << 4;
#pragma unroll
                                for (int q = 0; q < 4; ++q) {
                                    const uint32_t a = __shfl_sync(0xffffffffu, w[q], from);
                                    const uint32_t b = __shfl_sync(0xffffffffu, w[q], from + 1);
                                    const uint32_t e = __shfl_sync(0xffffffffu, w[q], from + 2);
                                    const uint32_t f = __shfl_sync(0xffffffffu, w[q], from + 3);
                                    // rows past the last whole quad stay where they are
                                    if (r0 + 4 * q + 3 < cs.M)
                                        w[q] = __byte_perm(__byte_perm(a, b, pick), __byte_perm(e, f, pick), 0x5410u);
                                }
                            }
                            if (c == 0) quad[(st + 1) & 1][quarter * 32 + lane] = w[0];
                            tmem_st_32x32b_x4(tmem_base + t_lane + c * 4, w);
                        }
                    };
                    // two pieces in turn: the next one's TMEM load is under way meanwhile
                    uint32_t va[16], vb[16];
                    if (first < groups) tmem_ld_32x32b_x16(d + first * 16, va);
#pragma unroll 1
                    for (int c = first; c < groups; c += 2) {
                        tmem_ld_wait();
                        if (c + 1 < groups) tmem_ld_32x32b_x16(d + (c + 1) * 16, vb);
                        rows16(va, c);
                        if (c + 1 >= groups) break;
                        tmem_ld_wait();
                        if (c + 2 < groups) tmem_ld_32x32b_x16(d + (c + 2) * 16, va);
                        rows16(vb, c + 1);
                    }
                    if (!last) tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&bars->dempty[tiles & 1u]);
                        if (!last) mbar_arrive(&bars->xready);
                        if (g.trace && warp == 2) ntrace(g, tiles, NT_EPI_END, globaltimer_ns());
                    }
                }
            }
            if (n_aborted(bars)) break;
        }
        if (!ok) n_set_abort(bars);
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc(tmem_base, g.tmem_cols);
    }
}

// ------------------------------------------------------------------ host side

namespace {

int pad16(long m) { return (int)((m + 15) / 16 * 16); }

// Tiles, TMEM columns and the ring; two CTAs per SM where there are more blocks than SMs and
// half an SM holds a CTA (BF16 65536 x 64, 64, 64
// 14.2 -> 9.7 us); fewer blocks get the whole ring (2048, 128, 128 18.7 -> 17.5 us)
template <int OP>
bool narrow_layout(const StageArgs *st, int n, bool half, NarrowArgs &A)
{
    using G = NarrowGeo<OP>;
    int xa = 0, rows_max = 0, acc = 0;
    for (int i = 0; i < n; ++i) {
        NarrowStage &cs = A.st[i];
        cs.tiles = 1;
        if (i + 1 < n) {
            cs.rows = pad16(st[i].M);
            // the next stage's A: whole MMA steps of words
            xa = std::max(xa, (st[i].M + G::KS - 1) / G::KS * 8);
            acc = std::max(acc, cs.rows);
        } else {
            // tiles that divide the 256-row block of an INT8 tail, or lie in its only one
            cs.tiles = (st[i].M + 127) / 128;
            cs.rows = st[i].M > 256 ? 128 : pad16((st[i].M + cs.tiles - 1) / cs.tiles);
            A.acc_step = cs.tiles > 1 ? cs.rows : 0;
            acc = std::max(acc, cs.rows + A.acc_step);
        }
        rows_max = std::max(rows_max, cs.rows);
    }
    A.acc = (xa + 15) / 16 * 16;
    A.tmem_cols = half ? 256 : 512;
    if (A.acc + acc > A.tmem_cols) return false;
    A.slot_bytes = kNXBytes + rows_max * 128;
    A.ring = std::min(kNarrowMaxRing, ((half ? kNHalfSmem : kNMaxSmem) - kNFixed) / A.slot_bytes);
    A.smem = A.ring * A.slot_bytes + kNFixed;
    A.per_sm = half ? 2 : 1;
    A.nblocks = (st[0].N + kNBN - 1) / kNBN;
    return A.ring >= 3;
}

template <int OP>
bool narrow_layout(const StageArgs *st, int n, int num_sms, NarrowArgs &A)
{
    const bool half = (st[0].N + kNBN - 1) / kNBN > num_sms;
    return (half && narrow_layout<OP>(st, n, true, A)) || narrow_layout<OP>(st, n, false, A);
}

}  // namespace

bool narrow_eligible(const StageArgs *st, int n)
{
    if (n < 2 || n > kNarrowMaxStages) return false;
    const int op = st[0].op;
    if (op != OP_BF16 && op != OP_I8) return false;
    const long N = st[0].N;
    if (N < 1 || (N + kNBN - 1) / kNBN > (1l << 30)) return false;
    for (int i = 0; i < n; ++i) {
        if (st[i].op != op || st[i].N != N) return false;
        if (i + 1 < n && (st[i].M > kNarrowRows || st[i].M < 1)) return false;
    }
    return true;
}

// Microseconds of both kernels, fitted to measurements on B200 of 3100 random chains of 2 to
// 6 stages per type (N = 16 to 65536, K_1 = 16 to 8400, last stage of up to 4096 rows, registered
// weights). Narrow: a block's stages one after the other (per stage, per k-block, per row, per
// tile of the last), the blocks of one SM in turn, or two at a time. Fused: a stage's tiles over
// all CTA pairs; it reads each INT8 tail row's quad per column. (More than 144 rows leave the
// first stage of a BF16 chain fewer ring slots.) The lower one of the two is the faster, or
// within 5 % of it, at 99.5 % of them, and within 17 % at the rest. Measured, us, narrow / fused: BF16 256,256,256 at N = 9216 12 / 18, at 65536 39 / 41;
// 4532,12,2244 at 96 45 / 33; 4472,8,80,16,1288 at 2308 68 / 74; INT8 4800,192,56,336 at 4096
// 22 / 41; 136,8,80,36,28,28,3156 at 688 42 / 73; 364,232,20,2584 at 16 34 / 23.
bool narrow_preferred(const StageArgs *st, int n, int num_sms)
{
    static thread_local NarrowArgs A;
    const bool i8 = st[0].op == OP_I8;
    if (!(i8 ? narrow_layout<OP_I8>(st, n, num_sms, A) : narrow_layout<OP_BF16>(st, n, num_sms, A))) return false;
    const double kb_elems = i8 ? 128.0 : 64.0;
    const long N = st[0].N, pairs = num_sms / 2;
    double block = 0.0, fused = i8 ? 5.0 : 4.8;
    for (int i = 0; i < n; ++i) {
        const double kb = std::ceil(st[i].K / kb_elems), rows = A.st[i].rows;
        if (i + 1 == n)
            block += A.st[i].tiles * (i8 ? 1.33 + 0.063 * kb : 1.23 + 0.14 * kb);
        else if (i8)
            block += 0.46 + 0.0068 * rows + kb * (i ? 0.354 : 0.317 + 0.00023 * rows);
        else
            block += 0.64 + 0.0074 * rows + kb * (i ? 0.23 : 0.28 + 0.0014 * std::max(0.0, rows - 144.0));
        const double rounds =
            std::ceil((double)((st[i].M + 255) / 256) * ((N + 255) / 256) / pairs);
        fused += i8 ? 4.1 + kb * rounds * 0.33 + (rounds - 1.0) * 4.0
                    : 4.7 + kb * rounds * 0.29 + (rounds - 1.0) * 5.7;
        if (st[i].tail_hi > st[i].tail_lo) fused += 10.8 * std::min(1.0, N / 256.0);
    }
    const double rounds = std::ceil((double)((N + kNBN - 1) / kNBN) / num_sms);
    const double again = A.per_sm > 1 ? (i8 ? 0.87 : 1.07) : (i8 ? 1.19 : 1.57);
    const double narrow = (i8 ? 3.2 : 2.8) + block * (1.0 + (rounds - 1.0) * again);
    return narrow < fused;
}

namespace {

template <int OP>
cudaError_t narrow_attr()
{
    static std::mutex mu;
    static unsigned long long done = 0;
    std::lock_guard<std::mutex> lk(mu);
    int dev = 0;
    cudaGetDevice(&dev);
    if (done >> (dev & 63) & 1) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(tc_narrow_kernel<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, kNMaxSmem);
    if (e == cudaSuccess) done |= 1ull << (dev & 63);
    return e;
}

template <int OP>
cudaError_t plan_narrow_op(const StageArgs *st, int n, int num_sms, NarrowArgs &out, int &grid)
{
    using G = NarrowGeo<OP>;
    const CUtensorMapDataType dt = OP == OP_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
    // parameter blocks of the last few operand sets (tensor maps encoded once)
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    struct Built {
        std::vector<long> key;
        NarrowArgs P;
    };
    static std::vector<std::unique_ptr<Built>> built;
    int dev = 0;
    cudaGetDevice(&dev);
    std::vector<long> key = {dev, num_sms, n};
    for (int i = 0; i < n; ++i) {
        const StageArgs &a = st[i];
        const long v[] = {a.M, a.N, a.K, (long)a.w, a.ld_w, (long)a.x, a.ld_x, a.epi, (long)a.out,
                          a.ld_out, a.permute, a.m_written, a.tail_lo, a.tail_hi,
                          (long)a.w_tail, a.ld_w_tail, a.tail_row0};
        key.insert(key.end(), std::begin(v), std::end(v));
    }
    NarrowArgs *P = nullptr;
    for (size_t i = 0; i < built.size(); ++i)
        if (built[i]->key == key) {
            std::unique_ptr<Built> b = std::move(built[i]);
            built.erase(built.begin() + i);
            built.push_back(std::move(b));
            P = &built.back()->P;
            break;
        }
    if (!P) {
        std::unique_ptr<Built> b(new Built);
        memset(&b->P, 0, sizeof b->P);
        NarrowArgs &A = b->P;
        if (!narrow_layout<OP>(st, n, num_sms, A)) return cudaErrorNotSupported;
        if (!make_map(&A.tm_x, dt, G::elt, st[0].x, st[0].K, st[0].N, st[0].ld_x, G::BOX_N, G::BK))
            return cudaErrorNotSupported;
        for (int i = 0; i < n; ++i) {
            const StageArgs &a = st[i];
            NarrowStage &cs = A.st[i];
            if (!make_map(&A.tm_w[i], dt, G::elt, a.w, a.M, a.K, a.ld_w, G::BK, cs.rows))
                return cudaErrorNotSupported;
            A.tm_wt[i] = A.tm_w[i];
            if (a.tail_hi > a.tail_lo &&
                !make_map(&A.tm_wt[i], dt, G::elt, a.w_tail, a.M - a.tail_row0, a.K, a.ld_w_tail, G::BK,
                          cs.rows))
                return cudaErrorNotSupported;
            cs.M = a.M;
            cs.K = a.K;
            cs.permute = a.permute;
            cs.tail_lo = a.tail_lo;
            cs.tail_hi = a.tail_hi;
            cs.tail_row0 = a.tail_row0;
            cs.w_tail = static_cast<const uint8_t *>(a.w_tail);
            cs.ld_w_tail = a.ld_w_tail;
        }
        A.b = static_cast<const uint8_t *>(st[0].x);
        A.ldb = st[0].ld_x;
        A.out = static_cast<uint32_t *>(st[n - 1].out);
        A.ldo = st[n - 1].ld_out;
        A.out_rows = st[n - 1].m_written;
        A.op = OP;
        A.n = n;
        A.N = st[0].N;
        b->key.swap(key);
        if (built.size() >= 8) built.erase(built.begin());
        built.push_back(std::move(b));
        P = &built.back()->P;
    }
    const cudaError_t e = narrow_attr<OP>();
    if (e != cudaSuccess) return e;
    out = *P;  // a copy: the entry may go once the lock is released
    grid = std::min(P->nblocks, num_sms * P->per_sm);
    return cudaSuccess;
}

}  // namespace

cudaError_t plan_narrow(const StageArgs *st, int n, int num_sms, NarrowArgs &out, int &grid)
{
    if (!narrow_eligible(st, n)) return cudaErrorNotSupported;
    return st[0].op == OP_BF16 ? plan_narrow_op<OP_BF16>(st, n, num_sms, out, grid)
                               : plan_narrow_op<OP_I8>(st, n, num_sms, out, grid);
}

int narrow_units_per_cta(const NarrowArgs &P, int grid)
{
    return (P.nblocks + grid - 1) / grid * (P.n - 1 + P.st[P.n - 1].tiles);
}

cudaError_t launch_narrow(NarrowArgs &P, int grid, int *status, cudaStream_t s)
{
    P.status = status;
    return launch_overlapped(P.op == OP_BF16 ? tc_narrow_kernel<OP_BF16> : tc_narrow_kernel<OP_I8>, dim3(grid),
                             kNThreads, P.smem, s, P);
}

}  // namespace fg
