// FP32 (3xTF32) chains with narrow intermediates, kept in tensor memory: the
// column chain.
//
// The reference runs all stages of a 32-column panel back to back on one core
// and writes each stage's output straight into the next stage's packed operand
// (multigemm/src/flashgemm.c:123-148; kernel_f32.h:470), so its intermediates
// never leave the core. Its own test chains are wide and narrow: N up to 65536
// activation columns, K_1 up to 8400, intermediates of 16 to 336 rows
// (multigemm/test/test_f32_3.c:14-48). Here one CTA runs a 128-column block of
// such a chain from B to C.
//
// Each stage computes the transposed product D^T = X^T W^T: the block's 128
// columns are the MMA's M, the stage's rows (padded to 16) its N. Both D and the A
// operand X^T live in tensor memory, where lane n is column n of the block and a
// TMEM column is one row of the stage (D) or one k (A). So the result of a stage
// lies exactly as the next stage's operand has to: an epilogue thread reads its
// column's sums, splits them into the TF32 pair (hi, lo) and writes them back as the
// next A, with no shared memory, no swizzle and no proxy fence between. The first
// stage's operand comes the same way: B lands by TMA as plain FP32, four splitter
// warps read it (a thread its own column, conflict-free) and put (hi, lo) into a ring
// of 16-deep granules in TMEM. Only the weights are shared-memory operands.
//
// What bounds it: the thread that issues the MMAs (about 70 clocks for each, 67 for a
// commit, 96 for a wait that is already over) and the tensor pipe (three TF32 products
// per 8 k of 48 clocks each up to 96 rows, rows / 2 above), hence one MMA for two of the
// products where it fits, one commit per k-block, and waits tested ahead; and, on many
// columns, reading B once. The launch-per-stage path that it replaces wrote B's split to
// memory and read it back (3x its bytes) and paid a launch and a memory round trip per
// stage. Measured (B200, us a call, weights split per call, that path -> this): 12544 x 864,
// 96, 24, 144 102 -> 33; 65536 x 288, 32, 24, 144 163 -> 49; 50176 x 288, 32, 16, 96 125 ->
// 38; 16384 x 1296, 144, 32, 192 185 -> 63; 3136 x the same 80 -> 59.
//
// The arithmetic is that path's: per 8 k the correction terms lo * hi, then hi * lo,
// into their own accumulator and hi * hi into the chunk's (hi * [hi | lo] as one MMA over the
// stacked weights, into adjacent accumulators); every `kchunk` k-blocks
// of 32 the chunk's sum goes to FP32 registers, the correction is added once at the
// end; so the results are the same bits.
//
// Warp 0 is the TMA producer, warp 1 allocates TMEM and issues MMAs, warps 2-5 split,
// warps 6-9 run the epilogues (a warp of each group per TMEM lane quarter). Accumulators
// are [d0 | c | d1]: two chunk sums around the correction. TMEM from the bottom: stage
// 0's accumulators, or a later stage's A operand and then its accumulators (dead and
// live parts never meet: every MMA of a stage has completed, and every warp of a lane
// quarter has read its sums, before the quarter's operand is written); the granule ring above all of them, so
// that the next block's input is split while this block's last stages run. Every wait
// is bounded (fg_ptx.cuh); no CTA waits on another.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "fg_tc_common.cuh"

namespace fg {

namespace {

constexpr int kCBN = 128;                     // columns per block (MMA M)
constexpr int kCBK = 32;                      // k per k-block (a 128-byte weight row)
constexpr int kCXBytes = kCBN * kCBK * 4;     // a k-block of B: 32 rows of 128 floats
constexpr int kCMaxRing = 8, kCMaxGran = 8;
// Warps: TMA producer, MMA issuer, 4 splitters, EW epilogue warps
__host__ __device__ constexpr int c_threads(int ew) { return 32 * (6 + ew); }
constexpr int kCFixed = 512 + 1024;           // barriers, alignment
constexpr int kCMaxSmem = 232448;
constexpr int kCHalfSmem = 113 * 1024;        // two CTAs per SM
// Two builds: up to 48 rows per tile (half of TMEM and of shared memory, two CTAs per
// SM, so that one CTA's chain of stages fills the other's waits; 4 epilogue warps) and up
// to 144 (8 epilogue warps, two per TMEM lane quarter)
constexpr int kCSmallRows = 48, kCRows = 144;

struct ColStage {
    CUtensorMap tm_hi, tm_lo;  // weights, K-major boxes of `rows` rows x 128 bytes
    int M, K, kchunk;
    int rows, tiles;           // rows per tile (a multiple of 16); more than one tile: last stage only
    int acc;                   // TMEM column of its accumulators
    int stack;                 // rows <= 128: hi and lo weights as one operand of 2 x rows
};

struct alignas(64) ColArgs {
    CUtensorMap tm_x;          // B: boxes of 128 columns x 32 rows, no swizzle
    ColStage st[kPanelMaxStages];
    float *C;
    long ldc;
    int n, N, nblocks;
    int ring, slot_bytes;      // shared-memory ring: B's k-block, then hi and lo weight boxes
    int gran, gran_k, gran0;   // A ring: granules, k per granule (16 or 32), first TMEM column
    int later_rounds;          // ring rounds of a block after its first stage
    int tmem_cols, smem, small;
    int *status;
};

struct __align__(8) ColBars {
    uint64_t full[kCMaxRing];                      // shared-memory ring: TMA bytes
    uint64_t empty[kCMaxRing];                     // MMAs retired, and the 4 splitter warps are past it
    uint64_t afull[kCMaxGran], aempty[kCMaxGran];  // A ring: 4 splitter warps / 16-deep granules: MMAs retired
    uint64_t dfull[2], dempty[2];                  // chunk sums (MMAs retired / epilogue warps)
    uint64_t cfull;                                // a tile's MMAs have all retired
    uint64_t drained;                              // the epilogue warps have read all of the tile
    uint64_t xready;                               // the next stage's A operand is in place
    uint64_t mma_done;
    uint32_t tmem_base;
    int abort;
};
static_assert(sizeof(ColBars) <= 512, "barrier block");

__device__ __forceinline__ void c_set_abort(ColBars *b) { *reinterpret_cast<volatile int *>(&b->abort) = 1; }
__device__ __forceinline__ bool c_aborted(ColBars *b) { return *reinterpret_cast<volatile int *>(&b->abort) != 0; }

// A position in a ring and the parity of its current round.
struct RingPos {
    int i = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void next(int n)
    {
        if (++i == n) {
            i = 0;
            ph ^= 1;
        }
    }
};

}  // namespace

// NG: 16-row groups of the widest tile per epilogue warp; EW: epilogue warps; PER: CTAs per SM
template <int NG, int EW, int PER>
__global__ void __launch_bounds__(c_threads(EW), PER) tc_column_kernel(const __grid_constant__ ColArgs g)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    uint8_t *smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    ColBars *bars = reinterpret_cast<ColBars *>(smem + g.ring * g.slot_bytes);
    int *status = g.status;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;

    // k-block kb of a stage's tile t into ring slot i: the weights' boxes, and B's for stage 0.
    // Weights lie (hi, lo) for a chunk summed in [d0 | c], (lo, hi) for one in [c | d1].
    auto load = [&](int st, int blk, int t, int kb, int i, bool lo_first) {
        const ColStage &cs = g.st[st];
        const int w_bytes = cs.rows * 128;
        uint8_t *p = smem + i * g.slot_bytes;
        mbar_arrive_expect_tx(&bars->full[i], 2u * w_bytes + (st == 0 ? kCXBytes : 0));
        if (st == 0) tma_load_2d(p, &g.tm_x, &bars->full[i], blk * kCBN, kb * kCBK);
        tma_load_2d(p + kCXBytes, lo_first ? &cs.tm_lo : &cs.tm_hi, &bars->full[i], kb * kCBK, t * cs.rows);
        tma_load_2d(p + kCXBytes + w_bytes, lo_first ? &cs.tm_hi : &cs.tm_lo, &bars->full[i], kb * kCBK,
                    t * cs.rows);
    };
    auto chunk_blocks = [&](int st) {
        const int nkb = (g.st[st].K + kCBK - 1) / kCBK;
        return g.st[st].kchunk > 0 ? g.st[st].kchunk : nkb;
    };
    const int first_loads = min(g.ring, (g.st[0].K + kCBK - 1) / kCBK);

    if (threadIdx.x == 0) {
        for (int r = 0; r < kCMaxRing; ++r) {
            mbar_init(&bars->full[r], 1);
            mbar_init(&bars->empty[r], 5);
        }
        for (int r = 0; r < kCMaxGran; ++r) {
            mbar_init(&bars->afull[r], 4);
            mbar_init(&bars->aempty[r], 1);
        }
        for (int d = 0; d < 2; ++d) {
            mbar_init(&bars->dfull[d], 1);
            mbar_init(&bars->dempty[d], EW);
        }
        mbar_init(&bars->cfull, 1);
        mbar_init(&bars->drained, EW);
        mbar_init(&bars->xready, EW);
        mbar_init(&bars->mma_done, 1);
        bars->abort = 0;
        fence_mbar_init();
        // the ring's first round needs no wait, and nobody else: under way before the
        // CTA meets, and before the later stages' tensor maps are fetched
        overlap_wait();
        for (int kb = 0; kb < first_loads; ++kb)
            load(0, blockIdx.x, 0, kb, kb, (kb / chunk_blocks(0)) & 1);
        for (int i = 1; i < g.n; ++i) {
            tma_prefetch_desc(&g.st[i].tm_hi);
            tma_prefetch_desc(&g.st[i].tm_lo);
        }
    }
    if (warp == 1) tmem_alloc(&bars->tmem_base, g.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    overlap_next();
    overlap_wait();

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            RingPos s;
            uint32_t pending = (1u << first_loads) - 1, pending_ph = 0;
            int skip = first_loads;
            uint32_t chunks = 0;  // chunks of the tiles before
            for (int blk = blockIdx.x; blk < g.nblocks; blk += gridDim.x) {
                for (int st = 0; st < g.n; ++st) {
                    const int nkb = (g.st[st].K + kCBK - 1) / kCBK, kchunk = chunk_blocks(st);
                    for (int t = 0; t < g.st[st].tiles; ++t, chunks += (nkb + kchunk - 1) / kchunk)
                        for (int kb = 0; kb < nkb; ++kb, s.next(g.ring)) {
                            if (skip > 0) {  // loaded above
                                --skip;
                                continue;
                            }
                            if (!mbar_wait(&bars->empty[s.i], s.ph ^ 1, status, KERR_WAIT_EMPTY)) {
                                c_set_abort(bars);
                                goto producer_done;
                            }
                            load(st, blk, t, kb, s.i, (chunks + kb / kchunk) & 1u);
                            pending |= 1u << s.i;
                            pending_ph = (pending_ph & ~(1u << s.i)) | (s.ph << s.i);
                        }
                }
                if (c_aborted(bars)) break;
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
            RingPos s, a;
            uint32_t chunks = 0;  // chunk sums started: buffer chunks & 1, round chunks >> 1
            uint32_t tiles = 0, xr = 0;
            const uint64_t w_desc0 = smem_desc(smem_u32(smem) + kCXBytes, 16, 1024, SMEM_SW128);
            const uint32_t w_hi32 = (uint32_t)(w_desc0 >> 32);  // descriptors differ in the low word
            const bool whole = g.gran_k == 32;  // a granule is a k-block
            bool ok = true;
            for (int blk = blockIdx.x; ok && blk < g.nblocks; blk += gridDim.x) {
                for (int st = 0; ok && st < g.n; ++st) {
                    const ColStage &cs = g.st[st];
                    const int K = cs.K, rows = cs.rows, ntiles = cs.tiles;
                    const int nkb = (K + kCBK - 1) / kCBK;
                    const int kchunk = chunk_blocks(st);
                    const bool stack = cs.stack, first = st == 0;
                    const uint32_t idesc = make_idesc(1, 2, 2, 0, 0, kCBN, rows);
                    const uint32_t idesc2 = make_idesc(1, 2, 2, 0, 0, kCBN, stack ? 2 * rows : rows);
                    const uint32_t half = (uint32_t)(rows * 128) >> 4;
                    const uint32_t acc = tmem_base + cs.acc, c_tmem = acc + rows;
                    const uint32_t x_rows = first ? 0u : (uint32_t)g.st[st - 1].rows;
                    if (!first) {
                        ok = mbar_wait(&bars->xready, xr & 1u, status, KERR_WAIT_FULL);
                        ++xr;
                    }
                    // the barrier that says a k-block's operands are in place: its granule (the
                    // splitters waited for the slot's bytes, weights included) or its slot
                    auto ready_bar = [&](bool next) -> uint64_t * {
                        const RingPos &r = first ? a : s;
                        const int n = first ? g.gran : g.ring;
                        const int i = !next ? r.i : r.i + 1 == n ? 0 : r.i + 1;
                        return first ? &bars->afull[i] : &bars->full[i];
                    };
                    auto ready_ph = [&](bool next) -> uint32_t {
                        const RingPos &r = first ? a : s;
                        const int n = first ? g.gran : g.ring;
                        return next && r.i + 1 == n ? r.ph ^ 1 : r.ph;
                    };
                    for (int t = 0; ok && t < ntiles; ++t, ++tiles) {
                        // the accumulators (and what overlies them) are free once the tile before is read
                        if (!(ok = mbar_wait(&bars->drained, (tiles & 1u) ^ 1u, status, KERR_WAIT_ACC_EMPTY)))
                            break;
                        uint32_t more_c = 0, d_tmem = acc, s_tmem = acc, hi_off = 0, lo_off = half;
                        int left = 0;  // k-blocks left of the chunk
                        bool ready = false, free_d = false;  // waits found to be over ahead of time
                        for (int kb = 0; kb < nkb; ++kb) {
                            const bool begin = left == 0;
                            if (begin) {
                                const uint32_t b = chunks & 1u;
                                if (!free_d && !(ok = mbar_wait(&bars->dempty[b], ((chunks >> 1) & 1u) ^ 1u,
                                                                status, KERR_WAIT_ACC_EMPTY)))
                                    break;
                                free_d = false;
                                d_tmem = acc + (b ? 2 * rows : 0);
                                s_tmem = b ? c_tmem : acc;  // [c | d1] or [d0 | c]
                                hi_off = b ? half : 0;
                                lo_off = b ? 0 : half;
                                left = kchunk;
                            }
                            const uint32_t w0 = (uint32_t)w_desc0 + ((uint32_t)(s.i * g.slot_bytes) >> 4);
                            const uint32_t wh = w0 + hi_off, wl = w0 + lo_off;
                            const int left_k = K - kb * kCBK;
                            // step k of 8: A's columns at x (hi) and xl (lo), the weights' bytes 32 k on
                            auto step3 = [&](uint32_t x, uint32_t xl, int k, uint32_t more_d) {
                                tc_mma_ts_tf32(c_tmem, xl, wh + 2 * k, w_hi32, idesc, more_c);
                                tc_mma_ts_tf32(c_tmem, x, wl + 2 * k, w_hi32, idesc, 1);
                                tc_mma_ts_tf32(d_tmem, x, wh + 2 * k, w_hi32, idesc, more_d);
                                more_c = 1;
                            };
                            if (first && !whole) {
                                for (int k0 = 0; k0 < 4 && k0 * 8 < left_k; k0 += 2) {
                                    if (!ready &&
                                        !(ok = mbar_wait(&bars->afull[a.i], a.ph, status, KERR_WAIT_FULL)))
                                        break;
                                    tc_fence_after();
                                    ready = mbar_test(ready_bar(true), ready_ph(true));
                                    const uint32_t x = tmem_base + g.gran0 + a.i * 32;
                                    step3(x, x + 16, k0, !begin || k0);
                                    if (k0 * 8 + 8 < left_k) step3(x + 8, x + 24, k0 + 1, 1);
                                    tc_commit(&bars->aempty[a.i]);
                                    a.next(g.gran);
                                }
                                if (!ok) break;
                            } else {
                                if (!ready && !(ok = mbar_wait(ready_bar(false), ready_ph(false), status,
                                                               KERR_WAIT_FULL)))
                                    break;
                                tc_fence_after();
                                // asked now, looked at after this k-block's MMAs are issued
                                ready = mbar_test(ready_bar(true), ready_ph(true));
                                // hi at column 0 and lo after the previous stage's padded rows, or a granule
                                const uint32_t x = tmem_base + (first ? g.gran0 + a.i * 64 : kb * kCBK);
                                const uint32_t xl = x + (first ? (uint32_t)kCBK : x_rows);
                                auto step2 = [&](int k) {
                                    tc_mma_ts_tf32(c_tmem, xl + 8 * k, wh + 2 * k, w_hi32, idesc, 1);
                                    tc_mma_ts_tf32(s_tmem, x + 8 * k, w0 + 2 * k, w_hi32, idesc2, 1);
                                };
                                // a chunk's first step starts its sum, while the correction runs on
                                if (begin || !stack)
                                    step3(x, xl, 0, !begin);
                                else
                                    step2(0);
                                if (stack && left_k >= kCBK) {
#pragma unroll
                                    for (int k = 1; k < 4; ++k) step2(k);
                                } else if (left_k >= kCBK) {
#pragma unroll
                                    for (int k = 1; k < 4; ++k) step3(x + 8 * k, xl + 8 * k, k, 1);
                                } else {
                                    for (int k = 1; k * 8 < left_k; ++k) step3(x + 8 * k, xl + 8 * k, k, 1);
                                }
                                if (first) a.next(g.gran);
                            }
                            tc_commit(&bars->empty[s.i]);
                            s.next(g.ring);
                            if (--left == 0 || kb + 1 == nkb) {
                                tc_commit(&bars->dfull[chunks & 1u]);
                                ++chunks;
                                left = 0;
                                if (kb + 1 < nkb) free_d = mbar_test(&bars->dempty[chunks & 1u], ((chunks >> 1) & 1u) ^ 1u);
                            }
                        }
                        if (!ok) break;
                        tc_commit(&bars->cfull);
                    }
                }
                if (c_aborted(bars)) break;
            }
            if (!ok) c_set_abort(bars);
            tc_commit(&bars->mma_done);
            mbar_wait(&bars->mma_done, 0, status, KERR_WAIT_FULL);
        }
    } else if (warp < 6) {
        // ------------------------------------------------------------ splitters
        const int quarter = warp & 3;  // TMEM lanes this warp may access
        const uint32_t t_lane = (uint32_t)(quarter * 32) << 16;
        RingPos s, a;
        const int gran_cols = 2 * g.gran_k;
        bool ok = true;
        // G k of this thread's column into the next granule: hi, then lo, once the MMAs
        // that read it last have retired (free: that is known)
        auto put = [&](const float *x, auto g_tag, uint64_t *used, uint32_t used_ph, bool free) -> bool {
            constexpr int G = decltype(g_tag)::value;
            uint32_t h[G], l[G];
#pragma unroll
            for (int k = 0; k < G; ++k) {
                const float v = x[k * kCBN], hf = f32_to_tf32_rne(v);
                h[k] = __float_as_uint(hf);
                l[k] = __float_as_uint(f32_to_tf32_rne(v - hf));
            }
            if (!free && !mbar_wait(used, used_ph, status, KERR_WAIT_EMPTY)) return false;
            tc_fence_after();
            const uint32_t to = tmem_base + g.gran0 + a.i * gran_cols + t_lane;
            if constexpr (G == 32) {
                tmem_st_32x32b_x32(to, h);
                tmem_st_32x32b_x32(to + 32, l);
            } else {
                tmem_st_32x32b_x16(to, h);
                tmem_st_32x32b_x16(to + 16, l);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->afull[a.i]);
            a.next(g.gran);
            return true;
        };
        // The k-block that used a whole granule before: g.gran rounds ago in this block's first
        // stage, else in the last block's, its later rounds in between. Its slot's empty
        // barrier says when its MMAs have retired; further back than the ring is long,
        // the slot has been filled anew and waited for since.
        for (int blk = blockIdx.x; ok && blk < g.nblocks; blk += gridDim.x) {
            for (int st = 0; ok && st < g.n; ++st) {
                const int K = g.st[st].K, nkb = (K + kCBK - 1) / kCBK;
                const int rounds = g.st[st].tiles * nkb;
                for (int i = 0; i < rounds; ++i) {
                    // every round of every slot is waited for and released, also those
                    // without input: a parity tells two rounds apart, not three
                    if (!(ok = mbar_wait(&bars->full[s.i], s.ph, status, KERR_WAIT_FULL))) break;
                    if (st == 0) {  // one tile: i is the k-block (rows past K are zeros)
                        const float *x = reinterpret_cast<const float *>(smem + s.i * g.slot_bytes) +
                                         quarter * 32 + lane;
                        if (g.gran_k == 32) {
                            const int back = g.gran + (i < g.gran ? g.later_rounds : 0);
                            const bool free = (blk == (int)blockIdx.x && i < g.gran) || back > g.ring;
                            // round s - back: the ring is at least as long, so at most one turn ago
                            int j = s.i - back;
                            uint32_t ph = s.ph;
                            if (j < 0) {
                                j += g.ring;
                                ph ^= 1;
                            }
                            ok = put(x, std::integral_constant<int, 32>{}, &bars->empty[free ? 0 : j], ph, free);
                        } else {
                            ok = put(x, std::integral_constant<int, 16>{}, &bars->aempty[a.i], a.ph ^ 1, false);
                            if (ok && K - i * kCBK > 16)
                                ok = put(x + 16 * kCBN, std::integral_constant<int, 16>{}, &bars->aempty[a.i],
                                         a.ph ^ 1, false);
                        }
                        if (!ok) break;
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars->empty[s.i]);
                    s.next(g.ring);
                }
            }
            if (c_aborted(bars)) break;
        }
        if (!ok) c_set_abort(bars);
    } else {
        // ------------------------------------------------------------ epilogues
        const int quarter = warp & 3;
        constexpr int STEP = EW / 4;              // warps that share a lane quarter
        const int first = (warp - 6) >> 2;        // this warp's 16-row groups: first, first + STEP, ...
        const uint32_t t_lane = (uint32_t)(quarter * 32) << 16;
        uint32_t chunks = 0, tiles = 0;
        bool ok = true;
        for (int blk = blockIdx.x; ok && blk < g.nblocks; blk += gridDim.x) {
            const int col = blk * kCBN + quarter * 32 + lane;
            for (int st = 0; ok && st < g.n; ++st) {
                const ColStage &cs = g.st[st];
                const int nkb = (cs.K + kCBK - 1) / kCBK;
                const int kchunk = cs.kchunk > 0 ? cs.kchunk : nkb;
                const int nchunk = (nkb + kchunk - 1) / kchunk;
                const int groups = cs.rows / 16;
                const uint32_t acc = tmem_base + cs.acc + t_lane;
                for (int t = 0; ok && t < cs.tiles; ++t, ++tiles) {
                    float sum[16 * NG];
#pragma unroll
                    for (int j = 0; j < 16 * NG; ++j) sum[j] = 0.f;
                    auto add = [&](uint32_t from) {
#pragma unroll
                        for (int i = 0; i < NG; ++i)
                            if (first + i * STEP < groups) {
                                uint32_t v[16];
                                tmem_ld_32x32b_x16(from + (first + i * STEP) * 16, v);
                                tmem_ld_wait();
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    sum[i * 16 + j] = sum[i * 16 + j] + __uint_as_float(v[j]);
                            }
                    };
                    for (int i = 0; i < nchunk; ++i, ++chunks) {
                        const uint32_t b = chunks & 1u;
                        if (!(ok = mbar_wait(&bars->dfull[b], (chunks >> 1) & 1u, status, KERR_WAIT_ACC_FULL)))
                            break;
                        tc_fence_after();
                        add(acc + (b ? 2 * cs.rows : 0));
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars->dempty[b]);
                    }
                    if (!ok || !(ok = mbar_wait(&bars->cfull, tiles & 1u, status, KERR_WAIT_ACC_FULL))) break;
                    tc_fence_after();
                    add(acc + cs.rows);
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars->drained);
                    if (st + 1 < g.n) {
                        // this column of the next stage's A: hi, then lo (rows past M are the
                        // zero products of zero-filled weights). It may overlie sums that the
                        // other warp of these lanes still reads.
                        if (STEP > 1 &&
                            !(ok = mbar_wait(&bars->drained, tiles & 1u, status, KERR_WAIT_ACC_FULL)))
                            break;
                        const uint32_t x = tmem_base + t_lane;
#pragma unroll
                        for (int i = 0; i < NG; ++i)
                            if (first + i * STEP < groups) {
                                uint32_t h[16], l[16];
#pragma unroll
                                for (int j = 0; j < 16; ++j) {
                                    const float hf = f32_to_tf32_rne(sum[i * 16 + j]);
                                    h[j] = __float_as_uint(hf);
                                    l[j] = __float_as_uint(f32_to_tf32_rne(sum[i * 16 + j] - hf));
                                }
                                const uint32_t at = x + (first + i * STEP) * 16;
                                tmem_st_32x32b_x16(at, h);
                                tmem_st_32x32b_x16(at + cs.rows, l);
                            }
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&bars->xready);
                    } else if (col < g.N) {
                        // rows of C: a warp stores 32 consecutive columns at a time
                        // (a running pointer, and no test per row where all 16 are there: with
                        // both a row costs 85 clocks instead of 34)
#pragma unroll
                        for (int i = 0; i < NG; ++i) {
                            const int r0 = (first + i * STEP) * 16;  // row in the tile
                            const int m = min(cs.rows, cs.M - t * cs.rows) - r0;
                            float *cp = g.C + (size_t)(t * cs.rows + r0) * g.ldc + col;
                            if (m >= 16) {
#pragma unroll
                                for (int j = 0; j < 16; ++j, cp += g.ldc) *cp = sum[i * 16 + j];
                            } else if (m > 0) {
#pragma unroll
                                for (int j = 0; j < 16; ++j, cp += g.ldc)
                                    if (j < m) *cp = sum[i * 16 + j];
                            }
                        }
                    }
                }
            }
            if (c_aborted(bars)) break;
        }
        if (!ok) c_set_abort(bars);
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

// Tiles, TMEM columns and rings of a chain on one of the two builds; false where it
// does not fit.
bool column_layout(int n, const long *M, const long *K, bool small, ColArgs &A)
{
    const int rows_max = small ? kCSmallRows : kCRows;
    const int cols = small ? 256 : 512;
    const int usable = cols - 2 * 32;  // at least two granules of 16 k
    int end = 0, widest = 0, later = 0;
    for (int i = 0; i < n; ++i) {
        ColStage &cs = A.st[i];
        cs.M = (int)M[i];
        cs.K = (int)K[i];
        cs.acc = i > 0 ? 2 * A.st[i - 1].rows : 0;
        cs.tiles = 1;
        if (i + 1 < n) {
            if (M[i] > rows_max) return false;
            cs.rows = pad16(M[i]);
        } else {
            const int most = std::min(rows_max, (usable - cs.acc) / 3 / 16 * 16);
            // a first stage that is the last would stream B once per tile
            if (most < 16 || (n == 1 && M[i] > most)) return false;
            cs.tiles = (int)((M[i] + most - 1) / most);
            cs.rows = pad16((M[i] + cs.tiles - 1) / cs.tiles);
        }
        cs.stack = cs.rows <= 128;
        end = std::max(end, cs.acc + 3 * cs.rows);
        if (i > 0) later += cs.tiles * ((cs.K + kCBK - 1) / kCBK);
        widest = std::max(widest, cs.rows);
    }
    if (end > usable) return false;
    A.n = n;
    A.tmem_cols = cols;
    A.gran0 = end;
    A.gran_k = cols - end >= 2 * 64 ? 32 : 16;  // whole k-blocks where two of them fit
    A.gran = std::min(kCMaxGran, (cols - end) / (2 * A.gran_k));
    A.slot_bytes = kCXBytes + 2 * widest * 128;
    A.ring = std::min(kCMaxRing, ((small ? kCHalfSmem : kCMaxSmem) - kCFixed) / A.slot_bytes);
    A.smem = A.ring * A.slot_bytes + kCFixed;
    A.small = small;
    A.later_rounds = later;
    // a granule's last use is looked up at most one turn of the ring back
    if (A.gran_k == 32) A.gran = std::min(A.gran, A.ring);
    return A.ring >= 3;
}

bool column_layout(int n, const long *M, const long *K, ColArgs &A)
{
    return column_layout(n, M, K, true, A) || column_layout(n, M, K, false, A);
}

}  // namespace

// Microseconds of both ways, fitted to measurements on B200 of 436 random chains of 2 to 5
// stages (N = 16 to 65536, K_1 = 16 to 8400, registered weights). Here every SM runs whole
// blocks, a block's stages one after the other: a k-block of the first stage takes 0.62 (16-deep
// granules: 0.92), which a few blocks cannot share. The launch-per-stage path splits B
// through memory (12 bytes a value) and then spreads 128 x 128 tiles of each stage over all
// SMs, a k-block in 0.52, a stage's launch and drain in 6.6. So deep first stages and tall
// last ones on few columns stay there. Measured, column / stages: N = 64, K_1 = 3524, rows
// 32, 792 138 / 72; N = 96, 5276, 20, 560 183 / 102; N = 144, 5276, 48, 36, 268 114 / 117;
// N = 6624, 3532, 12, 64 77 / 130. The lower one is the faster at all but 5 of the 436, and
// within 11 % there. First stages of 129 to 144 rows and K_1 <= 2080 stay here up to 1.5 times
// the other estimate, in one launch as tests/test_gpu_column.py has them: N = 640, 2050, 144,
// 144 82 / 58, N = 900, 864, 130 33 / 25.
bool column_preferred(long N, int n, const long *M, const long *K, int num_sms)
{
    if (n < 1 || n > kPanelMaxStages || N < 1 || N > (1l << 30)) return false;
    for (int i = 0; i < n; ++i)
        if (M[i] < 1 || K[i] < 1 || M[i] > (1l << 30) || K[i] > (1l << 30)) return false;
    static thread_local ColArgs A;
    if (!column_layout(n, M, K, A)) return false;
    const double blocks = (double)((N + kCBN - 1) / kCBN), mb = 1e-6;
    const bool whole = A.gran_k == 32, shared = A.small && blocks > num_sms;
    double block = 0.0, staged = 2.2 + 0.218 * mb * 12.0 * K[0] * N;
    for (int i = 0; i < n; ++i) {
        const ColStage &cs = A.st[i];
        const double kb = (cs.K + kCBK - 1) / kCBK;
        const double per_kb = i > 0 ? 0.71 : !whole ? 0.92 + 0.0004 * cs.rows : shared ? 0.66 : 0.62;
        block += 0.67 + (cs.tiles - 1) * 0.21 + cs.tiles * (kb * per_kb + 0.0085 * cs.rows);
        const double waves = std::ceil((double)((M[i] + 127) / 128) * blocks / num_sms);
        staged += 6.6 + waves * kb * 0.52 + (waves - 1.0) * 2.0 + 0.0104 * mb * 12.0 * M[i] * N;
    }
    const double rounds = std::ceil(blocks / (num_sms * (A.small ? 2.0 : 1.0)));
    const double here = 3.4 + rounds * block + 0.028 * mb * 4.0 * (K[0] + M[n - 1]) * N;
    return here < staged * (A.st[0].rows > 128 && K[0] <= 2080 ? 1.5 : 1.0);
}

cudaError_t launch_column(const PanelChainArgs &a, int num_sms, int *status, cudaStream_t s)
{
    // launch parameters of the last few operand sets (tensor maps encoded once)
    static std::mutex mu;
    struct Built {
        PanelChainArgs key;
        ColArgs g;
    };
    static std::vector<std::unique_ptr<Built>> built;
    static unsigned long long known = 0;
    static thread_local ColArgs g;
    {
        std::lock_guard<std::mutex> lk(mu);
        int dev = 0;
        cudaGetDevice(&dev);
        if (!(known >> (dev & 63) & 1)) {
            cudaError_t e = cudaFuncSetAttribute(tc_column_kernel<kCSmallRows / 16, 4, 2>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, kCHalfSmem);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(tc_column_kernel<(kCRows / 16 + 1) / 2, 8, 1>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kCMaxSmem);
            if (e != cudaSuccess) return e;
            known |= 1ull << (dev & 63);
        }
        Built *hit = nullptr;
        for (size_t i = 0; i < built.size(); ++i)
            if (memcmp(&built[i]->key, &a, sizeof a) == 0 && built[i]->g.status == status) {
                std::unique_ptr<Built> b = std::move(built[i]);
                built.erase(built.begin() + i);
                built.push_back(std::move(b));
                hit = built.back().get();
                break;
            }
        if (!hit) {
            std::unique_ptr<Built> b(new Built);
            memcpy(&b->key, &a, sizeof a);
            memset(&b->g, 0, sizeof b->g);
            ColArgs &A = b->g;
            if (!column_layout(a.n, a.M, a.K, A)) return cudaErrorNotSupported;
            if (!make_map(&A.tm_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.B, a.K[0], a.N, a.ldb, kCBN, kCBK,
                          CU_TENSOR_MAP_SWIZZLE_NONE))
                return cudaErrorNotSupported;
            for (int i = 0; i < a.n; ++i) {
                ColStage &cs = A.st[i];
                cs.kchunk = a.kchunk[i];
                if (!make_map(&cs.tm_hi, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.w_hi[i], a.M[i], a.K[i],
                              a.ldw[i], kCBK, cs.rows) ||
                    !make_map(&cs.tm_lo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.w_lo[i], a.M[i], a.K[i],
                              a.ldw[i], kCBK, cs.rows))
                    return cudaErrorNotSupported;
            }
            A.C = a.C;
            A.ldc = a.ldc;
            A.N = (int)a.N;
            A.nblocks = (int)((a.N + kCBN - 1) / kCBN);
            A.status = status;
            if (built.size() >= 8) built.erase(built.begin());
            built.push_back(std::move(b));
            hit = built.back().get();
        }
        g = hit->g;  // a copy: the entry may go once the lock is released
    }
    const int grid = std::min(g.nblocks, num_sms * (g.small ? 2 : 1));
    return g.small ? launch_overlapped(tc_column_kernel<kCSmallRows / 16, 4, 2>, dim3(grid), c_threads(4),
                                       g.smem, s, g)
                   : launch_overlapped(tc_column_kernel<(kCRows / 16 + 1) / 2, 8, 1>, dim3(grid),
                                       c_threads(8), g.smem, s, g);
}

}  // namespace fg
