// Tail of a DepthConvBlock (layers.py:115-159, layers_proxy.cpp:71-101) on tcgen05, CTA pairs:
//
//   x   = a . W0^T + b0 + r                               (dc.3 + shortcut; absent when cdc = 0)
//   t   = sum_{k<4} WSiLU(x . W1[4c+k]^T + b1[4c+k])      (ffn.0 + chunk add)
//   out = (t . W2^T + b2 + x) [* qscale]                  (ffn.2 + shortcut)
//
// As three launches the block's tail moves x and t through memory twice each and re-reads every
// weight tile for every 128-row tile: the quad GEMM alone then asks L2 for 400 MB in 26 us at
// 1080p (96 bytes per SM and clock at the MMA's rate), which bounds it, not the tensor cores.
// Here a pair of CTAs owns 256 rows: x stays in shared memory (128 rows per CTA, laid out as the
// swizzled A operand of ffn.0 and rewritten in place by both residual epilogues), t stays in
// tensor memory (the A operand of ffn.2), and each CTA stages half of every weight tile, so the
// weights cross L2 once per 256 rows.
//
// Per tile the MMA warp of the even CTA walks blocks of 128 output columns - dc.3's, ffn.0's, ffn.2's -
// each into one of three accumulators while sixteen epilogue warps drain the blocks before.  An MMA of
// this shape reads 4 KB of activations and 2 KB of weights from each SM's shared memory in 64 clocks and
// the weight copies write as much again, so the blocks use up most of shared memory's 128 bytes a
// clock (measured 70 clocks an MMA); 192-wide blocks in two accumulators leave the epilogues too few
// registers and take half as long again (75 us against 50 at 32640 pixels), 256-wide ones would leave no
// tensor memory for t.  The FP32 sums run over K in the same order as in the separate GEMMs and each
// epilogue applies the same operations in the same order, with x and t rounded to 16 bits where the
// separate launches stored them, so the result is bitwise theirs.
#include "dcb_sm100.cuh"

#include "gemm_sm100.cuh"
#include "host_util.h"

#include <cstring>
#include <mutex>
#include <type_traits>

namespace dcvc {

namespace {

constexpr int kRows = 128;              // rows per CTA (256 per pair)
constexpr int kNB = 128;                // output columns per block
constexpr int kAccs = 3;                // accumulators
constexpr int kSlabBytes = kRows * 128; // 64 16-bit columns of 128 rows
constexpr int kStageTiles = 2;          // 64-column K tiles per ring stage
constexpr int kTileBytes = kNB / 2 * 128;   // this CTA's half of a block's weight rows
constexpr int kStageBytes = kStageTiles * kTileBytes;
constexpr int kEpiWarps = 16;
constexpr int kFirstEpiWarp = 3;        // warps 0: weights, 1: MMA, 2: activations
constexpr int kThreads = 32 * (kFirstEpiWarp + kEpiWarps);
constexpr int kTmemCols = 512;
constexpr int kAccCol = 128;            // tensor memory: t in columns 0 .. 127, then the accumulators
constexpr long long kWaitLimit = 2000000000LL;  // ~1 s at 2 GHz
constexpr int kSmemLimit = 232448;
constexpr int kBarBytes = 1024;

template <typename T>
struct Act16;
template <>
struct Act16<__half> {
    static constexpr int kFormat = 0;
    static __device__ __forceinline__ uint32_t pack(float a, float b)
    {
        const __half2 h = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t u) { return __half22float2(*reinterpret_cast<__half2*>(&u)); }
};
template <>
struct Act16<__nv_bfloat16> {
    static constexpr int kFormat = 1;
    static __device__ __forceinline__ uint32_t pack(float a, float b)
    {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t*>(&h);
    }
    static __device__ __forceinline__ float2 unpack(uint32_t u)
    {
        return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
    }
};

// C, K0 = cdc (0: no dc.3), F = cffn.
template <int C, int K0, int F>
struct TailCfg {
    static constexpr int kXSlabs = C / 64;
    static constexpr int kASlabs = K0 / 64;
    static constexpr int kBlocksC = C / kNB;      // blocks of dc.3 and of ffn.2
    static constexpr int kBlocksT = 4 * F / kNB;  // blocks of ffn.0
    // The dc.3 operand has its own slabs where shared memory allows (its next tile then loads
    // while this one computes); else it sits in the upper x slabs.
    static constexpr bool kOwnA = K0 > 0 && (kXSlabs + kASlabs) * kSlabBytes <= 128 * 1024;
    [[maybe_unused]] static constexpr int kAFirst = kOwnA ? kXSlabs : kXSlabs - kASlabs;  // slab of the operand
    static constexpr int kSlabs = kXSlabs + (kOwnA ? kASlabs : 0);
    static constexpr int kRingOffset = kSlabs * kSlabBytes;
    static constexpr int kB1 = K0 > 0 ? C : 0, kB2 = kB1 + 4 * F;  // biases in shared memory: b0, b1, b2
    static constexpr int kBiasBytes = (kB2 + C) * 4;
    static constexpr int kStagesFit = (kSmemLimit - 1024 - kBarBytes - kBiasBytes - kRingOffset) / kStageBytes;
    static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
    static constexpr int kBarOffset = kRingOffset + kStages * kStageBytes;
    static constexpr int kBiasOffset = kBarOffset + kBarBytes;
    static constexpr int kBytes = kBiasOffset + kBiasBytes + 1024;
    static constexpr int kTStages = F / 128;
    static constexpr int kXStages = C / 128;     // 128 columns of x: what one stage of ffn.0 reads
    static constexpr int kBars = 2 * kStages + 2 * kAccs + 2 + kASlabs + kXStages + 2 * kXSlabs + kTStages;
    static_assert((C == 256 || C == 512) && K0 % 128 == 0 && (F == 128 || F == 256), "channel counts");
    static_assert(kAccCol >= F / 2 && kAccCol + kAccs * kNB <= kTmemCols, "tensor memory");
    static_assert(K0 == 0 || kOwnA || 2 * K0 <= C, "dc.3 operand in the upper half of x");
    static_assert(kStages >= 3 && kBytes <= kSmemLimit && kBars * 8 + 8 <= kBarBytes, "shared memory");
    static_assert(kBytes >= kTmemCtaMinSmem, "one CTA per SM");
    // ffn.2's blocks in the order that frees the dc.3 operand's slabs first
    static __device__ __forceinline__ int out_block(int i)
    {
        return K0 > 0 && !kOwnA ? (i + kBlocksC / 2) % kBlocksC : i;
    }
};

// Byte offset of the 16-byte chunk j of row r in a 128-byte-swizzled slab.
__device__ __forceinline__ int sw128_off(int r, int j) { return r * 128 + ((j ^ (r & 7)) << 4); }

template <typename T, int C, int K0, int F>
__global__ void __launch_bounds__(kThreads, 1)
    dcb_tail_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmX,
                    const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                    const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmO,
                    const DcbTailParams p)
{
    using G = TailCfg<C, K0, F>;
    using P = Act16<T>;
    constexpr int kStages = G::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem =
        reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = smem + G::kRingOffset;
    // Barriers that collect arrivals of both CTAs live in the even CTA (marked E); commits of the
    // MMA warp arrive in both CTAs.
    uint64_t* wfull = reinterpret_cast<uint64_t*>(smem + G::kBarOffset);  // E: weight stage landed in both CTAs
    uint64_t* wempty = wfull + kStages;
    uint64_t* accfull = wempty + kStages;
    uint64_t* accempty = accfull + kAccs;  // E
    uint64_t* adone = accempty + kAccs;      // dc.3's MMAs of a tile have read the operand
    uint64_t* drain = adone + 1;
    uint64_t* afull = drain + 1;           // E: operand slab landed in both CTAs
    uint64_t* xfull = afull + G::kASlabs;  // E: 128 columns of x complete in both CTAs (cdc > 0: see pair_pass)
    uint64_t* xfree = xfull + G::kXStages; // output stored from the slab
    uint64_t* tfull = xfree + G::kXSlabs;  // E: 128 values of t complete in both CTAs
    uint64_t* rfull = tfull + G::kTStages; // residual slab landed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(rfull + G::kXSlabs);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const int num_tiles = (p.M + 2 * kRows - 1) / (2 * kRows);
    const int unit = static_cast<int>(blockIdx.x >> 1);
    const int units = static_cast<int>(gridDim.x >> 1);
    const int row_off = static_cast<int>(rank) * kRows;
    // progress waits give up after `lim` cycles; the drains after an abort keep the full limit
    const long long lim = p.wait_limit > 0 ? p.wait_limit : kWaitLimit;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&wfull[s], 1);
            mbar_init(&wempty[s], 1);
        }
        for (int b = 0; b < kAccs; ++b) {
            mbar_init(&accfull[b], 1);
            mbar_init(&accempty[b], 2 * kEpiWarps);
        }
        mbar_init(adone, 1);
        mbar_init(drain, 1);
        for (int s = 0; s < G::kASlabs; ++s) {
            mbar_init(&afull[s], 1);
        }
        for (int s = 0; s < G::kXSlabs; ++s) {
            mbar_init(&rfull[s], 1);
            mbar_init(&xfree[s], 4);
        }
        for (int b = 0; b < G::kXStages; ++b) {
            // the four quadrants' warps of two slabs and the odd CTA's arrival for all of its, or two copies
            mbar_init(&xfull[b], K0 > 0 ? 8 + (rank == 0 ? 1 : 0) : 2);
        }
        for (int b = 0; b < G::kTStages; ++b) {
            mbar_init(&tfull[b], 4 * 2 * kEpiWarps);  // four blocks of ffn.0
        }
        *abort_flag = 0;
        fence_mbar_init();
    }
    const uint32_t tmem_base = pair_begin(tmem_slot, kTmemCols, warp == 1);
    griddep_launch_dependents();
    griddep_wait();

    auto fail = [&](int code) {
        *abort_flag = 1;
        report_error(p.err, code);
        return false;
    };

    if (warp == 0) {
        // ------------------------------------------------------------ weight tiles
        int stage = 0;
        uint32_t phase = 0;
        int issued = 0;
        // K columns 128 kb .. of block nb's weight rows: this CTA's half of them
        auto push = [&](const CUtensorMap* tm, int kb, int nb) {
            if (!mbar_wait_warp(&wempty[stage], phase ^ 1, lim)) {
                return fail(kErrGemmProducerTimeout);
            }
            if (elect_one()) {
                if (rank == 0) {
                    mbar_arrive_expect_tx(&wfull[stage], 2 * kStageBytes);  // both CTAs' halves
                }
                const uint32_t bar = cluster_map(&wfull[stage], 0);
#pragma unroll
                for (int t = 0; t < kStageTiles; ++t) {
                    tma_load_2d_pair(ring + stage * kStageBytes + t * kTileBytes, tm, bar, (kb * kStageTiles + t) * 64,
                                     nb * kNB + static_cast<int>(rank) * (kNB / 2));
                }
            }
            __syncwarp();
            ++issued;
            if (++stage == kStages) {
                stage = 0;
                phase ^= 1;
            }
            return true;
        };
        bool ok = true;
        for (int tile = unit; ok && tile < num_tiles && !warp_any(*abort_flag != 0); tile += units) {
            if constexpr (K0 > 0) {
                for (int nb = 0; ok && nb < G::kBlocksC; ++nb) {
                    for (int kb = 0; ok && kb < K0 / 128; ++kb) {
                        ok = push(&tmW0, kb, nb);
                    }
                }
            }
            for (int nb = 0; ok && nb < G::kBlocksT; ++nb) {
                for (int kb = 0; ok && kb < C / 128; ++kb) {
                    ok = push(&tmW1, kb, nb);
                }
            }
            for (int i = 0; ok && i < G::kBlocksC; ++i) {
                for (int kb = 0; ok && kb < F / 128; ++kb) {
                    ok = push(&tmW2, kb, G::out_block(i));
                }
            }
        }
        if (warp_any(*abort_flag != 0) && rank == 0) {
            // let the copies land before the CTA winds down
            for (int i = 0; i < (issued < kStages ? issued : kStages); ++i) {
                if (--stage < 0) {
                    stage = kStages - 1;
                    phase ^= 1;
                }
                mbar_wait_warp(&wfull[stage], phase, kWaitLimit / 16);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (even CTA)
        if (rank == 0) {
            const uint32_t idesc = make_idesc_f16(2 * kRows, kNB, P::kFormat);
            const uint32_t smem_addr = smem_u32(smem);
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool issued_any = false;
            auto need = [&](uint64_t* bar, uint32_t parity) {
                if (!mbar_wait_warp<true>(bar, parity, lim)) {
                    return fail(kErrGemmMmaTimeout);
                }
                tc_fence_after();
                return true;
            };
            // one stage (K columns 128 kb ..) of a block: the operand in slabs from `slab` on or
            // (slab < 0) in tensor memory
            auto kblock = [&](int slab, int kb) {
                if (!need(&wfull[stage], phase)) {
                    return false;
                }
                if (elect_one()) {
                    const uint32_t d = tmem_base + kAccCol + static_cast<uint32_t>(acc * kNB);
#pragma unroll
                    for (int t = 0; t < kStageTiles; ++t) {
                        const uint64_t bdesc = make_sw128_kmajor_desc(smem_addr + G::kRingOffset + stage * kStageBytes +
                                                                      t * kTileBytes);
                        if (slab >= 0) {
                            const uint64_t adesc = make_sw128_kmajor_desc(
                                smem_addr + (slab + kb * kStageTiles + t) * kSlabBytes);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                tc_mma_f16_pair(d, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | t | k) != 0 ? 1u : 0u);
                            }
                        } else {
                            const uint32_t ta = tmem_base + static_cast<uint32_t>((kb * kStageTiles + t) * 32);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                tc_mma_f16_pair_ts(d, ta + 8 * k, bdesc + 2 * k, idesc, (kb | t | k) != 0 ? 1u : 0u);
                            }
                        }
                    }
                    tc_commit_pair_both(&wempty[stage]);
                }
                __syncwarp();
                issued_any = true;
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1;
                }
                return true;
            };
            auto begin = [&] { return need(&accempty[acc], acc_phase ^ 1); };
            auto commit = [&](uint64_t* bar) {
                if (elect_one()) {
                    tc_commit_pair_both(bar);
                }
                __syncwarp();
            };
            auto finish = [&] {
                commit(&accfull[acc]);
                if (++acc == kAccs) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            };
            bool ok = p.stall_test == 0;
            uint32_t tp = 0;  // parity of the per-tile barriers
            for (int tile = unit; ok && tile < num_tiles && !warp_any(*abort_flag != 0); tile += units, tp ^= 1) {
                if constexpr (K0 > 0) {
                    for (int i = 0; ok && i < G::kBlocksC; ++i) {
                        ok = begin();
                        for (int kb = 0; ok && kb < K0 / 128; ++kb) {
                            for (int t = 0; ok && i == 0 && t < kStageTiles; ++t) {
                                ok = need(&afull[kb * kStageTiles + t], tp);
                            }
                            ok = ok && kblock(G::kAFirst, kb);
                        }
                        if (ok) {
                            finish();
                        }
                    }
                    if (ok) {
                        commit(adone);
                    }
                }
                for (int i = 0; ok && i < G::kBlocksT; ++i) {
                    ok = begin();
                    for (int kb = 0; ok && kb < C / 128; ++kb) {
                        ok = (i > 0 || need(&xfull[kb], tp)) && kblock(0, kb);
                    }
                    if (ok) {
                        finish();
                    }
                }
                for (int j = 0; ok && j < G::kBlocksC; ++j) {
                    ok = begin();
                    for (int kb = 0; ok && kb < F / 128; ++kb) {
                        ok = (j > 0 || need(&tfull[kb], tp)) && kblock(-1, kb);
                    }
                    if (ok) {
                        finish();
                    }
                }
            }
            if (warp_any(*abort_flag != 0) && issued_any) {
                if (elect_one()) {
                    tc_commit_pair_local(drain);
                }
                __syncwarp();
                mbar_wait_warp(drain, 0, kWaitLimit / 16);
            }
        } else if constexpr (K0 > 0) {
            // ---------------------------------------------------- the odd CTA's x, told to the even CTA
            const uint32_t even = cluster_map(smem, 0) - smem_u32(smem);
            bool ok = true;
            uint32_t tp = 0;
            for (int tile = unit; ok && tile < num_tiles && !warp_any(*abort_flag != 0); tile += units, tp ^= 1) {
                for (int b = 0; ok && b < G::kXStages; ++b) {
                    ok = pair_pass(&xfull[b], tp, even, lim) || fail(kErrGemmMmaTimeout);
                }
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ activation slabs
        uint32_t tp = 0;
        auto gate = [&](uint64_t* bar, uint32_t parity) {
            return mbar_wait_warp(bar, parity, lim) || fail(kErrGemmProducerTimeout);
        };
        // the barriers on which copies have been asked for, one bit each, and the parity of the last of them: what
        // has to land before the CTA winds down after an abort
        uint32_t copies = 0, copies_parity = 0, residuals = 0, residuals_parity = 0;
        auto note = [](uint32_t& set, uint32_t& par, int bit, uint32_t parity) {
            set |= 1u << bit;
            par = (par & ~(1u << bit)) | parity << bit;
        };
        // operand (afull) or ConvFFN input (xfull) slab of both CTAs, on barrier `i` of `bars`
        auto load = [&](const CUtensorMap* tm, uint64_t* bars, int i, uint32_t parity, int slab, int c, int m0) {
            if (elect_one()) {
                if (rank == 0) {
                    mbar_arrive_expect_tx(&bars[i], 2 * kSlabBytes);
                }
                tma_load_2d_pair(smem + slab * kSlabBytes, tm, cluster_map(&bars[i], 0), c, m0);
            }
            __syncwarp();
            note(copies, copies_parity, i, parity);
        };
        auto prefetch = [&](const CUtensorMap* tm, int slabs, int m0) {
            if (elect_one()) {
                for (int s = 0; s < slabs; ++s) {
                    tma_prefetch_2d(tm, s * 64, m0);
                }
            }
            __syncwarp();
        };
        auto load_residual = [&](int s, int m0) {
            if (elect_one()) {
                mbar_arrive_expect_tx(&rfull[s], kSlabBytes);
                tma_load_2d(smem + s * kSlabBytes, &tmX, &rfull[s], s * 64, m0);
            }
            __syncwarp();
            note(residuals, residuals_parity, s, tp);
        };
        bool ok = true;
        if constexpr (G::kOwnA) {
            for (int s = 0; s < G::kASlabs; ++s) {
                load(&tmA, afull, s, 0, G::kAFirst + s, s * 64, unit * 2 * kRows + row_off);
            }
        }
        for (int tile = unit; tile < num_tiles && ok && !warp_any(*abort_flag != 0); tile += units, tp ^= 1) {
            const int m0 = tile * 2 * kRows + row_off;
            const int m1 = m0 + units * 2 * kRows;  // this CTA's next tile
            const bool more = tile + units < num_tiles;
            if constexpr (K0 == 0) {
                for (int s = 0; ok && s < G::kXSlabs; ++s) {
                    ok = gate(&xfree[s], tp ^ 1);
                    if (ok) {
                        load(&tmX, xfull, s / 2, tp, s, s * 64, m0);
                    }
                }
            } else if constexpr (G::kOwnA) {
                for (int s = 0; ok && s < G::kXSlabs; ++s) {
                    ok = gate(&xfree[s], tp ^ 1);
                    if (ok) {
                        load_residual(s, m0);
                    }
                }
                if (more && ok) {
                    ok = gate(adone, tp);
                    for (int s = 0; ok && s < G::kASlabs; ++s) {
                        load(&tmA, afull, s, tp ^ 1, G::kAFirst + s, s * 64, m1);
                    }
                }
            } else {
                for (int s = 0; ok && s < G::kASlabs; ++s) {
                    ok = gate(&xfree[G::kAFirst + s], tp ^ 1);
                    if (ok) {
                        load(&tmA, afull, s, tp, G::kAFirst + s, s * 64, m0);
                    }
                }
                if (tile == unit) {
                    prefetch(&tmX, G::kXSlabs, m0);
                }
                for (int s = 0; ok && s < G::kAFirst; ++s) {
                    ok = gate(&xfree[s], tp ^ 1);
                    if (ok) {
                        load_residual(s, m0);
                    }
                }
                ok = ok && gate(adone, tp);
                for (int s = G::kAFirst; ok && s < G::kXSlabs; ++s) {
                    load_residual(s, m0);
                }
                if (more) {
                    prefetch(&tmA, G::kASlabs, m1);
                }
            }
            if (more) {
                prefetch(&tmX, G::kXSlabs, m1);
            }
        }
        if (warp_any(*abort_flag != 0)) {
            // let the copies land before the CTA winds down (those into both CTAs count on the even one's barriers)
            for (int s = 0; s < G::kXSlabs; ++s) {
                if ((residuals >> s) & 1u) {
                    mbar_wait_warp(&rfull[s], (residuals_parity >> s) & 1u, kWaitLimit / 16);
                }
                if (rank == 0 && ((copies >> s) & 1u)) {
                    mbar_wait_warp(K0 > 0 ? &afull[s] : &xfull[s], (copies_parity >> s) & 1u, kWaitLimit / 16);
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps
        const int quad = warp & 3;                      // TMEM lane quadrant this warp may access
        // ffn.0: which 32 of a block's 128 columns.  dc.3 and ffn.2: two sets of warps take blocks in
        // turn, a warp one slab (64 columns) of its block.
        const int grp = (warp - kFirstEpiWarp) >> 2;
        const int set = grp >> 1, side = grp & 1;
        const int row = quad * 32 + lane;               // this lane's row in the CTA's 128
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        int acc = 0;
        uint32_t acc_phase = 0;
        // arrivals on a barrier of the even CTA, after a __syncwarp
        const uint32_t even = cluster_map(smem, 0) - smem_u32(smem);
        auto arrive_tmem = [&](uint64_t* bar, uint32_t n) { mbar_arrive_tmem_if(lane == 0, smem_u32(bar) + even, n); };
        auto advance = [&] {
            if (++acc == kAccs) {
                acc = 0;
                acc_phase ^= 1;
            }
        };
        // The biases live in shared memory: with all but a few KB of the SM's memory taken by it, L1
        // holds next to nothing, and a bias (or a spilled register) read from L2 in every block
        // costs more than the rest of the block's arithmetic.
        float* bias = reinterpret_cast<float*>(smem + G::kBiasOffset);
        for (int i = threadIdx.x - 32 * kFirstEpiWarp; i < G::kB2 + C; i += 32 * kEpiWarps) {
            bias[i] = i < G::kB1 ? p.b0[i] : i < G::kB2 ? p.b1[i - G::kB1] : p.b2[i - G::kB2];
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
        const uint32_t smem_base = smem_u32(smem);
        uint32_t bias_addr;  // known from here on: reads of the biases cannot move above the barrier
        asm volatile("mov.u32 %0, %1;" : "=r"(bias_addr) : "r"(smem_u32(bias)) : "memory");
        auto wait_acc = [&] {
            if (!mbar_wait_warp(&accfull[acc], acc_phase, lim)) {
                return fail(kErrGemmEpilogueTimeout);
            }
            tc_fence_after();
            return true;
        };
        // frees the accumulator (for n of its 32 arrivals): this warp's loads from it are complete
        auto release_acc = [&](uint32_t n) {
            tc_fence_before();
            __syncwarp();
            arrive_tmem(&accempty[acc], n);
            advance();
        };
        auto load_acc = [&](uint32_t (&r)[32], int col) {
            tmem_ld_32x32b_x32(lane_base + kAccCol + acc * kNB + col, r);
        };
        // columns 8 j .. 8 j + 7 of loaded accumulators plus bias b
        auto add_bias = [&](float2 (&v)[4], const uint32_t (&r)[32], int j, int b) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float4 bj = lds128_const(bias_addr + (b + 8 * j + 4 * h) * 4);
                const int i = 8 * j + 4 * h;
                v[2 * h] = __fadd2_rn(make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])),
                                      make_float2(bj.x, bj.y));
                v[2 * h + 1] = __fadd2_rn(make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3])),
                                          make_float2(bj.z, bj.w));
            }
        };
        // The residual epilogue of this warp's slab of a block: acc + bias + the slab's row [* q], over
        // that row.  q: this lane's factors of the slab's columns (has_q: std::true_type; a run-time
        // test per value group costs as much as the rest of the group).
        auto residual_slab = [&](int s, int b, auto has_q, const T* q) {
            const uint32_t line = smem_base + s * kSlabBytes + row * 128;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                uint32_t r[32];
                uint4 u[4];
                load_acc(r, side * 64 + c * 32);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    u[j] = lds128(line + (((c * 4 + j) ^ (row & 7)) << 4));
                }
                tc_wait_ld();
                if (c == 1) {
                    release_acc(2);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float2 v[4];
                    add_bias(v, r, j, b + c * 32);
                    v[0] = __fadd2_rn(v[0], P::unpack(u[j].x));
                    v[1] = __fadd2_rn(v[1], P::unpack(u[j].y));
                    v[2] = __fadd2_rn(v[2], P::unpack(u[j].z));
                    v[3] = __fadd2_rn(v[3], P::unpack(u[j].w));
                    if constexpr (decltype(has_q)::value) {
                        const uint4 f = __ldg(reinterpret_cast<const uint4*>(q + c * 32 + j * 8));
                        v[0] = __fmul2_rn(v[0], P::unpack(f.x));
                        v[1] = __fmul2_rn(v[1], P::unpack(f.y));
                        v[2] = __fmul2_rn(v[2], P::unpack(f.z));
                        v[3] = __fmul2_rn(v[3], P::unpack(f.w));
                    }
                    sts128(line + (((c * 4 + j) ^ (row & 7)) << 4),
                           make_uint4(P::pack(v[0].x, v[0].y), P::pack(v[1].x, v[1].y), P::pack(v[2].x, v[2].y),
                                      P::pack(v[3].x, v[3].y)));
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
        };
        // xfree of the slab this warp stored last, once its store has read the slab
        int stored = -1;
        auto settle = [&] {
            bulk_wait_read0();  // lane 0 issued the store
            mbar_arrive_if(lane == 0 && stored >= 0, &xfree[stored >= 0 ? stored : 0]);
            stored = -1;
        };
        bool ok = true;
        uint32_t tp = 0;
        for (int tile = unit; ok && tile < num_tiles && !warp_any(*abort_flag != 0); tile += units, tp ^= 1) {
            const int row0 = tile * 2 * kRows + row_off + quad * 32;  // first row of this warp
            if constexpr (K0 > 0) {
                // dc.3: x = acc + b0 + residual, over the residual in its slab
#pragma unroll 1
                for (int nb = 0; ok && nb < G::kBlocksC; ++nb) {
                    if ((nb & 1) != set) {
                        advance();
                        continue;
                    }
                    const int s = nb * 2 + side;
                    if (!mbar_wait_warp(&rfull[s], tp, lim)) {
                        ok = fail(kErrGemmEpilogueTimeout);
                        break;
                    }
                    ok = wait_acc();
                    if (!ok) {
                        break;
                    }
                    residual_slab(s, s * 64, std::false_type{}, nullptr);
                    mbar_arrive_if(lane == 0, &xfull[s / 2]);
                }
            }
            // ffn.0: 32 columns -> 8 values of t per row, to tensor memory
#pragma unroll 1
            for (int nb = 0; ok && nb < G::kBlocksT; ++nb) {
                ok = wait_acc();
                if (!ok) {
                    break;
                }
                uint32_t r[32];
                load_acc(r, grp * 32);
                tc_wait_ld();
                release_acc(1);
                uint32_t o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float2 v[4];
                    add_bias(v, r, k, G::kB1 + nb * kNB + grp * 32);
                    const float2 w0 = wsilu2(v[0]), w1 = wsilu2(v[1]), w2 = wsilu2(v[2]), w3 = wsilu2(v[3]);
                    o[k] = P::pack(w0.x + w0.y + w1.x + w1.y, w2.x + w2.y + w3.x + w3.y);
                }
                tmem_st_32x32b_x4(lane_base + nb * (kNB / 8) + grp * 4, o);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                arrive_tmem(&tfull[nb / 4], 1);
            }
            // ffn.2: out = (acc + b2 + x) [* q], over x in its slab and stored from there
#pragma unroll 1
            for (int i = 0; ok && i < G::kBlocksC; ++i) {
                if ((i & 1) != set) {
                    advance();
                    continue;
                }
                const int s = G::out_block(i) * 2 + side;
                settle();
                ok = wait_acc();
                if (!ok) {
                    break;
                }
                if (p.qscale != nullptr) {
                    // this lane's row picks its image's factors in a packed batch
                    const int qm = min(row0 + lane, p.M - 1);
                    residual_slab(s, G::kB2 + s * 64, std::true_type{},
                                  reinterpret_cast<const T*>(p.qscale) +
                                      (p.q_rows > 0 ? static_cast<size_t>(qm / p.q_rows) * C : 0) + s * 64);
                } else {
                    residual_slab(s, G::kB2 + s * 64, std::false_type{}, nullptr);
                }
                tma_store_2d_if(lane == 0 && row0 < p.M, &tmO, smem_base + s * kSlabBytes + quad * 4096, s * 64, row0);
                bulk_commit();
                stored = s;
            }
            settle();
            __syncwarp();
        }
    }

    pair_end(tmem_base, kTmemCols, warp == 1);
}

template <typename T, int C, int K0, int F>
cudaError_t launch_tail(const CUtensorMap (&m)[6], const DcbTailParams& p, cudaStream_t stream)
{
    using G = TailCfg<C, K0, F>;
    auto kernel = dcb_tail_kernel<T, C, K0, F>;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [&] {
        attr_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kBytes);
    });
    if (attr_err != cudaSuccess) {
        return attr_err;
    }
    const int num_tiles = (p.M + 2 * kRows - 1) / (2 * kRows);
    const int pairs = num_tiles < num_sms() / 2 ? num_tiles : num_sms() / 2;
    return launch_pdl_cluster(kernel, dim3(2 * pairs), dim3(kThreads), G::kBytes, stream, 2, m[0], m[1], m[2], m[3],
                              m[4], m[5], p);
}

template <typename T>
cudaError_t dispatch_tail(const CUtensorMap (&m)[6], const DcbTailParams& p, cudaStream_t s)
{
    if (p.C == 512 && p.cffn == 256) {
        return p.cdc ? launch_tail<T, 512, 256, 256>(m, p, s) : launch_tail<T, 512, 0, 256>(m, p, s);
    }
    if (p.C == 256 && p.cffn == 256) {
        return p.cdc ? launch_tail<T, 256, 256, 256>(m, p, s) : launch_tail<T, 256, 0, 256>(m, p, s);
    }
    return p.cdc ? launch_tail<T, 256, 128, 128>(m, p, s) : launch_tail<T, 256, 0, 128>(m, p, s);
}

}  // namespace

bool dcb_tail_supported(int C, int cdc, int cffn, int n1)
{
    return n1 == 4 * cffn && num_sms() >= 2 &&
           ((C == 512 && cffn == 256 && (cdc == 0 || cdc == 256)) || (C == 256 && cffn == 256 && (cdc == 0 || cdc == 256)) ||
            (C == 256 && cffn == 128 && (cdc == 0 || cdc == 128)));
}

// The kernel's time goes in waves of one tile per pair of SMs, that of the separate launches with M, by a
// step where the 256 columns of dc.3 and ffn.2 (128-wide tiles of 512) no longer run in one round, at
// 128 * num_sms / 4 rows (one B200, inputs rotating through L2, microseconds fused / separate):
//   (512, 256, 256): M = 4736 22.1 / 16.9, 6144 22.5 / 23.5, 14400 24.3 / 36.2; 19200 (second wave just begun) 45.8 /
//     43.3, 23552 (a quarter full) 49.9 / 48.5, 24576 50.7 / 53.0, 32640 51.3 / 60.8; 38400 (third wave) 77.8 / 75.6,
//     42000 (almost a quarter) 80.0 / 77.6, 44000 77.5 / 81.7; 57600 (fourth) 108.7 / 107.5; 129600 202 / 226
//   (256, 256, 256): M = 4736 20.0 / 18.3, 5120 15.3 / 16.4, 14400 18.4 / 29.0, 19200 27.7 / 32.7, 38400 44.1 / 46.7,
//     129600 107 / 135
//   (256, 128, 128): M = 4736 13.1 / 12.3, 5120 12.5 / 14.4, 14400 13.8 / 21.3, 19200 21.0 / 26.1, 38400 32.5 / 36.5,
//     129600 71 / 91
// and against the one-SM ConvFFN kernel (ffn_sm100.cu; cdc = 0):
//   (512, 256): M = 390 17.1 / 38.6, 32640 40.0 / 89.0;  (256, 128): M = 390 9.2 / 11.6, 14400 10.9 / 13.3,
//     37888 18.6 / 19.2, 48000 27.2 / 26.7, 129600 57.7 / 59.4
bool dcb_tail_preferred(int M, int C, int cdc, int cffn, int n1)
{
    if (!gemm_pairs_allowed() || !dcb_tail_supported(C, cdc, cffn, n1)) {
        return false;
    }
    const int tiles = (M + 2 * kRows - 1) / (2 * kRows), pairs = num_sms() / 2;
    if (cdc == 0) {
        return cffn == 256 || tiles <= 2 * pairs;
    }
    const int over = tiles % pairs;  // tiles of a last wave that is not full
    if (C == 512 && over > 0 && 4 * over < pairs && (tiles / pairs == 1 || tiles / pairs == 2)) {
        return false;
    }
    return 4LL * ((M + kRows - 1) / kRows) > num_sms();
}

cudaError_t dcb_tail_sm100(int dtype, const DcbTailParams& p_in, cudaStream_t stream)
{
    DcbTailParams p = p_in;
    p.stall_test = gemm_take_stall(&p.wait_limit) ? 1 : 0;
    auto bad = [](const void* q) { return q == nullptr || (reinterpret_cast<uintptr_t>(q) & 15) != 0; };
    if (p.M <= 0 || (dtype != 0 && dtype != 1) || !dcb_tail_supported(p.C, p.cdc, p.cffn, 4 * p.cffn) || bad(p.x) ||
        p.ldx % 8 != 0 || bad(p.out) || p.ldo % 8 != 0 || bad(p.w1) || bad(p.w2) || p.b1 == nullptr || p.b2 == nullptr ||
        (p.cdc != 0 && (bad(p.a) || p.lda % 8 != 0 || bad(p.w0) || p.b0 == nullptr)) ||
        (reinterpret_cast<uintptr_t>(p.qscale) & 15) != 0) {
        return cudaErrorInvalidValue;
    }
    const CUtensorMapDataType dt = dtype == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    auto act = [&](CUtensorMap* m, const void* base, int cols, int ld, int rows) {
        return make_tmap_2d(m, dt, base, cols, p.M, static_cast<uint64_t>(ld) * 2, 64, rows, 128);
    };
    auto weight = [&](CUtensorMap* m, const void* base, int k, int n) {
        return make_tmap_2d(m, dt, base, k, n, static_cast<uint64_t>(k) * 2, 64, kNB / 2, 128);
    };
    CUtensorMap m[6];
    std::memset(m, 0, sizeof(m));
    if ((p.cdc != 0 && (!act(&m[0], p.a, p.cdc, p.lda, kRows) || !weight(&m[2], p.w0, p.cdc, p.C))) ||
        !act(&m[1], p.x, p.C, p.ldx, kRows) || !weight(&m[3], p.w1, p.C, 4 * p.cffn) ||
        !weight(&m[4], p.w2, p.cffn, p.C) || !act(&m[5], p.out, p.C, p.ldo, 32)) {
        return cudaErrorInvalidValue;
    }
    return dtype == 0 ? dispatch_tail<__half>(m, p, stream) : dispatch_tail<__nv_bfloat16>(m, p, stream);
}

}  // namespace dcvc
