// The quad GEMM (conv1x1_bias_wsilu_chunk_add) with its activations resident in shared memory:
//
//   out[m, c] = sum_{k<4} WSiLU(a[m] . W[4c+k]^T [* wscale] + b[4c+k])
//
// The tiled kernel (gemm_sm100.cu) stages 128 rows of A and 256 of W for every K block of every
// tile: at the MMA's rate that is 96 bytes per SM and clock from L2 (64 with cta_group::2), more
// than L2 delivers, and the same A rows are fetched again for each of the N / 256 column blocks.
// Here a pair of CTAs keeps 256 rows of A (128 per CTA, K / 64 swizzled slabs) while it walks the
// column blocks, so only half a W tile per CTA and K block streams (32 bytes per clock), and
// with nothing else in tensor memory the blocks are 256 wide in two accumulators, the shape in
// which cta_group::2 runs at full rate.  The (row tile, column block) units are dealt to the pairs in
// contiguous ranges of equal length, so that no pair has more than one unit above the average.  A slab
// is refilled with the next row tile's as soon as the last block's MMAs have read it.
//
// Sixteen epilogue warps (32 rows x 64 columns each) turn a block into 64 outputs per row and store
// them from registers, 32 bytes per lane.  Sums, epilogue and rounding are those of gemm_sm100:
// bitwise the same outputs.  In a loop it is bound by power: 4300 to 4540 clocks per unit against the
// MMAs' 4096, at an SM clock that drops to 1.3 to 1.55 GHz.
#include "gemm_sm100.cuh"

#include "host_util.h"

#include <cstring>
#include <mutex>
#include <type_traits>

namespace dcvc {

namespace {

constexpr int kRows = 128;               // rows per CTA
constexpr int kNB = 256;                 // columns per block
constexpr int kSlabBytes = kRows * 128;  // 128 bytes of K of 128 rows
constexpr int kTileBytes = kNB / 2 * 128;
constexpr int kMaxSlabs = 8;
constexpr int kMaxStages = 10;
constexpr int kMaxN = 4096;
constexpr int kEpiWarps = 16;
constexpr int kFirstEpiWarp = 3;
constexpr int kThreads = 32 * (kFirstEpiWarp + kEpiWarps);
constexpr int kTmemCols = 512;
constexpr long long kWaitLimit = 2000000000LL;
constexpr int kSmemLimit = 232448;
constexpr int kBarBytes = 512;

template <typename T>
__device__ __forceinline__ uint32_t pack16(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack16<__half>(float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack16<__nv_bfloat16>(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// K bytes per slab are 128: 64 16-bit or 128 8-bit values.  An 8-bit block of 128 K bytes takes the
// MMA half as long, so its ring stages hold two.
template <bool F8>
__host__ __device__ constexpr int stage_tiles()
{
    return F8 ? 2 : 1;
}

struct QuadLayout {
    int slabs;   // A slabs in shared memory (>= K slabs of one tile)
    int stages;  // W ring
    int bias_offset, bar_offset, bytes;
};

template <bool F8>
__host__ __device__ inline QuadLayout quad_layout(int kslabs, int n)
{
    QuadLayout l;
    const int bias = n * 4 * (F8 ? 2 : 1);
    const int stage = stage_tiles<F8>() * kTileBytes;
    const int room = kSmemLimit - 1024 - kBarBytes - bias;
    // room for the next row tile's slabs beside this one's where four W stages still fit
    l.slabs = 2 * kslabs <= kMaxSlabs && room - 2 * kslabs * kSlabBytes >= 4 * stage ? 2 * kslabs : kslabs;
    const int fit = (room - l.slabs * kSlabBytes) / stage;
    l.stages = fit > kMaxStages ? kMaxStages : fit;
    l.bias_offset = l.slabs * kSlabBytes + l.stages * stage;
    l.bar_offset = l.bias_offset + bias;
    l.bytes = l.bar_offset + kBarBytes + 1024;
    l.bytes = l.bytes < kTmemCtaMinSmem ? kTmemCtaMinSmem : l.bytes;  // (not at the sizes of today)
    return l;
}

template <typename T, bool F8>
__global__ void __launch_bounds__(kThreads, 1)
    quad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const GemmParams p,
                const bool wide_store)
{
    constexpr int kStageTiles = stage_tiles<F8>();
    constexpr int kStageBytes = kStageTiles * kTileBytes;
    constexpr int kKElems = F8 ? 128 : 64;
    const int kslabs = p.K / kKElems;
    const QuadLayout lay = quad_layout<F8>(kslabs, p.N);
    const long long lim = p.wait_limit > 0 ? p.wait_limit : kWaitLimit;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem =
        reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = smem + lay.slabs * kSlabBytes;
    // E: in the even CTA, counts both CTAs; commits of the MMA warp arrive in both
    uint64_t* wfull = reinterpret_cast<uint64_t*>(smem + lay.bar_offset);  // E
    uint64_t* wempty = wfull + kMaxStages;
    uint64_t* afull = wempty + kMaxStages;   // E
    uint64_t* aempty = afull + kMaxSlabs;
    uint64_t* accfull = aempty + kMaxSlabs;
    uint64_t* accempty = accfull + 2;        // E
    uint64_t* drain = accempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();
    const int nblocks = p.N / kNB;
    const long long num_units = static_cast<long long>((p.M + 2 * kRows - 1) / (2 * kRows)) * nblocks;
    const int pair = static_cast<int>(blockIdx.x >> 1), pairs = static_cast<int>(gridDim.x >> 1);
    // this pair's units: column block u % nblocks of row tile u / nblocks
    const int u0 = static_cast<int>(num_units * pair / pairs), u1 = static_cast<int>(num_units * (pair + 1) / pairs);
    const int row_off = static_cast<int>(rank) * kRows;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&wfull[s], 1);
            mbar_init(&wempty[s], 1);
        }
        for (int s = 0; s < kMaxSlabs; ++s) {
            mbar_init(&afull[s], 1);
            mbar_init(&aempty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&accfull[b], 1);
            mbar_init(&accempty[b], 2 * kEpiWarps);
        }
        mbar_init(drain, 1);
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
        if (!p.stall_test) {
            int stage = 0;
            uint32_t phase = 0;
            int issued = 0;
            bool ok = true;
            for (int u = u0; ok && u < u1 && !warp_any(*abort_flag != 0); ++u) {
                const int n0 = (u % nblocks) * kNB + static_cast<int>(rank) * (kNB / 2);
                for (int kb = 0; kb < kslabs; kb += kStageTiles) {
                    if (!mbar_wait_warp(&wempty[stage], phase ^ 1, lim)) {
                        ok = fail(kErrGemmProducerTimeout);
                        break;
                    }
                    if (elect_one()) {
                        if (rank == 0) {
                            mbar_arrive_expect_tx(&wfull[stage], 2 * kStageBytes);
                        }
                        const uint32_t bar = cluster_map(&wfull[stage], 0);
#pragma unroll
                        for (int t = 0; t < kStageTiles; ++t) {
                            tma_load_2d_pair(ring + stage * kStageBytes + t * kTileBytes, &tmW, bar,
                                             (kb + t) * kKElems, n0);
                        }
                    }
                    __syncwarp();
                    ++issued;
                    if (++stage == lay.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
            }
            if (warp_any(*abort_flag != 0) && rank == 0) {
                // let the copies land before the CTA winds down
                for (int i = 0; i < (issued < lay.stages ? issued : lay.stages); ++i) {
                    if (--stage < 0) {
                        stage = lay.stages - 1;
                        phase ^= 1;
                    }
                    mbar_wait_warp(&wfull[stage], phase, kWaitLimit / 16);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (even CTA)
        if (rank == 0) {
            // format 0 is F16 for kind::f16 and E4M3 for kind::f8f6f4
            const uint32_t idesc =
                make_idesc_f16(2 * kRows, kNB, !F8 && sizeof(T) == 2 && std::is_same<T, __nv_bfloat16>::value ? 1 : 0);
            const uint32_t slab_addr = smem_u32(smem), ring_addr = smem_u32(ring);
            int stage = 0, slab0 = 0;        // ring positions: next W stage, the row tile's first slab
            uint32_t phase = 0, aphase = 0;  // aphase: parity of slab0's fill
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
            bool ok = true;
            for (int u = u0; ok && u < u1 && !warp_any(*abort_flag != 0); ++u) {
                const bool first = u == u0 || u % nblocks == 0;               // of its row tile here
                const bool last = u + 1 == u1 || (u + 1) % nblocks == 0;
                ok = need(&accempty[acc], acc_phase ^ 1);
                const uint32_t d = tmem_base + static_cast<uint32_t>(acc * kNB);
                int slab = slab0;
                uint32_t sp = aphase;
                for (int kb = 0; ok && kb < kslabs; kb += kStageTiles) {
                    int sl[kStageTiles];
#pragma unroll
                    for (int t = 0; t < kStageTiles; ++t) {
                        sl[t] = slab;
                        ok = ok && (!first || need(&afull[slab], sp));
                        if (++slab == lay.slabs) {
                            slab = 0;
                            sp ^= 1;
                        }
                    }
                    ok = ok && need(&wfull[stage], phase);
                    if (!ok) {
                        break;
                    }
                    if (elect_one()) {
#pragma unroll
                        for (int t = 0; t < kStageTiles; ++t) {
                            const uint64_t adesc = make_sw128_kmajor_desc(slab_addr + sl[t] * kSlabBytes);
                            const uint64_t bdesc =
                                make_sw128_kmajor_desc(ring_addr + stage * kStageBytes + t * kTileBytes);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const uint32_t accumulate = (kb | t | k) != 0 ? 1u : 0u;
                                if constexpr (F8) {
                                    tc_mma_f8_pair(d, adesc + 2 * k, bdesc + 2 * k, idesc, accumulate);
                                } else {
                                    tc_mma_f16_pair(d, adesc + 2 * k, bdesc + 2 * k, idesc, accumulate);
                                }
                            }
                        }
                        tc_commit_pair_both(&wempty[stage]);
                        if (last) {
#pragma unroll
                            for (int t = 0; t < kStageTiles; ++t) {
                                tc_commit_pair_both(&aempty[sl[t]]);
                            }
                        }
                        if (kb + kStageTiles >= kslabs) {
                            tc_commit_pair_both(&accfull[acc]);
                        }
                    }
                    __syncwarp();
                    issued_any = true;
                    if (++stage == lay.stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (last) {
                    slab0 = slab;
                    aphase = sp;
                }
                acc ^= 1;
                acc_phase ^= acc == 0 ? 1u : 0u;
            }
            if (warp_any(*abort_flag != 0) && issued_any) {
                if (elect_one()) {
                    tc_commit_pair_local(drain);
                }
                __syncwarp();
                mbar_wait_warp(drain, 0, kWaitLimit / 16);
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ activation slabs
        if (!p.stall_test) {
            int slab = 0;
            uint32_t phase = 0;
            int issued = 0;
            bool ok = true;
            for (int u = u0; ok && u < u1 && !warp_any(*abort_flag != 0); u = (u / nblocks + 1) * nblocks) {
                const int m0 = (u / nblocks) * 2 * kRows + row_off;
                for (int kb = 0; kb < kslabs; ++kb) {
                    if (!mbar_wait_warp(&aempty[slab], phase ^ 1, lim)) {
                        ok = fail(kErrGemmProducerTimeout);
                        break;
                    }
                    if (elect_one()) {
                        if (rank == 0) {
                            mbar_arrive_expect_tx(&afull[slab], 2 * kSlabBytes);
                        }
                        tma_load_2d_pair(smem + slab * kSlabBytes, &tmA, cluster_map(&afull[slab], 0), kb * kKElems, m0);
                    }
                    __syncwarp();
                    ++issued;
                    if (++slab == lay.slabs) {
                        slab = 0;
                        phase ^= 1;
                    }
                }
            }
            if (warp_any(*abort_flag != 0) && rank == 0) {
                for (int i = 0; i < (issued < lay.slabs ? issued : lay.slabs); ++i) {
                    if (--slab < 0) {
                        slab = lay.slabs - 1;
                        phase ^= 1;
                    }
                    mbar_wait_warp(&afull[slab], phase, kWaitLimit / 16);
                }
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue warps
        const int quad = warp & 3;                    // TMEM lane quadrant this warp may access
        const int grp = (warp - kFirstEpiWarp) >> 2;  // which 64 of a block's 256 columns
        const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + grp * 64;
        // biases (and dequantisation factors) in shared memory: L1 has no room for them
        float* bias = reinterpret_cast<float*>(smem + lay.bias_offset);
        for (int i = threadIdx.x - 32 * kFirstEpiWarp; i < p.N; i += 32 * kEpiWarps) {
            bias[i] = p.bias[i];
            if constexpr (F8) {
                bias[p.N + i] = p.wscale[i];
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpiWarps) : "memory");
        uint32_t bias_addr;  // known from here on: reads of the biases cannot move above the barrier
        asm volatile("mov.u32 %0, %1;" : "=r"(bias_addr) : "r"(smem_u32(bias)) : "memory");
        const uint32_t even = cluster_map(smem, 0) - smem_u32(smem);
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int u = u0; ok && u < u1 && !warp_any(*abort_flag != 0); ++u) {
            const int col = (u % nblocks) * kNB + grp * 64;
            const int m = (u / nblocks) * 2 * kRows + row_off + quad * 32 + lane;
            if (!mbar_wait_warp(&accfull[acc], acc_phase, lim)) {
                ok = fail(kErrGemmEpilogueTimeout);
                break;
            }
            tc_fence_after();
            uint32_t o[8];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t r[32];
                tmem_ld_32x32b_x32(lane_base + acc * kNB + c * 32, r);
                tc_wait_ld();
                if (c == 1) {
                    tc_fence_before();
                    __syncwarp();
                    mbar_arrive_tmem_if(lane == 0, smem_u32(&accempty[acc]) + even, 1);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float2 v[4];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int i = 8 * k + 4 * h;
                        const uint32_t at = bias_addr + (col + c * 32 + i) * 4;
                        const float4 b = lds128_const(at);
                        const float2 lo = make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                        const float2 hi = make_float2(__uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
                        if constexpr (F8) {
                            const float4 f = lds128_const(at + p.N * 4);
                            v[2 * h] = __ffma2_rn(lo, make_float2(f.x, f.y), make_float2(b.x, b.y));
                            v[2 * h + 1] = __ffma2_rn(hi, make_float2(f.z, f.w), make_float2(b.z, b.w));
                        } else {
                            v[2 * h] = __fadd2_rn(lo, make_float2(b.x, b.y));
                            v[2 * h + 1] = __fadd2_rn(hi, make_float2(b.z, b.w));
                        }
                    }
                    const float2 w0 = wsilu2(v[0]), w1 = wsilu2(v[1]), w2 = wsilu2(v[2]), w3 = wsilu2(v[3]);
                    o[4 * c + k] = pack16<T>(w0.x + w0.y + w1.x + w1.y, w2.x + w2.y + w3.x + w3.y);
                }
            }
            if (m < p.M) {
                T* dst = reinterpret_cast<T*>(p.out) + static_cast<size_t>(m) * p.ldo + col / 4;
                if (wide_store) {
                    st_global_256(dst, o);
                } else {
                    reinterpret_cast<uint4*>(dst)[0] = make_uint4(o[0], o[1], o[2], o[3]);
                    reinterpret_cast<uint4*>(dst)[1] = make_uint4(o[4], o[5], o[6], o[7]);
                }
            }
            __syncwarp();
            acc ^= 1;
            acc_phase ^= acc == 0 ? 1u : 0u;
        }
    }

    pair_end(tmem_base, kTmemCols, warp == 1);
}

template <typename T, bool F8>
cudaError_t launch_quad(const CUtensorMap& a, const CUtensorMap& w, const GemmParams& p, cudaStream_t stream)
{
    auto kernel = quad_kernel<T, F8>;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [&] {
        attr_err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    });
    if (attr_err != cudaSuccess) {
        return attr_err;
    }
    const QuadLayout lay = quad_layout<F8>(p.K / (F8 ? 128 : 64), p.N);
    const long long units = static_cast<long long>((p.M + 2 * kRows - 1) / (2 * kRows)) * (p.N / kNB);
    const int pairs = static_cast<int>(units < num_sms() / 2 ? units : num_sms() / 2);
    const bool wide = p.ldo % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
    return launch_pdl_cluster(kernel, dim3(2 * pairs), dim3(kThreads), lay.bytes, stream, 2, a, w, p, wide);
}

}  // namespace

bool quad_sm100_eligible(int dtype, int M, int N, int K)
{
    const int kslabs = K / (dtype == kDtypeF8 ? 128 : 64);
    return num_sms() >= 2 && M > 0 && N % kNB == 0 && N <= kMaxN && K % (dtype == kDtypeF8 ? 256 : 64) == 0 &&
           kslabs >= 1 && kslabs <= kMaxSlabs &&
           (dtype == kDtypeF8 ? quad_layout<true>(kslabs, N).stages : quad_layout<false>(kslabs, N).stages) >= 3 &&
           static_cast<long long>((M + 2 * kRows - 1) / (2 * kRows)) * (N / kNB) < 0x7fffffff;
}

// Whether it is the faster form where no narrower tile runs all at once (gemm_pick_bn; us back to back, medians of
// alternating runs, tiled / this; M x N x K):
//   16-bit: 8160 x 1024 x 512 (128 units on 74 pairs) 9.7 / 11.0, 14400 (228) 15.4 / 15.8, 24000 (376) 23.6 / 24.0,
//   32640 (512) 33.5 / 30.2, 129600 134 / 103; 14400 x 1536 x 384 (342) 17.4 / 17.7, 24000 (564) 27.2 / 27.3, 32640
//   (768) 37.6 / 32.5; 12000 x 2048 x 512 (376) 23.7 / 24.4, 14400 (456) 27.6 / 26.9; 24000 x 1024 x 256 (376) 15.6 /
//   16.0, 32640 (512) 18.5 / 18.1; 32640 x 512 x 256 (256) 11.9 / 12.6
//   E4M3: 390 x 1024 x 512 5.7 / 6.0, 2040 5.9 / 6.2, 10000 (160) 11.3 / 11.0, 14400 (228) 13.9 / 13.0, 32640 22.4 /
//   19.7
// The tiled kernel's CTAs start on their own and it has stages for its first K blocks at once; the pair meets its
// peer, fills both CTAs' slabs and then runs the units of its range without a gap, so it needs some of them: six per
// pair, two of the shorter E4M3 ones.  A unit takes a pair about as long as a tile takes one SM in the tiled
// kernel, so rounds are compared.
bool quad_sm100_preferred(int dtype, int M, int N, int K)
{
    if (!gemm_pairs_allowed() || !quad_sm100_eligible(dtype, M, N, K)) {
        return false;
    }
    const int sms = num_sms(), pairs = sms / 2;
    const long long blocks = N / kNB;
    const long long units = (M + 2 * kRows - 1) / (2 * kRows) * blocks, tiles = (M + kRows - 1) / kRows * blocks;
    return units >= (dtype == kDtypeF8 ? 2 : 6) * pairs && (units + pairs - 1) / pairs <= (tiles + sms - 1) / sms;
}

cudaError_t quad_sm100(int dtype, const void* A, int lda, const void* W, const GemmParams& p, cudaStream_t stream)
{
    if (!quad_sm100_eligible(dtype, p.M, p.N, p.K) || p.bias == nullptr) {
        return cudaErrorInvalidValue;
    }
    const bool f8 = dtype == kDtypeF8;
    const CUtensorMapDataType dt = f8             ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                   : dtype == 0 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    const int esz = f8 ? 1 : 2, kbox = f8 ? 128 : 64;
    CUtensorMap a, w;
    std::memset(&a, 0, sizeof(a));
    std::memset(&w, 0, sizeof(w));
    if (!make_tmap_2d(&a, dt, A, p.K, p.M, static_cast<uint64_t>(lda) * esz, kbox, kRows, 128) ||
        !make_tmap_2d(&w, dt, W, p.K, p.N, static_cast<uint64_t>(p.K) * esz, kbox, kNB / 2, 128)) {
        return cudaErrorInvalidValue;
    }
    if (f8) {
        return launch_quad<__nv_bfloat16, true>(a, w, p, stream);
    }
    return dtype == 0 ? launch_quad<__half, false>(a, w, p, stream) : launch_quad<__nv_bfloat16, false>(a, w, p, stream);
}

}  // namespace dcvc
