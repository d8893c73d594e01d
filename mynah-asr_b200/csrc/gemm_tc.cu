// Dense contraction C[M,N] = A[M,K] * B[N,K]^T on the 5th-generation tensor cores.
//
// This is the large-M half of the quantised matmul (the reference's
// mynah_asr_qmat_mul, src/qmat.c:503-651, and mynah_asr_gemm_wt, src/backend.c:68-81):
// weights arrive already decoded to fp16 (hi, lo) planes resident in HBM, activations
// as fp16 (hi, lo) planes written by the producing kernel's epilogue.
//
//   * TMA (cp.async.bulk.tensor.2d, 128-byte swizzle, every CTA loads its own tiles) stages 128 x 64
//     A tiles and BN x 64 B tiles into a shared-memory ring guarded by mbarriers;
//   * one elected thread issues tcgen05.mma (kind::f16, M=128, N=BN, K=16) into TMEM
//     accumulators; with NTERMS=3 every k-step issues hi*hi into one accumulator and
//     lo*hi + hi*lo into a second one (the lo planes are pre-scaled by 2^11, the
//     epilogue adds the second accumulator back times 2^-11), so the product carries
//     ~22 significant bits per operand (f32-grade parity with the reference's sgemm);
//     with NTERMS=1 only hi*hi (fast mode);
//   * the issuing warps walk their loops whole and elect the lane that issues (warp_index, elect_one): operands of tcgen05 and TMA
//     then are uniform registers. As code of one lane of a diverged warp every MMA waited for its operands to be moved there:
//     three products of [12000 x 1024 x 4096] took 224 us instead of 202, 47 rows of it 33 instead of 25, [750 x 4096 x 1024] 25.4
//     instead of 22.7 (f32 out); a voice command on 17 layers 1.83 ms instead of 1.60, 15 s on 24 layers 5.73 instead of 5.06,
//     sixteen minutes 60.6 instead of 58.7. With parts of the kernel left out, [12000 x 4096 x 1024]: operand loads alone 126 us,
//     loads and MMAs 180, loads and epilogue 132, all 198; with a single product 49, 59, 72 and 87;
//   * the kernel is persistent (one CTA per SM walks the output tiles) and the
//     accumulators are double-buffered in TMEM, so the epilogue of one tile overlaps
//     the MMAs of the next; eight epilogue warps read the accumulator with tcgen05.ld
//     and apply the fused tail: + bias, SiLU / ReLU, then either store f32, accumulate into the residual
//     stream (x += alpha * y), or store the result as fp16 (hi, lo) planes for the
//     next contraction.
//
// Row stability: an output row depends only on its own A row and on B; the k order
// and the instruction sequence are the same for every tile position and every M, so
// a row's bits do not depend on what else is in the batch.
#include "gemm.h"

namespace mb {

static constexpr int BM = GEMM_BM;
static constexpr int BK = 64;
static constexpr int EPI_WARPS = 8;
static constexpr int GEMM_THREADS = (2 + EPI_WARPS) * 32;   // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue
static constexpr int SMEM_LIMIT = 232448;  // 227 KB

// AR: rows of an A tile that shared memory holds and TMA loads. The MMA always reads 128 rows; with at most 64 rows in
// all (AR = 64) the upper half of what it reads is whatever follows in the stage, and the accumulator rows it makes are
// never stored. A stage is then a third smaller and two CTAs fit one SM: a chained successor sets up, and asks for its
// weights, under its predecessor.
template <int BN, int NTERMS, int AR>
struct GemmCfg {
    static constexpr int NPLANES = NTERMS == 1 ? 1 : 2;
    static constexpr int A_BYTES = AR * BK * 2;
    static constexpr int B_BYTES = BN * BK * 2;
    static constexpr int STAGE_BYTES = NPLANES * (A_BYTES + B_BYTES);
    // the epilogue warps' turning buffers: only the wide tiles have them — the narrow ones serve contractions with few
    // rows, which are latency-bound and want every stage of the operand ring instead
    static constexpr bool BLOCK_EPILOGUE = BN >= 128;
    static constexpr int EPI_BYTES = BLOCK_EPILOGUE ? EPI_WARPS * GEMM_BLOCK_STAGE_FLOATS * 4 : 0;
    static constexpr int PER_SM = AR < BM ? 2 : 1;
    static constexpr int TAIL_BYTES = (BM - AR) * BK * 2;         // what the last stage's MMAs may read past its end
    static constexpr int STAGES_RAW = (SMEM_LIMIT / PER_SM - 2048 - 1024 * (PER_SM - 1) - TAIL_BYTES - EPI_BYTES) / STAGE_BYTES;
    static constexpr int STAGES = STAGES_RAW > 6 ? 6 : STAGES_RAW;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + TAIL_BYTES + EPI_BYTES + 2048;
    // NTERMS == 3 keeps a second accumulator for the cross terms (lo*hi + hi*lo);
    // everything is double-buffered so the epilogue of tile i overlaps the MMAs of tile i+1
    static constexpr int ACC_COLS = NTERMS == 1 ? BN : 2 * BN;
    static constexpr int TMEM_COLS = 2 * ACC_COLS < 32 ? 32 : 2 * ACC_COLS;
    static_assert(TMEM_COLS <= 512, "TMEM has 512 columns");
};

// Persistent kernel: one CTA per SM walks the output tiles (n fastest, so the CTAs in
// flight share a few A row-blocks while B stays L2-resident).
template <int BN, int NTERMS, int AR>
__global__ void __launch_bounds__(GEMM_THREADS, (AR < BM ? 2 : 1))
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA_hi, const __grid_constant__ CUtensorMap tmA_lo,
               const __grid_constant__ CUtensorMap tmB_hi, const __grid_constant__ CUtensorMap tmB_lo,
               const GemmEpilogue ep, const int M, const int N, const int K, const uint32_t stage_tx, int *status) {
    using Cfg = GemmCfg<BN, NTERMS, AR>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *tiles = smem;
    float *epi_stage = reinterpret_cast<float *>(smem + Cfg::STAGES * Cfg::STAGE_BYTES + Cfg::TAIL_BYTES);
    uint64_t *full_bar = reinterpret_cast<uint64_t *>(smem + Cfg::STAGES * Cfg::STAGE_BYTES + Cfg::TAIL_BYTES + Cfg::EPI_BYTES);
    uint64_t *empty_bar = full_bar + Cfg::STAGES;
    uint64_t *acc_full = empty_bar + Cfg::STAGES;      // [2] MMA -> epilogue
    uint64_t *acc_empty = acc_full + 2;                // [2] epilogue -> MMA
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int num_k = K / BK;
    const GemmUnits units(M, N, BN, gridDim.x);
    const int total = units.total;

    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA_hi);
        tma_prefetch_desc(&tmB_hi);
        if (NTERMS > 1) { tma_prefetch_desc(&tmA_lo); tma_prefetch_desc(&tmB_lo); }
        for (int s = 0; s < Cfg::STAGES; s++) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], EPI_WARPS); }
        mbar_fence_init();
    }
    if (warp == 1) { tc_alloc(tmem_slot, Cfg::TMEM_COLS); tc_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    chain_trigger();       // not before the allocation: a successor placed on this SM must not be first to take tensor memory

    if (warp == 0) {
        // ---------------------------------------------------------- TMA producer (one lane; the warp goes along)
        int s = 0, filled = 0;                         // ring position, k-blocks issued so far
        uint32_t ph = 1;
        bool ok = true;
        auto load_b = [&](int s, int kb, int n0) {
            uint8_t *bt = tiles + s * Cfg::STAGE_BYTES + Cfg::NPLANES * Cfg::A_BYTES;
            tma_load_2d(bt, &tmB_hi, kb * BK, n0, &full_bar[s]);
            if (NTERMS > 1) tma_load_2d(bt + Cfg::B_BYTES, &tmB_lo, kb * BK, n0, &full_bar[s]);
        };
        // the first ring of B tiles (weights) is asked for before the kernels in front have finished
        int ahead = 0;
        if (blockIdx.x < total) {
            int m0, n0, width;
            units.at(blockIdx.x, BN, m0, n0, width);
            ahead = num_k < Cfg::STAGES ? num_k : Cfg::STAGES;
            if (elect_one())
                for (int i = 0; i < ahead; i++) { mbar_expect_tx(&full_bar[i], stage_tx); load_b(i, i, n0); }
            __syncwarp();
        }
        chain_wait();
        for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x) {
            int m0, n0, width;
            units.at(tile, BN, m0, n0, width);               // a strip still loads BN rows of B: the MMAs read the first `width`
            for (int kb = 0; kb < num_k; kb++, filled++) {
                ok = mbar_wait_warp(&empty_bar[s], ph);
                if (!ok) break;
                if (elect_one()) {
                    uint8_t *st = tiles + s * Cfg::STAGE_BYTES;
                    if (filled >= ahead) mbar_expect_tx(&full_bar[s], stage_tx);
                    tma_load_2d(st, &tmA_hi, kb * BK, m0, &full_bar[s]);
                    if (NTERMS > 1) tma_load_2d(st + Cfg::A_BYTES, &tmA_lo, kb * BK, m0, &full_bar[s]);
                    if (filled >= ahead) load_b(s, kb, n0);
                }
                __syncwarp();
                if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
            }
        }
        if (!ok) {
            if (lane == 0) atomicExch(status, ST_TIMEOUT_PRODUCER);
            // let copies already in flight land before the CTA's shared memory goes away
            for (int j = filled > Cfg::STAGES ? filled - Cfg::STAGES : 0; j < filled; j++)
                mbar_wait_warp(&full_bar[j % Cfg::STAGES], (j / Cfg::STAGES) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (one lane; the warp goes along)
        int s = 0, lt = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < total && ok; tile += gridDim.x, lt++) {
            int m0, n0, width;
            units.at(tile, BN, m0, n0, width);
            const uint32_t idesc = umma_idesc_f16(BM, width), idesc_both = umma_idesc_f16(BM, NTERMS > 1 ? 2 * BN : BN);
            const int buf = lt & 1;
            const uint32_t acc = tmem_base + buf * Cfg::ACC_COLS;
            // the epilogue must have drained this accumulator (two tiles ago)
            ok = mbar_wait_warp(&acc_empty[buf], ((lt >> 1) & 1) ^ 1);
            if (!ok) break;
            tc_fence_after();
            for (int kb = 0; kb < num_k; kb++) {
                ok = mbar_wait_warp(&full_bar[s], ph);
                if (!ok) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t a = smem_u32(tiles + s * Cfg::STAGE_BYTES);
                    const uint64_t a_hi = umma_desc_sw128(a), a_lo = umma_desc_sw128(a + Cfg::A_BYTES);
                    const uint64_t b_hi = umma_desc_sw128(a + Cfg::NPLANES * Cfg::A_BYTES), b_lo = umma_desc_sw128(a + Cfg::NPLANES * Cfg::A_BYTES + Cfg::B_BYTES);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++) {
                        const uint64_t k = kk * 2;           // 16 fp16 = 32 bytes inside the swizzle atom, in units of 16
                        const uint32_t more = kk > 0 || kb > 0;
                        if (NTERMS == 1) {
                            tc_mma_f16(acc, a_hi + k, b_hi + k, idesc, more);
                            continue;
                        }
                        // The hi and the lo rows of B lie one below the other, as the two accumulators lie side by side: hi*hi and
                        // hi*lo can be one MMA of twice the width. With narrow tiles the MMA's fixed time is what counts (3.7 s of
                        // audio through 17 layers of 512: 2.24 -> 2.14 ms); from 64 columns on every MMA then waits for both
                        // accumulators of the one before it, which costs more than the second read of A (a minute through 24
                        // layers of 1024: 14.4 -> 15.1 ms). The first step has to clear both accumulators, and a strip's hi and lo
                        // rows do not touch.
                        const bool both = BN == 32 && width == BN && more;
                        if (!both) tc_mma_f16(acc, a_hi + k, b_hi + k, idesc, more);
                        tc_mma_f16(acc + BN, a_lo + k, b_hi + k, idesc, more);
                        if (both) tc_mma_f16(acc, a_hi + k, b_hi + k, idesc_both, 1);
                        else tc_mma_f16(acc + BN, a_hi + k, b_lo + k, idesc, 1);
                    }
                    tc_commit(&empty_bar[s]);                // frees the stage once these MMAs have read it
                    if (kb + 1 == num_k) tc_commit(&acc_full[buf]);
                }
                __syncwarp();
                if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
            }
            if (!ok && elect_one()) tc_commit(&acc_full[buf]);   // abandoned: the epilogue need not serve a wait of its own for it
        }
        if (!ok && lane == 0) atomicExch(status, ST_TIMEOUT_MMA);
    } else if (warp >= 2) {
        // -------------------------------------------------------------- epilogue
        const int lg = warp & 3;                       // TMEM lane group this warp may read
        const int half = (warp - 2) >> 2;              // even or odd 32-column chunks of the tile
        const int row = lg * 32 + lane;
        int lt = 0;
        bool fits = true;
        chain_wait();                                  // the residual is read and outputs are written only after the kernels in front
        // by blocks wherever the alignment allows, also with one tile per CTA (gemm.h)
        const bool blk_ok = Cfg::BLOCK_EPILOGUE && gemm_block_ok(ep);
        float *stage = epi_stage + (warp - 2) * GEMM_BLOCK_STAGE_FLOATS;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x, lt++) {
            int m0, n0, width;
            units.at(tile, BN, m0, n0, width);
            const int buf = lt & 1;
            const uint32_t acc = tmem_base + buf * Cfg::ACC_COLS + ((uint32_t)(lg * 32) << 16);
            if (!mbar_wait(&acc_full[buf], (lt >> 1) & 1)) {
                if (lane == 0) atomicExch(status, ST_TIMEOUT_EPILOGUE);
                break;
            }
            tc_fence_after();
            const int m = m0 + row;
            if (BN == 32) {
                // sixteen columns for each of the two warps of a lane group (one warp alone, a voice command on 17 layers of 512:
                // 2074 us instead of 2038)
                if (m0 + lg * 32 < M) {
                    float v[16], x[16];
                    tc_ld16(acc + (uint32_t)(half * 16), v);
                    if (NTERMS > 1) tc_ld16(acc + (uint32_t)(BN + half * 16), x);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; j++) if (NTERMS > 1) v[j] = fmaf(x[j], H16_LO_INV, v[j]);
                    if (m < M && n0 + half * 16 < N) fits &= gemm_epilogue_row(ep, v, m, n0 + half * 16, N);
                }
            } else if (num_k > 0) {
#pragma unroll 1
                for (int c = half; c < width / 32; c += 2) {
                    const int nb = n0 + c * 32;
                    const bool blk = blk_ok && nb + 32 <= N;            // warp-uniform
                    if (blk && m0 + lg * 32 >= M) continue;             // none of this warp's 32 rows exists
                    float4 res[8];
                    if (blk) gemm_block_prefetch(ep, m0 + lg * 32, M, nb, lane, res);
                    if (blk) {
                        // two halves of 16 columns: fewer live registers than the whole 32 x (hi*hi, cross) at once
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            float v[16];
                            tc_ld16(acc + (uint32_t)(c * 32 + h * 16), v);
                            if (NTERMS > 1) {
                                float x[16];
                                tc_ld16(acc + (uint32_t)(BN + c * 32 + h * 16), x);
                                tc_wait_ld();
#pragma unroll
                                for (int j = 0; j < 16; j++) v[j] = fmaf(x[j], H16_LO_INV, v[j]);
                            } else {
                                tc_wait_ld();
                            }
                            gemm_block_stage(v, h, stage, lane);
                        }
                        fits &= gemm_block_store(ep, res, m0 + lg * 32, M, nb, stage, lane, [](float4 t, int) { return t; });
                        continue;
                    }
                    float v[32];
                    tc_ld32(acc + (uint32_t)(c * 32), v);
                    if (NTERMS > 1) {
                        float x[32];
                        tc_ld32(acc + (uint32_t)(BN + c * 32), x);
                        tc_wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; j++) v[j] = fmaf(x[j], H16_LO_INV, v[j]);
                    } else {
                        tc_wait_ld();
                    }
                    if (m < M && nb < N) {
                        fits &= gemm_epilogue_row(ep, v, m, nb, N);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
        if (!fits) atomicCAS(status, ST_OK, ST_RANGE);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tc_dealloc(tmem_base, Cfg::TMEM_COLS);
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// fp16 [rows, K] row-major with row stride ld (halves): box = 64 (K) x box_rows, 128B swizzle.
static int make_map(CUtensorMap *m, const __half *base, int rows, int K, int ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) { set_error("cuTensorMapEncodeTiled entry point unavailable"); return -1; }
    if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld % 8) != 0) {
        set_error("gemm_tc: operand base/stride not 16-byte aligned");
        return -1;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return -1; }
    return 0;
}

template <int BN, int NTERMS, int AR>
static int launch(const GemmOperand &A, const GemmOperand &B, const GemmEpilogue &ep, int M, int N, int K,
                  int *status, cudaStream_t stream, bool chain) {
    using Cfg = GemmCfg<BN, NTERMS, AR>;
    CUtensorMap ta_hi, ta_lo, tb_hi, tb_lo;
    // a single row tile loads the rows there are (in eights, the swizzle atom): rows of zeros cost shared-memory writes
    const int a_rows = M < AR ? (int)align_up((size_t)M, 8) : AR;
    if (make_map(&ta_hi, A.hi, M, K, A.ld, a_rows)) return -1;
    if (make_map(&tb_hi, B.hi, N, K, B.ld, BN)) return -1;
    if (NTERMS > 1) {
        if (make_map(&ta_lo, A.lo, M, K, A.ld, a_rows)) return -1;
        if (make_map(&tb_lo, B.lo, N, K, B.ld, BN)) return -1;
    } else {
        ta_lo = ta_hi; tb_lo = tb_hi;
    }
    static PerDevice configured = {};
    int dev = 0;
    if (configured.below(Cfg::SMEM_BYTES, &dev)) {
        MB_CUDA(cudaFuncSetAttribute(gemm_tc_kernel<BN, NTERMS, AR>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     Cfg::SMEM_BYTES));
        configured.record(dev, Cfg::SMEM_BYTES);
    }
    const int sms = device_sm_count();
    // fewer tiles than SMs: the kernel cuts them into column strips (GemmUnits) when the grid leaves room
    const int total = cdiv(N, BN) * cdiv(M, BM), strips = BN % 128 == 0 ? 4 : BN % 64 == 0 ? 2 : 1;
    dim3 grid(total >= sms ? sms : total * strips <= sms ? total * strips : total * 2 <= sms && strips >= 2 ? total * 2 : total);
    const uint32_t stage_tx = Cfg::NPLANES * (uint32_t)(a_rows * BK * 2 + Cfg::B_BYTES);
    MB_CUDA(launch_kernel(gemm_tc_kernel<BN, NTERMS, AR>, grid, dim3(GEMM_THREADS), Cfg::SMEM_BYTES, stream, chain, 1,
                          ta_hi, ta_lo, tb_hi, tb_lo, ep, M, N, K, stage_tx, status));
    return 0;
}

int gemm_tc(const GemmOperand &A, const GemmOperand &B, const GemmEpilogue &ep, int M, int N, int K, int nterms,
            int *status, cudaStream_t stream, bool chain) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % BK != 0) { set_error("gemm_tc: K=%d must be a positive multiple of %d", K, BK); return -1; }
    if (nterms != 1 && (!A.lo || !B.lo)) { set_error("gemm_tc: 3-term mode needs lo planes"); return -1; }
    // Narrower N tiles when the output has too few 128-wide tiles to occupy the SMs (small M: decoder
    // positions, streaming chunks): more CTAs pull the operands. An output element sees the same k order
    // and the same instruction sequence whatever the tile width, so its bits do not change with it.
    const int sms = device_sm_count();
    // waves of CTAs x time of one tile (the MMAs scale with the tile width and K, prologue and epilogue do not: as much as 48
    // columns of K = 1024); what a last partial wave is cut into counts with its strips' width (GemmUnits). Below one wave
    // the strips do not count, although launch() cuts them: a strip still reads its tile's whole operands and waits for a
    // wide tile's set-up, and narrow tiles take hi hi and hi lo as one MMA. Counted, one utterance of 1 to 19 s takes 1.19 to
    // 1.25 times as long on 17 layers of d = 512 (2065 us becomes 2582), 1.13 to 1.20 on 24 of 1024, eight of 3 to 20 s the same.
    const int tm = cdiv(M, BM), fixed = K >= 49152 ? 1 : 49152 / K;
    int bn = 128;
    long best = -1;
    for (int cand = 128; cand >= 32; cand >>= 1) {
        const int tiles = tm * cdiv(N, cand), rem = tiles % sms;
        const int split = tiles < sms ? 1 : rem * 4 <= sms && cand % 128 == 0 ? 4 : rem * 2 <= sms && cand % 64 == 0 ? 2 : 1;
        const long cost = (long)(tiles / sms) * (cand + fixed) + (rem ? cand / split + fixed : 0);
        if (best < 0 || cost < best) { best = cost; bn = cand; }
    }
    const bool low = M <= 64;                        // one half-height row tile
#define GEMM_GO(BN_, NT_) (low ? launch<BN_, NT_, 64>(A, B, ep, M, N, K, status, stream, chain) : launch<BN_, NT_, 128>(A, B, ep, M, N, K, status, stream, chain))
    if (nterms == 1) {
        if (bn == 128 && N >= 256) return launch<256, 1, 128>(A, B, ep, M, N, K, status, stream, chain);
        if (bn == 128) return launch<128, 1, 128>(A, B, ep, M, N, K, status, stream, chain);
        return bn == 64 ? GEMM_GO(64, 1) : GEMM_GO(32, 1);
    }
    if (bn == 128) return launch<128, 3, 128>(A, B, ep, M, N, K, status, stream, chain);
    return bn == 64 ? GEMM_GO(64, 3) : GEMM_GO(32, 3);
#undef GEMM_GO
}

}  // namespace mb
