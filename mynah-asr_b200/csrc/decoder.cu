// Greedy decoders on device.
//
// CTC (the reference's mynah_asr_ctc_decode, src/decoder_ctc.c:36-61): the head
// GEMM runs on the contraction kernel; argmax_rows picks the first maximum of
// logit + bias per frame; the collapse (drop repeats, drop blank = V-1) is a scan
// over T integers done by the caller.
//
// RNNT / TDT (mynah_asr_greedy_decode and greedy_decode_tdt, src/decoder.c:129-265):
// strictly sequential per utterance, so a batch of up to 16 utterances advances in
// lock step inside ONE persistent cooperative kernel — no launch or host round trip
// per step. Every step is a few grid-wide phases separated by grid barriers:
//   head    logits[b] = head . relu(enc[b][t_b] + g[b]); a warp owns 16 rows of the
//           V (+durations) rows for all utterances and emits first-argmax candidates
//   select  the candidates meet in one 64-bit maximum per utterance; every CTA applies the
//           emission rule to its own copy of the utterances' state, no barrier behind it: non-blank -> emit, advance by the predicted duration (RNNT: 0),
//           blank with duration 0 -> 1, max_symbols guard (src/decoder.c:161-176)
//   lstm    (only if some utterance emitted) a row block is 4 hidden units x 4 gates of
//           [W_ih | W_hh] against [input ; previous h] of all utterances, then the cell
//           update; layers are separated by a grid barrier
//   proj    g[b] = decoder_projector(h_last[b])
// What bounds it is latency: 49 MB of weights per emitting step come from L2 in 9 us, the four phases take 19 us with one
// utterance (36 k cycles) and 28 with sixteen (53 k; 35 behind the contractions of a large batch, which leave the clock at the
// power cap). 26 and 40 with the selection as a phase of its own, weights asked for only behind the barriers and the cells of a
// row block updated by one warp.
// The matvecs run on the warp-level tensor-core path with the utterances as the N
// dimension: weights as fp16 (hi, lo) planes (a decoded Q4_0/Q8_0 weight is exact in
// that form), activations split the same way, three MMAs per k-step, f32 accumulate —
// f32-grade like the reference's sgemv/sgemm path.
#include "kernels.h"
#include "model.h"

namespace mb {

// -------------------------------------------------------------- argmax per row
__global__ void __launch_bounds__(256)
argmax_kernel(const float *__restrict__ logits, int ld, const float *__restrict__ bias, int V, int *__restrict__ best) {
    __shared__ float sv[256];
    __shared__ int si[256];
    chain_trigger();
    chain_wait();
    const float *row = logits + (size_t)blockIdx.x * ld;
    float bv = -3.0e38f;
    int bi = 0x7fffffff;
    for (int k = threadIdx.x; k < V; k += 256) {
        const float v = row[k] + (bias ? bias[k] : 0.0f);
        if (v > bv) { bv = v; bi = k; }          // ascending k per thread: first maximum kept
    }
    sv[threadIdx.x] = bv; si[threadIdx.x] = bi;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            const float v = sv[threadIdx.x + o];
            const int i = si[threadIdx.x + o];
            if (v > sv[threadIdx.x] || (v == sv[threadIdx.x] && i < si[threadIdx.x])) { sv[threadIdx.x] = v; si[threadIdx.x] = i; }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) best[blockIdx.x] = si[0];
}

int argmax_rows(const float *logits, int ld, const float *bias, int T, int V, int *best, cudaStream_t st, bool chain) {
    if (T <= 0) return 0;
    MB_CUDA(launch_kernel(argmax_kernel, dim3(T), dim3(256), 0, st, chain, 1, logits, ld, bias, V, best));
    return 0;
}

// ------------------------------------------------------- RNNT / TDT lock-step

// ---- tensor-core matvec for a batch of up to 16 utterances ----------------------
// out[r][b] = sum_k W[r][k] * X[b][k] with W as fp16 (hi, lo) planes streamed from L2 and
// X as fp16 (hi, lo) planes in shared memory. A warp owns 16 weight rows (the M side
// of mma.m16n8k16) and the 16 utterances are two N blocks; three MMAs per k-step
// (hi*hi, lo*hi, hi*lo) give f32-grade products. k is consumed in a permuted order
// that lets both operands be fetched with 16-byte loads: within a 32-wide chunk lane
// (g, t) holds k = 8t..8t+7 of its rows, and k-step s uses elements 4s..4s+3 of them —
// the same assignment on both operands, so the sum is unchanged.
static constexpr int XPAD = 32;                       // halves of padding per X row (bank spread)

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint4 ld_weight(const __half *p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// A warp's 16 weight rows (fragment rows g and g + 8) and its sums. Weights do not depend on the state: ask() sends for the
// first AHEAD chunks of 32 k, which a phase does before it waits at the grid barrier in front of it (the loads are volatile,
// they stay there), so that the L2 delivers them meanwhile. NB: blocks of eight utterances.
template <int NB>
struct RowTask {
    static constexpr int AHEAD = 5;
    const __half *hi, *lo;
    int oA, oB;                                       // the lane's columns of its two rows
    uint4 ah[AHEAD], bh[AHEAD], al[AHEAD], bl[AHEAD];
    float d0[NB][4], d1[NB][4];                       // hi x hi; the terms with a low plane
    __device__ __forceinline__ void at(const __half *whi, const __half *wlo, int ld, int rowA, int rowB, int lane) {
        hi = whi; lo = wlo;
        oA = rowA * ld + 8 * (lane & 3); oB = rowB * ld + 8 * (lane & 3);
#pragma unroll
        for (int n = 0; n < NB; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) d0[n][i] = d1[n][i] = 0.f;
    }
    __device__ __forceinline__ void ask(int c0, int c1) {
#pragma unroll
        for (int i = 0; i < AHEAD; i++)
            if (c0 + i < c1) {
                const int o = (c0 + i) * 32;
                ah[i] = ld_weight(hi + oA + o); bh[i] = ld_weight(hi + oB + o); al[i] = ld_weight(lo + oA + o); bl[i] = ld_weight(lo + oB + o);
            }
    }
    __device__ __forceinline__ void chunk(uint4 a, uint4 b, uint4 c, uint4 d, const __half *xhi, const __half *xlo, int xs) {
        uint4 xh[NB], xl[NB];
#pragma unroll
        for (int n = 0; n < NB; n++) {
            xh[n] = *reinterpret_cast<const uint4 *>(xhi + n * 8 * xs);
            xl[n] = *reinterpret_cast<const uint4 *>(xlo + n * 8 * xs);
        }
        // k-step 0: elements 0..3, k-step 1: elements 4..7
#pragma unroll
        for (int n = 0; n < NB; n++) {
            mma_f16(d0[n], a.x, b.x, a.y, b.y, xh[n].x, xh[n].y);
            mma_f16(d1[n], c.x, d.x, c.y, d.y, xh[n].x, xh[n].y);
            mma_f16(d1[n], a.x, b.x, a.y, b.y, xl[n].x, xl[n].y);
        }
#pragma unroll
        for (int n = 0; n < NB; n++) {
            mma_f16(d0[n], a.z, b.z, a.w, b.w, xh[n].z, xh[n].w);
            mma_f16(d1[n], c.z, d.z, c.w, d.w, xh[n].z, xh[n].w);
            mma_f16(d1[n], a.z, b.z, a.w, b.w, xl[n].z, xl[n].w);
        }
    }
    // adds chunks [c0, c1), the first of them asked for before
    __device__ __forceinline__ void add(int c0, int c1, const __half *xhi, const __half *xlo, int xs, int lane) {
        xhi += (size_t)(lane >> 2) * xs + 8 * (lane & 3);
        xlo += (size_t)(lane >> 2) * xs + 8 * (lane & 3);
#pragma unroll
        for (int i = 0; i < AHEAD; i++)
            if (c0 + i < c1) chunk(ah[i], bh[i], al[i], bl[i], xhi + (c0 + i) * 32, xlo + (c0 + i) * 32, xs);
        for (int c = c0 + AHEAD; c < c1; c += AHEAD) {
            ask(c, c1);
#pragma unroll
            for (int i = 0; i < AHEAD; i++)
                if (c + i < c1) chunk(ah[i], bh[i], al[i], bl[i], xhi + (c + i) * 32, xlo + (c + i) * 32, xs);
        }
    }
    // to red[warp][4 n + i][lane]: rows g (i = 0, 1) and g + 8 (2, 3) x utterances 8 n + 2 t, + 1
    __device__ __forceinline__ void put(float *red, int lane, int wib) const {
#pragma unroll
        for (int n = 0; n < NB; n++)
#pragma unroll
            for (int i = 0; i < 4; i++) red[(wib * 8 + n * 4 + i) * 32 + lane] = fmaf(d1[n][i], H16_LO_INV, d0[n][i]);
    }
};
// The matvecs' tasks: a row block of 16 rows in NSL slices of K, a warp each.
static constexpr int LSTM_NSL = 4, HEAD_NSL = 2;
struct Task { int rb, sl, c0, c1; bool on; };
__device__ __forceinline__ Task task_of(int base, int wib, int nsl, int nrb, int chunks) {
    Task k;
    k.rb = (base + wib) / nsl; k.sl = (base + wib) % nsl; k.on = k.rb < nrb;
    const int per = (chunks + nsl - 1) / nsl;
    k.c0 = k.sl * per; k.c1 = k.c0 + per < chunks ? k.c0 + per : chunks;
    return k;
}

// Writes f32 rows [16][K] (rows >= B zero) as (hi, lo) planes into shared memory.
// Two passes — every global load of the CTA is issued before the first shared store —
// so the loads overlap instead of queueing behind stores the compiler cannot prove
// independent. value4(b, k) returns elements k..k+3 of row b.
static constexpr int STAGE_NV = 16;                   // float4 per thread: covers K <= 1024
template <typename F>
__device__ __forceinline__ void stage_x(__half *xhi, __half *xlo, int xs, int koff, int K, int B, F value4) {
    // sixteen threads per row, 16-byte columns c0, c0 + 16, ...: no division, 256 contiguous bytes per row step
    const int b = threadIdx.x >> 4, c0 = threadIdx.x & 15, k4n = K >> 2;
    float4 v[STAGE_NV];
#pragma unroll
    for (int j = 0; j < STAGE_NV; j++) {
        const int c = c0 + 16 * j;
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < k4n && b < B) v[j] = value4(b, c * 4);
    }
#pragma unroll
    for (int j = 0; j < STAGE_NV; j++) {
        const int c = c0 + 16 * j;
        if (c < k4n) {
            __align__(8) __half h[4], l[4];
            split_h16(v[j].x, h[0], l[0]); split_h16(v[j].y, h[1], l[1]);
            split_h16(v[j].z, h[2], l[2]); split_h16(v[j].w, h[3], l[3]);
            *reinterpret_cast<uint2 *>(xhi + b * xs + koff + c * 4) = *reinterpret_cast<uint2 *>(h);
            *reinterpret_cast<uint2 *>(xlo + b * xs + koff + c * 4) = *reinterpret_cast<uint2 *>(l);
        }
    }
}
__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Rows that already exist as fp16 (hi, lo) planes in global memory (hidden states, embedding rows) go to
// the X tile with 16-byte asynchronous copies: no registers, no conversion, one wait for all of them.
// row_hi(b) / row_lo(b) return the H halves of utterance b; columns [koff, koff + H) of the tile are written.
__device__ __forceinline__ void cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory"); }
template <typename FH, typename FL>
__device__ __forceinline__ void stage_planes(__half *xhi, __half *xlo, int xs, int koff, int H, int B, FH row_hi, FL row_lo) {
    const int cpr = H >> 3;                               // 16-byte chunks per row
    for (int idx = threadIdx.x; idx < B * cpr; idx += blockDim.x) {
        const int b = idx / cpr, c = idx - b * cpr;
        cp16(xhi + b * xs + koff + 8 * c, row_hi(b) + 8 * c);
        cp16(xlo + b * xs + koff + 8 * c, row_lo(b) + 8 * c);
    }
}

// Sigmoid that never exponentiates a positive argument (the reference's mynah_asr_sigmoid, src/qmat.h:31-35), without a branch on the
// sign or a division, so that a cell's gates overlap. The quotient is the product with the reciprocal, corrected by its residual
// (P. W. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990). Largest
// relative error against float64 over four million arguments: 1.36e-7 for x >= 0, 2.35e-7 down to -87. 244 steps of one utterance (a
// minute of audio): 10.70 ms a call become 10.48.
__device__ __forceinline__ float dec_sigmoid(float x) {
    const float e = expf(-fabsf(x)), num = x >= 0.0f ? 1.0f : e, den = 1.0f + e;
    const float r = reciprocal(den), y = num * r;
    return fmaf(fmaf(-den, y, num), r, y);
}

// What every CTA knows of the utterances, kept in step by applying the same rule to the same maxima
struct GreedyShared {
    int t[DEC_MAX_B], len[DEC_MAX_B], off[DEC_MAX_B];            // frame, frames, first row in enc
    int eh[DEC_MAX_B], no[DEC_MAX_B], tok[DEC_MAX_B], emit[DEC_MAX_B];
    unsigned long long best[DEC_MAX_B][2];                       // this CTA's candidates: token, duration
    int stop;
};

// All CTAs have come `target / gridDim.x` times. One counter; 2.2 k cycles against 2.9 k of the cooperative groups' barrier.
// Bounded: a wait that runs out sets the status and the abort flag, and every CTA leaves (false).
__device__ __forceinline__ void greedy_arrive(const GreedyDev &p, unsigned &target) {
    target += gridDim.x;
    __syncthreads();
    // the block barrier before and the release make the CTA's writes visible with the arrival, the acquire and the block
    // barrier behind it those of the others to all threads
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.scratch) : "memory");
}
__device__ __forceinline__ bool greedy_wait(const GreedyDev &p, GreedyShared &sh, unsigned target) {
    if (threadIdx.x == 0) {
        const long long t0 = clock64();
        unsigned v;
        for (int tries = 1;; tries++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p.scratch) : "memory");
            if (v >= target) break;
            if (tries & 63) continue;
            if (*reinterpret_cast<volatile int *>(p.scratch + 1) || clock64() - t0 > (1ll << 31)) {
                atomicExch(p.scratch + 1, 1);
                atomicCAS(p.status, ST_OK, ST_TIMEOUT_EPILOGUE);
                sh.stop = 1;
                break;
            }
        }
    }
    __syncthreads();
    return sh.stop == 0;
}

// (value, index) in one word: the larger word is the larger value, among equals the smaller index. 0 stands for none.
__device__ __forceinline__ unsigned long long cand_word(float v, int i) {
    const unsigned u = __float_as_uint(v + 0.0f);                // -0 counts as 0
    return ((unsigned long long)(u ^ ((u >> 31) ? 0xffffffffu : 0x80000000u)) << 32) | (0xffffffffu - (unsigned)i);
}
__device__ __forceinline__ int cand_index(unsigned long long w) { return w ? (int)(0xffffffffu - (unsigned)w) : 0x7fffffff; }

struct Cand { float v; int i; };
__device__ __forceinline__ void cand_take(Cand &a, float v, int i) {
    if (v > a.v || (v == a.v && i < a.i)) { a.v = v; a.i = i; }
}

// One stacked-LSTM layer (pred_step, src/decoder.c:73-99) for all utterances. A row block is 4 units x 4 gates (i, f, g, o); a
// slice of K is a piece of the previous h and the same piece of the input. Reads h[par], writes h[par^1]; c in place. Utterances
// that did not emit copy their state through.
// lstm_open, between arrival and wait of the barrier in front of the phase: the CTA's first tasks over the previous h, which is
// known by then, and the first weights over the input.
template <int NB>
__device__ __forceinline__ void lstm_rows(const GreedyDev &p, int l, const Task &k, int lane, RowTask<NB> &w) {
    // fragment row lr -> gate lr/4, unit rb*4 + lr%4
    const int g = lane >> 2, rowA = (g >> 2) * p.H + k.rb * 4 + (g & 3);
    w.at(p.wcat_hi[l], p.wcat_lo[l], 2 * p.H, rowA, rowA + 2 * p.H, lane);
    w.ask(p.H / 32 + k.c0, p.H / 32 + k.c1);
}
template <int NB>
__device__ __forceinline__ void lstm_open(const GreedyDev &p, int l, int par, __half *xhi, __half *xlo, int lane, int wib, RowTask<NB> &w) {
    const int H = p.H, B = p.B, xs = 2 * H + XPAD, hc = H / 32;
    const Task k = task_of(blockIdx.x * 8, wib, LSTM_NSL, H / 4, hc);
    if (k.on) lstm_rows<NB>(p, l, k, lane, w);
    if (blockIdx.x * 8 < H / 4 * LSTM_NSL) {          // a CTA without a row block to work on does not pull the activations either
        const __half *hold_hi = reinterpret_cast<const __half *>(p.h[par]) + (size_t)l * B * H, *hold_lo = hold_hi + (size_t)p.L * B * H;
        stage_planes(xhi, xlo, xs, H, H, B, [&](int b) { return hold_hi + (size_t)b * H; }, [&](int b) { return hold_lo + (size_t)b * H; });
        cp_wait_all();
    }
    __syncthreads();
    if (k.on) { w.add(hc + k.c0, hc + k.c1, xhi, xlo, xs, lane); w.ask(k.c0, k.c1); }
}
template <int NB>
__device__ __forceinline__ void lstm_phase(const GreedyDev &p, const GreedyShared &sh, int l, int par, __half *xhi, __half *xlo, float *red, int lane, int wib, RowTask<NB> &w) {
    const int H = p.H, B = p.B, xs = 2 * H + XPAD, hc = H / 32;
    // hidden states live as fp16 (hi, lo) planes: h[parity] = [hi: L][B][H] then [lo: L][B][H] halves
    const size_t nstate = (size_t)p.L * B * H;
    const __half *hold_hi = reinterpret_cast<const __half *>(p.h[par]) + (size_t)l * B * H, *hold_lo = hold_hi + nstate;
    __half *hnew_hi = reinterpret_cast<__half *>(p.h[par ^ 1]) + (size_t)l * B * H, *hnew_lo = hnew_hi + nstate;
    float *cc = p.c + (size_t)l * B * H;
    const __half *xin_hi = l == 0 ? nullptr : reinterpret_cast<const __half *>(p.h[par ^ 1]) + (size_t)(l - 1) * B * H;
    const __half *xin_lo = l == 0 ? nullptr : xin_hi + nstate;
    constexpr int NSL = LSTM_NSL;
    const int nrb = H / 4;
    for (int base = blockIdx.x * 8; base < nrb * NSL; base += gridDim.x * 8) {
        const bool again = base != (int)blockIdx.x * 8;
        const Task k = task_of(base, wib, NSL, nrb, hc);
        const int rb = k.rb;
        const bool on = k.on;
        // The four warps of a row block share its cells, (utterance, unit) by thread: one warp for all of them took 6.6 k cycles
        // with sixteen utterances. What a cell needs besides the sums — biases, previous state, emission flag — is fetched now.
        const int j = (wib & 3) * 32 + lane, b = j >> 2, unit = rb * 4 + (j & 3);
        const bool cell = on && b < B;                           // (B <= 16: the first two warps)
        float bih[4] = {0.f, 0.f, 0.f, 0.f}, bhh[4] = {0.f, 0.f, 0.f, 0.f}, cprev = 0.f;
        if (cell) {
#pragma unroll
            for (int q = 0; q < 4; q++) { bih[q] = p.b_ih[l][q * H + unit]; bhh[q] = p.b_hh[l][q * H + unit]; }
            cprev = cc[(size_t)b * H + unit];
        }
        if (!again) {
            if (l == 0)
                stage_planes(xhi, xlo, xs, 0, H, B, [&](int b) { return p.emb_hi + (size_t)sh.tok[b] * H; },
                             [&](int b) { return p.emb_lo + (size_t)sh.tok[b] * H; });
            else
                stage_planes(xhi, xlo, xs, 0, H, B, [&](int b) { return xin_hi + (size_t)b * H; }, [&](int b) { return xin_lo + (size_t)b * H; });
            cp_wait_all();
            __syncthreads();
        } else if (on) {
            lstm_rows<NB>(p, l, k, lane, w);
            w.add(hc + k.c0, hc + k.c1, xhi, xlo, xs, lane);
            w.ask(k.c0, k.c1);
        }
        if (on) {
            w.add(k.c0, k.c1, xhi, xlo, xs, lane);
            w.put(red, lane, wib);
        }
        __syncthreads();
        if (cell) {
            // gate q of unit u is fragment row 4 q + u: lane group 4 (q & 1) + u, upper or lower half by q >> 1
            float z[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int at = (wib & 4) * 8 + (b >> 3) * 4 + (q >> 1) * 2 + (b & 1), from = (4 * (q & 1) + (j & 3)) * 4 + ((b & 7) >> 1);
                float v = 0.f;
#pragma unroll
                for (int e = 0; e < NSL; e++) v += red[(at + e * 8) * 32 + from];
                z[q] = v + bih[q] + bhh[q];
            }
            const size_t o = (size_t)b * H + unit;
            if (sh.emit[b]) {
                const float cn = dec_sigmoid(z[1]) * cprev + dec_sigmoid(z[0]) * tanhf(z[2]);
                cc[o] = cn;
                __half hh, hl;
                split_h16(dec_sigmoid(z[3]) * tanhf(cn), hh, hl);
                hnew_hi[o] = hh; hnew_lo[o] = hl;
            } else {
                hnew_hi[o] = hold_hi[o]; hnew_lo[o] = hold_lo[o];
            }
        }
        __syncthreads();
    }
}

// g[b] = proj_b + proj_w . h_last[b] for the utterances that emitted. proj_open: the first weights, in front of the barrier's wait.
template <int NB>
__device__ __forceinline__ void proj_open(const GreedyDev &p, const Task &k, int lane, RowTask<NB> &w) {
    const int H = p.H, rA = k.rb * 16 + (lane >> 2), rB = rA + 8;
    if (!k.on) return;
    w.at(p.proj_hi, p.proj_lo, H, rA < H ? rA : H - 1, rB < H ? rB : H - 1, lane);
    w.ask(k.c0, k.c1);
}
template <int NB>
__device__ __forceinline__ void proj_phase(const GreedyDev &p, const GreedyShared &sh, int par, bool all, __half *xhi, __half *xlo, float *red, int lane, int wib, RowTask<NB> &w) {
    const int H = p.H, B = p.B, xs = 2 * H + XPAD;
    const size_t nstate = (size_t)p.L * B * H;
    const __half *hl_hi = reinterpret_cast<const __half *>(p.h[par]) + (size_t)(p.L - 1) * B * H, *hl_lo = hl_hi + nstate;
    constexpr int NSL = LSTM_NSL;
    const int nrb = (H + 15) / 16;
    for (int base = blockIdx.x * 8; base < nrb * NSL; base += gridDim.x * 8) {
        const bool again = base != (int)blockIdx.x * 8;
        const Task k = task_of(base, wib, NSL, nrb, H / 32);
        const int rb = k.rb;
        const bool on = k.on;
        if (again) proj_open<NB>(p, k, lane, w);
        // (utterance, row) by thread of the row block's four warps. The encoder value that the epilogue adds to g is fetched now,
        // under the contraction, and the projector bias of an utterance that emitted or the g that the others keep
        const int r = rb * 16 + (lane & 15);
        float ev[NB], addv[NB];
        bool fresh[NB], past[NB];
#pragma unroll
        for (int n = 0; n < NB; n++) {
            const int b = n * 8 + (wib & 3) * 2 + (lane >> 4);
            ev[n] = addv[n] = 0.f;
            fresh[n] = false; past[n] = true;
            if (on && r < H && b < B) {
                fresh[n] = all || sh.emit[b] != 0;
                addv[n] = fresh[n] ? p.proj_b[r] : p.g[(size_t)b * H + r];
                past[n] = sh.t[b] >= sh.len[b];
                if (!past[n]) ev[n] = p.enc[(size_t)(sh.off[b] + sh.t[b]) * H + r];
            }
        }
        if (!again) {
            stage_planes(xhi, xlo, xs, 0, H, B, [&](int b) { return hl_hi + (size_t)b * H; }, [&](int b) { return hl_lo + (size_t)b * H; });
            cp_wait_all();
            __syncthreads();
        }
        if (on) {
            w.add(k.c0, k.c1, xhi, xlo, xs, lane);
            w.put(red, lane, wib);
        }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < NB; n++) {
            const int b = n * 8 + (wib & 3) * 2 + (lane >> 4), lr = lane & 15;
            if (!on || r >= H || b >= B) continue;
            // g, and with it the joint input of the coming step for this utterance's current frame
            // (an utterance that did not emit keeps its g but may have moved to another frame)
            const size_t o = (size_t)b * H + r;
            float gv = addv[n];
            if (fresh[n]) {
                float v = 0.f;
#pragma unroll
                for (int e = 0; e < NSL; e++) v += red[(((wib & 4) + e) * 8 + n * 4 + (lr >> 3) * 2 + (b & 1)) * 32 + (lr & 7) * 4 + ((b & 7) >> 1)];
                gv = v + addv[n];
                p.g[o] = gv;
            }
            const float jv = past[n] ? 0.f : fmaxf(ev[n] + gv, 0.f);
            __half jh, jl;
            split_h16(jv, jh, jl);
            p.jx_hi[o] = jh; p.jx_lo[o] = jl;
        }
        __syncthreads();
    }
}

// A head block's first weights
template <int NB>
__device__ __forceinline__ void head_open(const GreedyDev &p, const Task &k, int lane, RowTask<NB> &w) {
    const int VL = p.V + p.ND, rA = k.rb * 16 + (lane >> 2), rB = rA + 8;
    if (!k.on) return;
    w.at(p.head_hi, p.head_lo, p.H, rA < VL ? rA : VL - 1, rB < VL ? rB : VL - 1, lane);
    w.ask(k.c0, k.c1);
}

template <int NB>
__global__ void __launch_bounds__(256, 1)
greedy_kernel(GreedyDev p) {
    extern __shared__ __align__(16) uint8_t dsm[];
    const int H = p.H, B = p.B, V = p.V, VL = p.V + p.ND;
    const int xs = 2 * H + XPAD;
    __half *xhi = reinterpret_cast<__half *>(dsm);
    __half *xlo = xhi + 16 * xs;
    float *red = reinterpret_cast<float *>(xlo + 16 * xs);          // [8 warps][8][32 lanes]
    RowTask<NB> w;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    __shared__ GreedyShared sh;
    unsigned target = 0;
    unsigned long long *cand = reinterpret_cast<unsigned long long *>(p.scratch + 16);
    if (threadIdx.x < DEC_MAX_B) {
        const int b = threadIdx.x;
        const bool on = b < B;
        sh.t[b] = on ? p.t[b] : 0; sh.len[b] = on ? p.enc_len[b] : 0; sh.off[b] = on ? p.enc_off[b] : 0;
        sh.eh[b] = on ? p.emitted_here[b] : 0; sh.no[b] = on ? p.n_out[b] : 0;
        sh.tok[b] = !on || p.init_state ? p.blank : p.last_tok[b]; sh.emit[b] = on && p.init_state;
        if (b == 0) sh.stop = 0;
    }
    int par = (!p.init_state && p.par_state) ? *p.par_state : 0;   // read before the first grid sync; written after the last
    for (int i = threadIdx.x; i < 16 * xs; i += blockDim.x) { xhi[i] = __float2half_rn(0.f); xlo[i] = __float2half_rn(0.f); }
    __syncthreads();                                               // rows of absent utterances stay zero for every plane copy

    constexpr int NSL = HEAD_NSL;
    const int nrb = (VL + 15) / 16;
    const Task first_head = task_of(blockIdx.x * 8, wib, NSL, nrb, H / 32), first_proj = task_of(blockIdx.x * 8, wib, LSTM_NSL, (H + 15) / 16, H / 32);
    // the prediction net on the tokens just emitted, from lstm_open of layer 0 to the head's first weights
    auto predict = [&](bool all) -> bool {
        for (int l = 0; l < p.L; l++) {
            lstm_phase<NB>(p, sh, l, par, xhi, xlo, red, lane, wib, w);
            greedy_arrive(p, target);
            if (l + 1 < p.L) lstm_open<NB>(p, l + 1, par, xhi, xlo, lane, wib, w);
            else proj_open<NB>(p, first_proj, lane, w);
            if (!greedy_wait(p, sh, target)) return false;
        }
        par ^= 1;
        proj_phase<NB>(p, sh, par, all, xhi, xlo, red, lane, wib, w);
        greedy_arrive(p, target);
        head_open<NB>(p, first_head, lane, w);
        return greedy_wait(p, sh, target);
    };
    if (p.init_state) {
        // SOS = blank on a zero state (src/decoder.c:151): run the prediction net once
        lstm_open<NB>(p, 0, par, xhi, xlo, lane, wib, w);
        if (!predict(true)) return;
    } else head_open<NB>(p, first_head, lane, w);
    bool jx_valid = p.init_state != 0;     // the planes of relu(enc[t] + g) left by the last projector phase are current

    // optional phase timers (clock64 of CTA 0): head, sync with the first layer opened, select, prediction net with its syncs, -, steps, emit steps, staging
    const bool timing = p.dbg != nullptr && blockIdx.x == 0 && threadIdx.x == 0;
    long long tq = timing ? clock64() : 0;
#define PHASE_MARK(slot) do { if (timing) { const long long n_ = clock64(); p.dbg[slot] += n_ - tq; tq = n_; } } while (0)
    for (int step = 0; step < p.max_steps; step++) {
        // ---- head: joint = relu(enc[t] + g) -> logits -> first-argmax candidates per row block
        // (an utterance past its end gets zeros)
        if (threadIdx.x < 2 * DEC_MAX_B) {
            (&sh.best[0][0])[threadIdx.x] = 0;
            if (blockIdx.x == 0) cand[(step + 1) % 3 * 2 * DEC_MAX_B + threadIdx.x] = 0;    // last read two steps ago
        }
        if (blockIdx.x * 8 < nrb * NSL && jx_valid) {
            stage_planes(xhi, xlo, xs, 0, H, B, [&](int b) { return p.jx_hi + (size_t)b * H; }, [&](int b) { return p.jx_lo + (size_t)b * H; });
            cp_wait_all();
        } else if (blockIdx.x * 8 < nrb * NSL)
        stage_x(xhi, xlo, xs, 0, H, B, [&](int b, int k) {
            const int row = sh.t[b] < sh.len[b] ? sh.off[b] + sh.t[b] : -1;
            const float4 e = ld4(p.enc + (size_t)(row < 0 ? 0 : row) * H + k), gg = ld4(p.g + (size_t)b * H + k);
            const float z = row < 0 ? 0.f : 1.f;
            return make_float4(z * fmaxf(e.x + gg.x, 0.f), z * fmaxf(e.y + gg.y, 0.f), z * fmaxf(e.z + gg.z, 0.f), z * fmaxf(e.w + gg.w, 0.f));
        });
        __syncthreads();
        PHASE_MARK(7);
        for (int base = blockIdx.x * 8; base < nrb * NSL; base += gridDim.x * 8) {
            const Task k = task_of(base, wib, NSL, nrb, H / 32);
            const int rb = k.rb, sl = k.sl;
            const bool on = k.on;
            if (base != (int)blockIdx.x * 8) head_open<NB>(p, k, lane, w);
            const int rA = rb * 16 + g, rB = rA + 8;
            const float biasA = on && rA < VL ? p.head_b[rA] : 0.f, biasB = on && rB < VL ? p.head_b[rB] : 0.f;
            if (on) {
                w.add(k.c0, k.c1, xhi, xlo, xs, lane);
                w.put(red, lane, wib);
            }
            __syncthreads();
            if (on) {                                            // the block's two warps share the utterances
#pragma unroll
                for (int q = 0; q < NB; q++) {
                    const int nb = NB == 1 ? 0 : sl, e = NB == 1 ? sl : q, w0 = (wib & ~1) * 8 + nb * 4 + e;
                    const float va = red[w0 * 32 + lane] + red[(w0 + 8) * 32 + lane] + biasA;
                    const float vb = red[(w0 + 2) * 32 + lane] + red[(w0 + 10) * 32 + lane] + biasB;
                    Cand tk{-3.0e38f, 0x7fffffff}, du{-3.0e38f, 0x7fffffff};
                    if (rA < V) cand_take(tk, va, rA); else if (rA < VL) cand_take(du, va, rA);
                    if (rB < V) cand_take(tk, vb, rB); else if (rB < VL) cand_take(du, vb, rB);
                    // reduce over the eight lanes that hold the other rows of this utterance
#pragma unroll
                    for (int o = 4; o < 32; o <<= 1) {
                        cand_take(tk, __shfl_xor_sync(0xffffffffu, tk.v, o), __shfl_xor_sync(0xffffffffu, tk.i, o));
                        if (rb * 16 + 16 > V) cand_take(du, __shfl_xor_sync(0xffffffffu, du.v, o), __shfl_xor_sync(0xffffffffu, du.i, o));
                    }
                    const int b = nb * 8 + 2 * t + e;
                    if (g == 0 && b < B) {
                        if (tk.i != 0x7fffffff) atomicMax(&sh.best[b][0], cand_word(tk.v, tk.i));
                        if (du.i != 0x7fffffff) atomicMax(&sh.best[b][1], cand_word(du.v, du.i));
                    }
                    }
            }
            __syncthreads();
        }
        unsigned long long *best = cand + step % 3 * 2 * DEC_MAX_B;
        if (threadIdx.x < 2 * B) {
            const unsigned long long w = (&sh.best[0][0])[threadIdx.x];
            if (w) atomicMax(best + threadIdx.x, w);
        }
        PHASE_MARK(0);
        greedy_arrive(p, target);
        lstm_open<NB>(p, 0, par, xhi, xlo, lane, wib, w);       // most steps emit
        if (!greedy_wait(p, sh, target)) return;
        PHASE_MARK(1);
        // ---- select: the emission rule, by every CTA for itself
        int em = 0;
        bool over = true;
        if (threadIdx.x < B) {
            const int b = threadIdx.x;
            int tb = sh.t[b];
            const unsigned long long bt = __ldcg(best + 2 * b), bd = __ldcg(best + 2 * b + 1);
            if (tb < sh.len[b]) {
                const int k = cand_index(bt);
                int dur = p.ND > 0 ? (bd ? p.durations[cand_index(bd) - V] : 0) : (k == p.blank ? 1 : 0);
                if (k != p.blank) {
                    const int no = sh.no[b], eh = sh.eh[b] + 1;
                    if (no < p.cap) {
                        if (blockIdx.x == 0) { p.tokens[(size_t)b * p.cap + no] = k; p.frames[(size_t)b * p.cap + no] = tb; }
                        sh.no[b] = no + 1;
                    }
                    em = 1;
                    sh.tok[b] = k < V ? k : 0;
                    sh.eh[b] = eh;
                    if (dur == 0 && eh >= p.max_symbols) dur = 1;
                } else if (dur == 0) {
                    dur = 1;
                }
                if (dur > 0) sh.eh[b] = 0;
                tb += dur;
                sh.t[b] = tb;
            }
            sh.emit[b] = em;
            over = tb >= sh.len[b];
        }
        const int any_emit = __syncthreads_or(em), all_done = __syncthreads_and(over);
        PHASE_MARK(2);
        if (timing) { p.dbg[5] += 1; p.dbg[6] += any_emit != 0; }
        if (any_emit) {
            if (!predict(false)) return;
            PHASE_MARK(3);
        } else head_open<NB>(p, first_head, lane, w);
        jx_valid = any_emit != 0;
        if (all_done) break;
    }
#undef PHASE_MARK
    if (blockIdx.x == 0 && threadIdx.x < B) {
        const int b = threadIdx.x;
        p.t[b] = sh.t[b]; p.emitted_here[b] = sh.eh[b]; p.n_out[b] = sh.no[b]; p.last_tok[b] = sh.tok[b]; p.emit[b] = sh.emit[b];
        if (b == 0 && p.par_state) *p.par_state = par;
    }
}

__global__ void sigmoid_kernel(const float *__restrict__ x, float *__restrict__ out, int n, int cell) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = cell ? dec_sigmoid(x[i]) : sigmoid_fast(x[i]);
}
int sigmoids(const float *x, float *out, int n, int cell, cudaStream_t st) {
    sigmoid_kernel<<<cdiv(n, 256), 256, 0, st>>>(x, out, n, cell);
    MB_CUDA(cudaGetLastError());
    return 0;
}

int greedy_launch(const GreedyDev &p, cudaStream_t st, int want_blocks) {
    int dev = 0, sms = 0, coop = 0;
    MB_CUDA(cudaGetDevice(&dev));
    MB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MB_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) { set_error("greedy decode: device lacks cooperative launch"); return -1; }
    void (*const kernel)(GreedyDev) = p.B <= 8 ? greedy_kernel<1> : greedy_kernel<2>;
    const size_t smem = 2 * 16 * (size_t)(2 * p.H + XPAD) * sizeof(__half) + 8 * 32 * 8 * sizeof(float);
    if (smem > 48 * 1024)
        MB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    MB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem));
    if (per_sm < 1) { set_error("greedy decode: kernel does not fit an SM"); return -1; }
    int blocks = want_blocks > 0 && want_blocks < sms ? want_blocks : sms;
    if (blocks < p.B) { set_error("greedy decode: batch %d exceeds SM count", p.B); return -1; }
    GreedyDev pc = p;
    void *args[] = {&pc};
    MB_CUDA(cudaLaunchCooperativeKernel((void *)kernel, dim3(blocks), dim3(256), args, smem, st));
    return 0;
}

}  // namespace mb
