// The few-row chains as one persistent kernel.
//
// A streaming step or an AED position is a few hundred dependent operations of at most 128 rows. As launches, chained and
// replayed from a graph, each of them costs 9-11 us (set-up, tensor-memory allocation, slice sums over a cluster, LayerNorm
// by the last warp to arrive) where its bytes would need one. Here one cooperative launch walks the whole chain; what
// separates two operations is a grid barrier (about 1 us):
//   * a CTA keeps its place: a row tile of at most sixteen rows and every ngroups-th unit of eight weight rows. It sums a
//     unit over all of K itself (eight warps take alternate 64-wide pieces of K, added in warp order), so nothing is
//     exchanged between CTAs inside an operation, and a row's bits do not depend on how many other rows there are;
//   * weights are the stored 8-bit blocks (1.06 bytes per parameter instead of 4 as operand planes) in fragment order; a
//     producer warp streams them into a ring of shared memory with bulk copies and runs ahead through the barriers, so
//     that HBM works while the chain waits for its latencies;
//   * the products are mma.sync m16n8k16 on the integers themselves (exact in fp16) against the activations' (hi, lo)
//     planes, summed per 32-element block, then one f32 multiply-add per block with its scale: the quantised weight is
//     never rounded. (tcgen05 wants 128 rows on one side: a unit of eight weight rows per SM is what keeps all SMs busy
//     with N = 1024 and no exchange of partial sums.)
//   * with few rows the LayerNorms are computed where their result is staged, by every CTA; with more, as an operation that
//     spreads the rows over the CTAs. The conv module's middle sits in the epilogue of the contraction before it.
// Measured: a step of 24 layers of d = 1024 takes 1.34 ms for one stream (2.74 as launches), 2.25 for 22, 4.1 for 64 with
// decoding (4.8), 5.3 for 120 (5.9); AED with 32 + 8 layers takes 31 ms for one sentence (48.7), 61 for eight (78).
// Values that other CTAs write are read past the L1 (ld.cg, cp.async.cg). All waits are bounded: one that runs out sets the
// status word and the abort flag, and every CTA leaves. Nothing may spill: beside 220 KB of shared memory the L1 holds less
// than the stacks of 256 threads, and every spilled value then goes to the L2.
#include "fewrow.h"

#include <string.h>

#include "kernels.h"
#include "ln_row.cuh"

namespace mb {

static constexpr int FR_WARPS = 8, FR_THREADS = FR_WARPS * 32, FR_LAUNCH = FR_THREADS + 128;
static constexpr int FR_SLAB = 1024;                     // K per staged slab and per ring piece
static constexpr int FR_PAIR_BYTES = 544;                // 64 k x 8 rows: 512 bytes of quants, 32 of scales
static constexpr int FR_PAIRS = FR_SLAB / 64;
static constexpr int FR_PIECE = FR_PAIRS * FR_PAIR_BYTES;
static constexpr int FR_STAGES = 8;
static constexpr int FR_GU = 4;                          // units whose sums a CTA holds at a time
static constexpr int FR_CONV_K = 9;                      // depthwise width with a register path
static constexpr int FR_MAX_GEMMS = FR_MAX_LAYERS * 8;   // contractions of a chain (their weights' places sit in shared memory)
static constexpr int FR_XS = FR_SLAB + 32;               // halves per staged row: rows four 16-byte columns apart, no bank conflicts
static constexpr int FR_XPLANE = 32 * FR_XS * 2;         // bytes of one plane of 32 rows
static constexpr int FR_RED_FLOATS = FR_WARPS * FR_GU * 128;      // (also four LayerNorm vectors)
static constexpr int FR_VALS = FR_GU * 128;
static constexpr int FR_SMEM = FR_STAGES * FR_PIECE + 2 * FR_XPLANE + FR_RED_FLOATS * 4 + FR_VALS * 4 + FR_MAX_GEMMS * 16 + 256;
static_assert(FR_SMEM <= 230000, "shared memory");
static_assert(FR_RED_FLOATS >= 4 * FR_SLAB, "LayerNorm vectors");
static_assert(FR_GU * 128 == 2 * FR_THREADS, "two outputs per thread and group");

// ------------------------------------------------------------------------------------------------ weight tiles
bool fr_can_tile(const QWeight &w) {
    return (w.fmt == FMT_GGML_Q8_0 || w.fmt == FMT_GGML_Q4_0) && w.raw && w.k % 64 == 0 && (w.k <= FR_SLAB || w.k % FR_SLAB == 0);
}
size_t fr_tile_bytes(int n, int k) { return (size_t)cdiv(n, 8) * (k / 64) * FR_PAIR_BYTES; }

// one thread per (unit, pair, lane): lane (g, t) holds elements 8 t .. 8 t + 7 of both blocks of row g
template <int FMT>
__global__ void fr_retile_kernel(const uint8_t *__restrict__ raw, uint8_t *__restrict__ dst, int n, int k, int glu) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const int pairs = k / 64, units = (n + 7) / 8;
    if (i >= (size_t)units * pairs * 32) return;
    const int lane = (int)(i & 31), p = (int)((i >> 5) % pairs), u = (int)((i >> 5) / pairs), g = lane >> 2, t = lane & 3;
    const int row = glu ? (g < 4 ? 4 * u + g : n / 2 + 4 * u + g - 4) : 8 * u + g;
    constexpr int BB = FMT == FMT_GGML_Q8_0 ? 34 : 18;
    __align__(16) uint8_t q[16];
    __half sc[2];
    for (int b = 0; b < 2; b++) {
        const uint8_t *blk = raw + ((size_t)(row < n ? row : 0) * (k / 32) + 2 * p + b) * BB;
        for (int j = 0; j < 8; j++) {
            const int e = 8 * t + j;
            int v;
            if (FMT == FMT_GGML_Q8_0) v = (int8_t)blk[2 + e];
            else v = (e < 16 ? blk[2 + e] & 15 : blk[2 + e - 16] >> 4) - 8;
            q[8 * b + j] = row < n ? (uint8_t)(int8_t)v : 0;
        }
        sc[b] = __ushort_as_half(row < n ? (unsigned short)(blk[0] | (blk[1] << 8)) : (unsigned short)0);
    }
    uint8_t *pair = dst + ((size_t)u * pairs + p) * FR_PAIR_BYTES;
    *reinterpret_cast<uint4 *>(pair + lane * 16) = *reinterpret_cast<const uint4 *>(q);
    // scales: [t][block][2]: rows 2 t and 2 t + 1 of block 0, then of block 1
    if (t == 0)
        for (int b = 0; b < 2; b++) reinterpret_cast<__half *>(pair + 512)[(g >> 1) * 4 + b * 2 + (g & 1)] = sc[b];
}
int fr_retile(const QWeight &w, uint8_t *dst, bool glu, cudaStream_t st) {
    if (!fr_can_tile(w) || (glu && w.n % 8)) { set_error("fr_retile: weight [%d, %d] of format %d has no streaming tiles", w.n, w.k, w.fmt); return -1; }
    const size_t n = (size_t)cdiv(w.n, 8) * (w.k / 64) * 32;
    if (w.fmt == FMT_GGML_Q8_0) fr_retile_kernel<FMT_GGML_Q8_0><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(w.raw, dst, w.n, w.k, glu);
    else fr_retile_kernel<FMT_GGML_Q4_0><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(w.raw, dst, w.n, w.k, glu);
    MB_CUDA(cudaGetLastError());
    note_launch();
    return 0;
}

// ----------------------------------------------------------------------------------------------------- helpers
__device__ __forceinline__ void fr_sync() { asm volatile("bar.sync 1, %0;" ::"n"(FR_THREADS) : "memory"); }   // the computing warps

__device__ __forceinline__ void fr_bulk(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
// not volatile: the products of the four blocks of a piece are independent and may interleave
__device__ __forceinline__ void fr_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four int8 -> two half2, exact: the byte q + 128 under the exponent of 1024, minus 1152
__device__ __forceinline__ void fr_widen(uint32_t q, uint32_t &h0, uint32_t &h1) {
    const uint32_t u = q ^ 0x80808080u;
    const __half2 k = __halves2half2(__ushort_as_half(0xE480), __ushort_as_half(0xE480));       // -1152
    const uint32_t a = __byte_perm(u, 0x64646464u, 0x4140), b = __byte_perm(u, 0x64646464u, 0x4342);
    const __half2 x = __hadd2(*reinterpret_cast<const __half2 *>(&a), k), y = __hadd2(*reinterpret_cast<const __half2 *>(&b), k);
    h0 = *reinterpret_cast<const uint32_t *>(&x);
    h1 = *reinterpret_cast<const uint32_t *>(&y);
}
__device__ __forceinline__ void fr_cp16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fr_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void fr_cp_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

struct alignas(16) FrWeights { const uint8_t *w; int N, K; };

struct FrShared {
    uint8_t *ring;                        // FR_STAGES pieces
    uint8_t *xs;                          // [plane][32 rows]: two slabs of 16 rows, or all slabs of few rows one behind the other
    float *red, *vals;                    // partial sums per warp; finished sums of a group
    uint64_t *full, *empty;
    volatile int *stop;                   // the computing warps have left, or a wait ran out
    const FrWeights *tab;                 // the chain's contractions in order
    float *best_v;                        // running maximum per row of the tile (FR_EPI_ARGMAX)
    int *best_i;
    __device__ __forceinline__ __half *x(int row, int plane) const { return reinterpret_cast<__half *>(xs + plane * FR_XPLANE) + row * FR_XS; }
};

struct FrPlace {                          // the CTA's place
    int ng, row0, rows;                   // unit group, first row and rows of the tile
    int tid, warp, lane;
};

// Every CTA has arrived `target / gridDim.x` times. False: a wait ran out here or elsewhere.
__device__ __forceinline__ bool fr_grid_sync(const FrArgs &a, const FrShared &s, const FrPlace &c, unsigned target) {
    fr_sync();
    if (c.tid == 0) {
        // the block barrier before and the release make the CTA's writes visible with the arrival, the acquire and the block
        // barrier behind it those of the others to all warps
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
        const long long t0 = clock64();
        unsigned v;
        for (int tries = 1;; tries++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
            if (v >= target) break;
            if (tries & 63) continue;
            if (*reinterpret_cast<volatile unsigned *>(a.bar + 1) || clock64() - t0 > (1ll << 31)) {
                atomicExch(a.bar + 1, 1u);
                atomicCAS(a.status, ST_OK, ST_TIMEOUT_EPILOGUE);
                *s.stop = 1;
                break;
            }
        }
    }
    fr_sync();
    return *s.stop == 0;
}

// --------------------------------------------------------------------------------------------------- LayerNorms
// LayerNorm of rows that are spread over 8 / NC warps each: a warp holds the NC 128-wide chunks sub, sub + 8 / NC, .. of its row,
// a lane four columns of each. The statistics are ln_stats' (ln_row.cuh), formed chunk by chunk in chunk order whatever NC is, so
// that a row's bits do not depend on how many rows share the CTA. slot: the exchange buffer of this use. All warps call it.
template <int NC>
__device__ __forceinline__ void fr_ln(const FrShared &s, float4 (&v)[NC], const float *w, const float *b, int K, float first, int row, int sub, int lane, int slot) {
    constexpr int WPR = FR_WARPS / NC;
    const int n4 = K >> 2;
    const double x0 = (double)first, rk = 1.0 / (double)K;
    double2 *part = reinterpret_cast<double2 *>(s.vals) + slot * 64 + row * 8;
    double t[NC], q[NC];
#pragma unroll
    for (int i = 0; i < NC; i++) {
        t[i] = q[i] = 0.0;
        if (lane + 32 * (sub + WPR * i) < n4) {
            const double d0 = (double)v[i].x - x0, d1 = (double)v[i].y - x0, d2 = (double)v[i].z - x0, d3 = (double)v[i].w - x0;
            t[i] = (d0 + d1) + (d2 + d3);
            q[i] = fma(d0, d0, d1 * d1) + fma(d2, d2, d3 * d3);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < NC; i++) { t[i] += __shfl_xor_sync(0xffffffffu, t[i], o); q[i] += __shfl_xor_sync(0xffffffffu, q[i], o); }
#pragma unroll
    for (int i = 0; i < NC; i++) if (lane == 0) part[sub + WPR * i] = make_double2(t[i], q[i]);
    fr_sync();
    double sum = 0.0, sq = 0.0;
#pragma unroll
    for (int j = 0; j < FR_WARPS; j++) { const double2 p = part[j]; sum += p.x; sq += p.y; }
    const double m = sum * rk, ve = fma(-sum, m, sq) * rk + 1e-5;
    const float muf = (float)(x0 + m), inv = (float)rsqrt(ve);
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const int at = lane + 32 * (sub + WPR * i);
        if (at < n4) {
            const float4 ww = reinterpret_cast<const float4 *>(w)[at], bb = reinterpret_cast<const float4 *>(b)[at];
            v[i] = make_float4(((v[i].x - muf) * inv) * ww.x + bb.x, ((v[i].y - muf) * inv) * ww.y + bb.y,
                               ((v[i].z - muf) * inv) * ww.z + bb.z, ((v[i].w - muf) * inv) * ww.w + bb.w);
        }
    }
}

// The turn to AED position p for row b (a warp): the first maximum over the candidate groups is the token of position p - 1;
// `keeper` does the utterance's bookkeeping (src/decoder_aed.c:211-223). Returns the token at p.
__device__ __forceinline__ int fr_aed_turn(const FrArgs &a, int lane, int b, int p, bool keeper) {
    int *st = a.st;
    if (p == 0) return st[b];
    float bv = -3.0e38f;
    int bi = 0x7fffffff;
    for (int i = lane; i < a.ngroups; i += 32) {
        const float v = __ldcg(a.cand_v + (size_t)b * a.ngroups + i);
        const int k = __ldcg(a.cand_i + (size_t)b * a.ngroups + i);
        if (v > bv || (v == bv && k < bi)) { bv = v; bi = k; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v = __shfl_xor_sync(0xffffffffu, bv, o);
        const int k = __shfl_xor_sync(0xffffffffu, bi, o);
        if (v > bv || (v == bv && k < bi)) { bv = v; bi = k; }
    }
    const int B = a.B, n_prompt = st[3 * B + b];
    const int cur = p < n_prompt ? a.prompts[b * a.max_prompt + p] : bi < a.V ? bi : 0;
    if (keeper && lane == 0 && !st[2 * B + b]) {
        bool fin = false;
        if (p >= n_prompt) {
            const int n = st[B + b];
            if (bi == a.eos || n >= st[5 * B + b]) fin = true;
            else { a.tokens[(size_t)b * a.cap_stride + n] = bi; st[B + b] = n + 1; }
        }
        if (p >= st[4 * B + b]) fin = true;
        if (fin) { st[2 * B + b] = 1; atomicAdd(st + 6 * B, 1); }
    }
    return cur;
}

// Rows row0, row0 + 1, .. (n of them, NC at a time) through the operation's LayerNorms. FUSED: into the X tile of a contraction,
// every unit group for itself; else into the planes o_hi, o_lo. first_group: this CTA keeps LN2's rows and an AED row's books.
template <int NC, bool FUSED, bool AED>
__device__ __forceinline__ void fr_rows(const FrArgs &a, const FrOp &op, const FrShared &s, const FrPlace &c, int row0, int n, bool first_group, int p) {
    constexpr int WPR = FR_WARPS / NC;                           // warps per row
    bool fits = true;
    const int K = op.K, n4 = K >> 2, sub = c.warp % WPR, slot = c.warp / WPR;
    // the LayerNorms' vectors, by all threads, into the (idle) sums' place while the rows are on their way
    const bool two = op.rows == FR_ROWS_LN2 || (AED && op.rows == FR_ROWS_AED_NEXT);
    float *lw = s.red, *lb = lw + FR_SLAB, *lw0 = lb + FR_SLAB, *lb0 = lw0 + FR_SLAB;
    for (int i = c.tid; i < n4; i += FR_THREADS) {
        fr_cp16(smem_u32(lw + 4 * i), op.ln_w + 4 * i);
        fr_cp16(smem_u32(lb + 4 * i), op.ln_b + 4 * i);
        if (two) { fr_cp16(smem_u32(lw0 + 4 * i), op.ln0_w + 4 * i); fr_cp16(smem_u32(lb0 + 4 * i), op.ln0_b + 4 * i); }
    }
    fr_cp_commit();
    float *firsts = s.best_v;                                    // the second LayerNorm's first value of every row
    for (int r0 = 0; r0 < n; r0 += NC) {
        const int r = r0 + slot, m = row0 + (r < n ? r : 0);
        const bool on = r < n;
        float4 v[NC];
        float first;
        if (AED && op.rows == FR_ROWS_AED_NEXT) {
            const int cur = fr_aed_turn(a, c.lane, m, p, on && first_group && sub == 0), at = p < a.max_seq ? p : a.max_seq - 1;
            const float *e = a.emb + (size_t)cur * K, *pe = a.pos + (size_t)at * K;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int col = c.lane + 32 * (sub + WPR * i);
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (col < n4) {
                    const float4 x = __ldg(reinterpret_cast<const float4 *>(e) + col), y = __ldg(reinterpret_cast<const float4 *>(pe) + col);
                    v[i] = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
                }
            }
            first = __ldg(e) + __ldg(pe);
        } else {
            const float *x = op.x + (size_t)m * K;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int col = c.lane + 32 * (sub + WPR * i);
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (col < n4) v[i] = __ldcg(reinterpret_cast<const float4 *>(x) + col);
            }
            first = __ldcg(x);
        }
        fr_cp_wait();
        fr_sync();
        if (two) {
            fr_ln<NC>(s, v, lw0, lb0, K, first, slot, sub, c.lane, 0);
            if (first_group && on) {
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    const int col = c.lane + 32 * (sub + WPR * i);
                    if (col < n4) reinterpret_cast<float4 *>(op.x_copy + (size_t)m * K)[col] = v[i];
                }
            }
            if (sub == 0 && c.lane == 0) firsts[slot] = v[0].x;
            fr_sync();
            first = firsts[slot];
        }
        fr_ln<NC>(s, v, lw, lb, K, first, slot, sub, c.lane, 1);
        if (op.rows == FR_ROWS_LN_SILU) {
#pragma unroll
            for (int i = 0; i < NC; i++) v[i] = make_float4(silu_f(v[i].x), silu_f(v[i].y), silu_f(v[i].z), silu_f(v[i].w));
        }
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int col = c.lane + 32 * (sub + WPR * i);
            if (col >= n4 || !on) continue;
            __align__(8) __half h[4], l[4];
            fits &= split_h16(v[i].x, h[0], l[0]); fits &= split_h16(v[i].y, h[1], l[1]);
            fits &= split_h16(v[i].z, h[2], l[2]); fits &= split_h16(v[i].w, h[3], l[3]);
            __half *ph = FUSED ? s.x(r, 0) : op.o_hi + (size_t)m * K, *pl = FUSED ? s.x(r, 1) : op.o_lo + (size_t)m * K;
            *reinterpret_cast<uint2 *>(ph + 4 * col) = *reinterpret_cast<const uint2 *>(h);
            *reinterpret_cast<uint2 *>(pl + 4 * col) = *reinterpret_cast<const uint2 *>(l);
        }
        // (the exchange buffers of the next rows: its first barrier comes after everybody's reads of this round)
    }
    if (!fits) atomicCAS(a.status, ST_OK, ST_RANGE);
}

// --------------------------------------------------------------------------------------------------- contraction
// slab `sl` of the tile's planes to rows `at` on (asynchronous)
__device__ __forceinline__ void fr_stage_planes(const FrOp &op, const FrShared &s, const FrPlace &c, int sl, int ks, int at, bool lo) {
    const int per = ks >> 3, n = c.rows * per;
    for (int i = c.tid; i < n; i += FR_THREADS) {
        const int r = i / per, col = (i - r * per) * 8;
        const size_t o = (size_t)(c.row0 + r) * op.K + (size_t)sl * FR_SLAB + col;
        fr_cp16(smem_u32(s.x(at + r, 0) + col), op.a_hi + o);
        if (lo) fr_cp16(smem_u32(s.x(at + r, 1) + col), op.a_lo + o);
    }
    fr_cp_commit();
}

// the finished sum of (row, column) of unit u of the group: the warps' parts in warp order
__device__ __forceinline__ float fr_sum(const FrShared &s, int u, int row, int col) {
    const int at = (((row & 7) * 4 + (col >> 1)) << 2) + ((row >> 3) << 1) + (col & 1);
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < FR_WARPS; w++) v += s.red[(w * FR_GU + u) * 128 + at];
    return v;
}

// bias and residual of the (up to two) outputs a thread will store, asked for under the products
struct FrPre { float b[2], r[2]; };
__device__ __forceinline__ void fr_prefetch(const FrArgs &a, const FrOp &op, const FrPlace &c, int first, int nu, FrPre &pre) {
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int i = c.tid + q * FR_THREADS, u = i >> 7, row = (i >> 3) & 15, n = (c.ng + (first + u) * a.ngroups) * 8 + (i & 7);
        const bool on = u < nu && row < c.rows && n < op.N && op.epi <= FR_EPI_F32;
        pre.b[q] = on && op.bias ? __ldg(op.bias + n) : 0.f;
        pre.r[q] = on && op.epi == FR_EPI_RESID ? __ldcg(op.res + (size_t)(c.row0 + row) * op.ldo + n) : 0.f;
    }
}

template <bool AED>
__device__ __forceinline__ void fr_epilogue(const FrArgs &a, const FrOp &op, const FrShared &s, const FrPlace &c, int first, int nu, int mine, const FrPre &pre) {
    bool fits = true;                                            // unit of slot u: ng + (first + u) ngroups
    if (op.epi >= FR_EPI_GLU_CONV) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int i = c.tid + q * FR_THREADS, u = i >> 7, row = (i >> 3) & 15, col = i & 7, unit = c.ng + (first + u) * a.ngroups;
            if (u >= nu) continue;
            float v = fr_sum(s, u, row, col);
            const int n = AED ? unit * 8 + col : (col < 4 ? unit * 4 + col : op.N / 2 + unit * 4 + col - 4);
            if (op.bias && n < op.N) v += op.bias[n];
            s.vals[i] = v;
        }
        fr_sync();
        if (AED) {
            const int row = c.tid >> 4, j = c.tid & 15;             // sixteen threads per row
            float bv = -3.0e38f;
            int bi = 0x7fffffff;
            for (int i = j; i < nu * 8; i += 16) {
                const int n = (c.ng + (first + (i >> 3)) * a.ngroups) * 8 + (i & 7);
                const float v = s.vals[(i >> 3) * 128 + row * 8 + (i & 7)];
                if (n < op.N && (v > bv || (v == bv && n < bi))) { bv = v; bi = n; }
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                const float v = __shfl_xor_sync(0xffffffffu, bv, o);
                const int k = __shfl_xor_sync(0xffffffffu, bi, o);
                if (v > bv || (v == bv && k < bi)) { bv = v; bi = k; }
            }
            if (j == 0) {
                if (first == 0 || bv > s.best_v[row] || (bv == s.best_v[row] && bi < s.best_i[row])) { s.best_v[row] = bv; s.best_i[row] = bi; }
                if (first + nu >= mine && row < c.rows) {
                    a.cand_v[(size_t)(c.row0 + row) * a.ngroups + c.ng] = s.best_v[row];
                    a.cand_i[(size_t)(c.row0 + row) * a.ngroups + c.ng] = s.best_i[row];
                }
            }
            return;
        }
        // GLU rows behind the cached ones of their stream, the depthwise taps, the cache moved on
        const int Q = a.Q, ns = c.rows / Q, k = op.conv_k, d = a.d;
        for (int i = c.tid; i < nu * ns * 4; i += FR_THREADS) {
            const int j = i & 3, sl = (i >> 2) % ns, u = (i >> 2) / ns, ch = (c.ng + (first + u) * a.ngroups) * 4 + j, stream = c.row0 / Q + sl;
            float *cc = op.conv_cache + (size_t)stream * (k - 1) * d + ch;
            const float *val = s.vals + u * 128 + sl * Q * 8 + j, *w = op.dw_w + (size_t)ch * k;
            auto glu = [&](int t) { return val[t * 8] * sigmoid_fast(val[t * 8 + 4]); };
            if (k == FR_CONV_K) {                                // the usual width: taps and cached rows in registers
                float wk[FR_CONV_K], row[FR_CONV_K];
#pragma unroll
                for (int r = 0; r < FR_CONV_K; r++) { wk[r] = __ldg(w + r); if (r + 1 < FR_CONV_K) row[r] = cc[(size_t)r * d]; }
                for (int t = 0; t < Q; t++) {
                    row[FR_CONV_K - 1] = glu(t);
                    float o = 0.f;
#pragma unroll
                    for (int r = 0; r < FR_CONV_K; r++) o = fmaf(wk[r], row[r], o);
                    op.out[(size_t)(c.row0 + sl * Q + t) * d + ch] = o;
#pragma unroll
                    for (int r = 0; r + 1 < FR_CONV_K; r++) row[r] = row[r + 1];
                }
#pragma unroll
                for (int r = 0; r + 1 < FR_CONV_K; r++) cc[(size_t)r * d] = row[r];
                continue;
            }
            auto seq = [&](int r) { return r < k - 1 ? cc[(size_t)r * d] : glu(r - (k - 1)); };   // cached rows, then the chunk's
            for (int t = 0; t < Q; t++) {
                float o = 0.f;
                for (int r = 0; r < k; r++) o = fmaf(w[r], seq(t + r), o);
                op.out[(size_t)(c.row0 + sl * Q + t) * d + ch] = o;
            }
            for (int r = 0; r < k - 1; r++) cc[(size_t)r * d] = seq(Q + r);        // r ascending: seq(Q + r) is not yet overwritten
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int i = c.tid + q * FR_THREADS, u = i >> 7, row = (i >> 3) & 15, col = i & 7, n = (c.ng + (first + u) * a.ngroups) * 8 + col, m = c.row0 + row;
        if (u >= nu || row >= c.rows || n >= op.N) continue;
        float v = fr_sum(s, u, row, col) + pre.b[q];
        if (op.act == ACT_SILU) v = v * __frcp_rn(1.0f + __expf(-v));
        else if (op.act == ACT_RELU) v = fmaxf(v, 0.0f);
        if (op.epi == FR_EPI_PLANES) {
            __half h, l;
            fits &= split_h16(v, h, l);
            op.o_hi[(size_t)m * op.N + n] = h;
            op.o_lo[(size_t)m * op.N + n] = l;
        } else if (op.epi == FR_EPI_RESID) {
            op.out[(size_t)m * op.ldo + n] = pre.r[q] + op.alpha * v;
        } else if (op.epi == FR_EPI_QKV && n >= op.n_split) {
            const int e = n - op.n_split, half_n = (op.N - op.n_split) / 2;
            __half h, l;
            fits &= split_h16(v, h, l);
            (e < half_n ? op.o_hi : op.o_lo)[(size_t)m * half_n + (e < half_n ? e : e - half_n)] = h;
        } else {
            op.out[(size_t)m * op.ldo + n] = v;
        }
    }
    if (!fits) atomicCAS(a.status, ST_OK, ST_RANGE);
}

// The products of one piece (unit, slab): acc += this warp's 64-wide parts of K. FULL: a slab of 1024, two parts per warp; else
// parts beyond np do not exist.
template <int TERMS>
__device__ __forceinline__ void fr_pair(const uint8_t *pair, const FrPlace &c, const uint4 (&xh)[2][2], const uint4 (&xl)[2][2], float (&acc)[4]) {
    const uint4 wq = *reinterpret_cast<const uint4 *>(pair + c.lane * 16);
    const uint2 sc = *reinterpret_cast<const uint2 *>(pair + 512 + (c.lane & 3) * 8);
    float ch[2][4], cl[2][4];
    uint32_t w[2][4];
#pragma unroll
    for (int b = 0; b < 2; b++) {
        fr_widen(b ? wq.z : wq.x, w[b][0], w[b][1]);
        fr_widen(b ? wq.w : wq.y, w[b][2], w[b][3]);
#pragma unroll
        for (int i = 0; i < 4; i++) ch[b][i] = cl[b][i] = 0.f;
    }
#pragma unroll
    for (int b = 0; b < 2; b++) {
        fr_mma(ch[b], xh[b][0].x, xh[b][1].x, xh[b][0].y, xh[b][1].y, w[b][0], w[b][1]);
        if (TERMS > 1) fr_mma(cl[b], xl[b][0].x, xl[b][1].x, xl[b][0].y, xl[b][1].y, w[b][0], w[b][1]);
    }
#pragma unroll
    for (int b = 0; b < 2; b++) {
        fr_mma(ch[b], xh[b][0].z, xh[b][1].z, xh[b][0].w, xh[b][1].w, w[b][2], w[b][3]);
        if (TERMS > 1) fr_mma(cl[b], xl[b][0].z, xl[b][1].z, xl[b][0].w, xl[b][1].w, w[b][2], w[b][3]);
    }
#pragma unroll
    for (int b = 0; b < 2; b++) {
        const float2 d = __half22float2(*reinterpret_cast<const __half2 *>(b ? &sc.y : &sc.x));
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i] = fmaf((i & 1) ? d.y : d.x, TERMS > 1 ? fmaf(cl[b][i], H16_LO_INV, ch[b][i]) : ch[b][i], acc[i]);
    }
}

// One slab of a group of nu units: the rows' fragments stay in registers for all of them.
template <int TERMS, bool FULL>
__device__ __forceinline__ bool fr_slab(const FrArgs &a, const FrShared &s, const FrPlace &c, int xrow, int np, int nu, unsigned &it, bool ok, float (&acc)[FR_GU][4]) {
    const int g = c.lane >> 2, t = c.lane & 3;
    uint4 xh[2][2][2], xl[2][2][2];                              // [part][block][row g / g + 8]
    // a row that the tile does not have is the first one again; its sums are never stored
    const int r0 = xrow + (g < c.rows ? g : 0), r1 = xrow + (g + 8 < c.rows ? g + 8 : 0);
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int pr = c.warp + q * FR_WARPS;
        if (!FULL && pr >= np) continue;
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int at = pr * 64 + b * 32 + 8 * t;
            xh[q][b][0] = *reinterpret_cast<const uint4 *>(s.x(r0, 0) + at);
            xh[q][b][1] = *reinterpret_cast<const uint4 *>(s.x(r1, 0) + at);
            if (TERMS > 1) {
                xl[q][b][0] = *reinterpret_cast<const uint4 *>(s.x(r0, 1) + at);
                xl[q][b][1] = *reinterpret_cast<const uint4 *>(s.x(r1, 1) + at);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < FR_GU; u++) {
        if (u >= nu) break;
        const unsigned stg = it % FR_STAGES;
        if (ok && !__all_sync(0xffffffffu, mbar_wait(&s.full[stg], (it / FR_STAGES) & 1))) {
            ok = false;
            if (c.lane == 0) { *s.stop = 1; atomicExch(a.bar + 1, 1u); atomicCAS(a.status, ST_OK, ST_TIMEOUT_MMA); }
        }
        it++;
        if (!ok) continue;
        const uint8_t *piece = s.ring + stg * FR_PIECE + c.warp * FR_PAIR_BYTES;
#pragma unroll
        for (int q = 0; q < 2; q++)
            if (FULL || c.warp + q * FR_WARPS < np) fr_pair<TERMS>(piece + q * FR_WARPS * FR_PAIR_BYTES, c, xh[q], xl[q], acc[u]);
        __syncwarp();
        if (c.lane == 0) mbar_arrive(&s.empty[stg]);
    }
    return ok;
}

// One contraction over this CTA's rows and units. it: ring pieces consumed so far. A wait that runs out sets the stop flag;
// the warp then goes through the rest without waiting or computing, and the grid barrier behind the operation ends it all.
template <bool AED, int TERMS>
__device__ __forceinline__ void fr_gemm(const FrArgs &a, const FrOp &op, const FrShared &s, const FrPlace &c, int p, unsigned &it) {
    const int units = (op.N + 7) >> 3, mine = units > c.ng ? (units - c.ng + a.ngroups - 1) / a.ngroups : 0;
    const int ks = op.K < FR_SLAB ? op.K : FR_SLAB, slabs = op.K <= FR_SLAB ? 1 : op.K / FR_SLAB, np = ks >> 6;
    if (AED && op.epi == FR_EPI_ARGMAX && mine == 0 && c.tid < c.rows) {
        a.cand_v[(size_t)(c.row0 + c.tid) * a.ngroups + c.ng] = -3.0e38f;
        a.cand_i[(size_t)(c.row0 + c.tid) * a.ngroups + c.ng] = 0x7fffffff;
    }
    const bool planes = op.rows == FR_ROWS_PLANES, all = c.rows * slabs <= 32;
    if (!planes) {
        // group 0 leaves LN2's rows behind and keeps the AED books even where no unit is its own
        if (mine > 0 || c.ng == 0) {
            if (c.rows == 1) fr_rows<1, true, AED>(a, op, s, c, c.row0, c.rows, c.ng == 0, p);
            else if (c.rows == 2) fr_rows<2, true, AED>(a, op, s, c, c.row0, c.rows, c.ng == 0, p);
            else fr_rows<4, true, AED>(a, op, s, c, c.row0, c.rows, c.ng == 0, p);
        }
        fr_sync();
    }
    if (mine == 0) return;
    bool ok = true;
    for (int first = 0; first < mine; first += FR_GU) {
        const int nu = mine - first < FR_GU ? mine - first : FR_GU;
        float acc[FR_GU][4];
#pragma unroll
        for (int u = 0; u < FR_GU; u++) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.f;
        // few rows: all slabs are asked for at once, and once; else two slabs in turn, again for every group of units
        if (planes && first == 0 && all) {
            for (int sl = 0; sl < slabs; sl++) fr_stage_planes(op, s, c, sl, ks, sl * c.rows, TERMS > 1);
        } else if (planes && !all) {
            if (first) fr_sync();
            fr_stage_planes(op, s, c, 0, ks, 0, TERMS > 1);
        }
        FrPre pre;
        fr_prefetch(a, op, c, first, nu, pre);
        for (int sl = 0; sl < slabs; sl++) {
            if (planes && (!all || (first == 0 && sl == 0))) {
                fr_cp_wait();
                fr_sync();
                if (!all && sl + 1 < slabs) fr_stage_planes(op, s, c, sl + 1, ks, ((sl + 1) & 1) * 16, TERMS > 1);
            }
            const int xrow = !planes ? 0 : all ? sl * c.rows : (sl & 1) * 16;
            if (np == FR_PAIRS) ok = fr_slab<TERMS, true>(a, s, c, xrow, np, nu, it, ok, acc);
            else ok = fr_slab<TERMS, false>(a, s, c, xrow, np, nu, it, ok, acc);
        }
#pragma unroll
        for (int u = 0; u < FR_GU; u++)
            if (u < nu) *reinterpret_cast<float4 *>(s.red + (c.warp * FR_GU + u) * 128 + c.lane * 4) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
        fr_sync();
        fr_epilogue<AED>(a, op, s, c, first, nu, mine, pre);
        if (first + FR_GU < mine) fr_sync();                     // the sums are read before the next group writes its own
    }
}

// The producer warp asks for every piece of every contraction in the order the warps use them: groups of FR_GU units, in a
// group slab by slab, unit by unit.
__device__ __forceinline__ void fr_produce(const FrArgs &a, const FrShared &s, const FrPlace &c) {
    unsigned it = 0;
    bool ok = true;
    for (int p = 0; p <= a.positions && ok; p++)
        for (int i = 0; i < a.n_gemms && ok; i++) {
            const int units = (s.tab[i].N + 7) >> 3, K = s.tab[i].K, ks = K < FR_SLAB ? K : FR_SLAB, slabs = K <= FR_SLAB ? 1 : K / FR_SLAB;
            const uint32_t bytes = (uint32_t)(ks >> 6) * FR_PAIR_BYTES;
            const size_t step = (size_t)a.ngroups * slabs * bytes;
            const uint8_t *w = s.tab[i].w + (size_t)c.ng * slabs * bytes;
            for (int left = units > c.ng ? (units - c.ng + a.ngroups - 1) / a.ngroups : 0; left > 0 && ok; left -= FR_GU, w += FR_GU * step)
                for (int sl = 0; sl < slabs && ok; sl++)
                    for (int u = 0; u < FR_GU && u < left; u++) {
                        const unsigned stg = it % FR_STAGES;
                        const long long t0 = clock64();
                        while (!mbar_try_wait(&s.empty[stg], ((it / FR_STAGES) & 1) ^ 1))
                            // other CTAs may hold the chain up at a barrier: give up when the computing warps have (their waits are shorter)
                            if (*s.stop || clock64() - t0 > (1ll << 33)) { ok = false; break; }
                        if (!ok) break;
                        mbar_expect_tx(&s.full[stg], bytes);
                        fr_bulk(smem_u32(s.ring + stg * FR_PIECE), w + u * step + (size_t)sl * bytes, bytes, &s.full[stg]);
                        it++;
                    }
        }
    // copies still in flight must land before the CTA's shared memory goes away
    for (unsigned j = it > FR_STAGES ? it - FR_STAGES : 0; j < it; j++) mbar_wait(&s.full[j % FR_STAGES], (j / FR_STAGES) & 1);
}

// ---------------------------------------------------------------------------------------------------- attentions
// One query over n keys, in eight lists: list w holds the keys w, w + 8, ... A warp walks a list in rounds of KB keys: all key
// and value rows of a round are asked for at once (one round covers a list of the usual 71 streaming keys), the scores stay in
// its lanes, the softmax is a running maximum per list. A lane owns four columns; dk is a multiple of 4 up to 128. The lists
// meet in fr_context, in list order: the bits are the same whether eight warps take one list each or one warp takes all.
bool fr_attn_fits(int dk) { return dk % 4 == 0 && dk <= 128; }

// load(j, u) fetches key and value of key j into slot u, score(u) is the lane's part of the dot product, value(u) its columns
template <int KB, typename FL, typename FS, typename FV>
__device__ __forceinline__ void fr_list(float *part, float2 *ml, int list, int n, int dk, int lane, FL load, FS score, FV value) {
    const bool on = lane * 4 < dk;
    float m = -INFINITY, l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = list; j0 < n; j0 += KB * FR_WARPS) {
#pragma unroll
        for (int u = 0; u < KB; u++) load(j0 + FR_WARPS * u < n ? j0 + FR_WARPS * u : j0, u);
        float sc[KB], mx = m;
#pragma unroll
        for (int u = 0; u < KB; u++) sc[u] = on ? score(u) : 0.f;
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1)
#pragma unroll
            for (int u = 0; u < KB; u++) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o2);
#pragma unroll
        for (int u = 0; u < KB; u++) { if (j0 + FR_WARPS * u >= n) sc[u] = -INFINITY; mx = fmaxf(mx, sc[u]); }
        const float f = expf(m - mx);
        m = mx; l *= f;
        o.x *= f; o.y *= f; o.z *= f; o.w *= f;
#pragma unroll
        for (int u = 0; u < KB; u++) {
            const float w = expf(sc[u] - m);
            const float4 v = value(u);
            l += w;
            o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
        }
    }
    if (on) *reinterpret_cast<float4 *>(part + list * 128 + lane * 4) = o;
    if (lane == 0) ml[list] = make_float2(m, l);
}
__device__ __forceinline__ void fr_context(const FrOp &op, const float *part, const float2 *ml, size_t out, int i) {
    float mx = ml[0].x, sum = 0.f, v = 0.f;
#pragma unroll
    for (int w = 1; w < FR_WARPS; w++) mx = fmaxf(mx, ml[w].x);
#pragma unroll
    for (int w = 0; w < FR_WARPS; w++) {
        const float f = expf(ml[w].x - mx);                      // an empty list: exp(-inf) = 0
        sum = fmaf(f, ml[w].y, sum);
        v = fmaf(f, part[w * 128 + i], v);
    }
    __half hi, lo;
    split_h16(v / sum, hi, lo);
    op.o_hi[out + i] = hi;
    op.o_lo[out + i] = lo;
}
__device__ __forceinline__ float4 fr_unpack(uint2 a) {
    const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(&a.x)), y = __half22float2(*reinterpret_cast<const __half2 *>(&a.y));
    return make_float4(x.x, x.y, y.x, y.y);
}
__device__ __forceinline__ uint2 fr_ld8(const __half *p) { return __ldcg(reinterpret_cast<const uint2 *>(p)); }
__device__ __forceinline__ float fr_dot(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }

// score(t, j) = ((q_t + u) . k_j + (q_t + v) . rk[K - 1 - valid - t + j]) / sqrt(dk) over [cached frames ; chunk]; afterwards the
// chunk's k / v rows go to their ring slots (update_kv_cache, src/encoder.c:763-776): a (stream, head) is read by its own task alone.
__device__ __forceinline__ void fr_stream_attn(const FrArgs &a, const FrOp &op, const FrShared &s, const FrPlace &c, int start) {
    constexpr int KB = 9;
    const int H = a.H, dk = a.dk, d = a.d, Q = a.Q, left = a.left, valid = a.valid, K = valid + Q, tasks = a.S * H;
    // one task per warp when there are enough of them to fill the chip (no block barriers, loads of eight tasks in flight per
    // SM), else one per CTA (64 streams x 8 heads: 39 k -> 15 k cycles)
    const bool warps = tasks >= 3 * (int)gridDim.x;
    float *part = reinterpret_cast<float *>(s.xs) + (warps ? c.warp * FR_WARPS * 128 : 0);
    float2 *ml = reinterpret_cast<float2 *>(s.red) + (warps ? c.warp * FR_WARPS : 0);
    const float scale = 1.0f / sqrtf((float)dk);
    const int i0 = c.lane * 4 < dk ? c.lane * 4 : 0;
    for (int task = warps ? c.warp * gridDim.x + blockIdx.x : blockIdx.x; task < tasks; task += warps ? FR_WARPS * gridDim.x : gridDim.x) {
        const int st = task / H, h = task - st * H;
        const size_t cbase = ((size_t)st * H + h) * left * dk, nbase = (size_t)st * Q * d + h * dk;
        for (int t = 0; t < Q; t++) {
            const size_t row = (size_t)st * Q + t;
            const __half *rk = op.rk + (size_t)(K - 1 - valid - t) * op.ldrk + h * dk + i0;
            const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(op.q + row * op.ldq + h * dk + i0));
            const float4 bu = __ldg(reinterpret_cast<const float4 *>(op.bias_u + h * dk + i0)), bv = __ldg(reinterpret_cast<const float4 *>(op.bias_v + h * dk + i0));
            const float4 qu = make_float4(q4.x + bu.x, q4.y + bu.y, q4.z + bu.z, q4.w + bu.w), qv = make_float4(q4.x + bv.x, q4.y + bv.y, q4.z + bv.z, q4.w + bv.w);
            uint2 kk[KB], rr[KB], vv[KB];
            auto load = [&](int j, int u) {
                int x = start + j;
                if (x >= left) x -= left;
                const size_t o = j < valid ? cbase + (size_t)x * dk + i0 : nbase + (size_t)(j - valid) * d + i0;
                kk[u] = fr_ld8((j < valid ? op.kc : op.kn) + o);
                rr[u] = fr_ld8(rk + (size_t)j * op.ldrk);
                vv[u] = fr_ld8((j < valid ? op.vc : op.vn) + o);
            };
            auto score = [&](int u) { return (fr_dot(qu, fr_unpack(kk[u])) + fr_dot(qv, fr_unpack(rr[u]))) * scale; };
            auto value = [&](int u) { return fr_unpack(vv[u]); };
            for (int list = warps ? 0 : c.warp; list < (warps ? FR_WARPS : c.warp + 1); list++) fr_list<KB>(part, ml, list, K, dk, c.lane, load, score, value);
            if (warps) {
                __syncwarp();
                for (int i = c.lane; i < dk; i += 32) fr_context(op, part, ml, row * d + h * dk, i);
                __syncwarp();
            } else {
                fr_sync();
                if (c.tid < dk) fr_context(op, part, ml, row * d + h * dk, c.tid);
                fr_sync();
            }
        }
        const int i1 = warps ? c.lane : c.tid, step = warps ? 32 : FR_THREADS;
        for (int i = i1; i < Q * dk; i += step) {
            const int t = i / dk, e = i - t * dk;
            int x = start + valid + t;
            while (x >= left) x -= left;
            op.kc[cbase + (size_t)x * dk + e] = __ldcg(op.kn + nbase + (size_t)t * d + e);
            op.vc[cbase + (size_t)x * dk + e] = __ldcg(op.vn + nbase + (size_t)t * d + e);
        }
    }
}

// One query per utterance over its own past (src/decoder_aed.c:186-197), f32 cache [B][max_len][d].
__device__ __forceinline__ void fr_aed_self(const FrArgs &a, const FrOp &op, const FrShared &s, const FrPlace &c, int p) {
    constexpr int KB = 10;
    const int H = a.H, dk = a.dk, d = a.d;
    float *part = reinterpret_cast<float *>(s.xs);
    float2 *ml = reinterpret_cast<float2 *>(s.red);
    const float scale = 1.0f / sqrtf((float)dk);
    const int i0 = c.lane * 4 < dk ? c.lane * 4 : 0;
    for (int task = blockIdx.x; task < a.B * H; task += gridDim.x) {
        const int b = task / H, h = task - b * H;
        const float *row = op.q + (size_t)b * op.ldq + h * dk;
        float *Kc = op.ck + (size_t)b * a.max_len * d + h * dk, *Vc = op.cv + (size_t)b * a.max_len * d + h * dk;
        const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(row + i0));
        float4 kk[KB], vv[KB];
        fr_list<KB>(part, ml, c.warp, p + 1, dk, c.lane,
                    [&](int j, int u) {                          // this position's row straight from the projection
                        kk[u] = __ldcg(reinterpret_cast<const float4 *>(j < p ? Kc + (size_t)j * d + i0 : row + d + i0));
                        vv[u] = __ldcg(reinterpret_cast<const float4 *>(j < p ? Vc + (size_t)j * d + i0 : row + 2 * d + i0));
                    },
                    [&](int u) { return fr_dot(q4, kk[u]) * scale; }, [&](int u) { return vv[u]; });
        fr_sync();
        if (c.tid < dk) {
            Kc[(size_t)p * d + c.tid] = __ldcg(row + d + c.tid);
            Vc[(size_t)p * d + c.tid] = __ldcg(row + 2 * d + c.tid);
            fr_context(op, part, ml, (size_t)b * d + h * dk, c.tid);
        }
        fr_sync();
    }
}

// One query per utterance over its projected encoder frames (src/decoder_aed.c:199-202), (hi, lo) planes by (utterance, head).
__device__ __forceinline__ void fr_aed_cross(const FrArgs &a, const FrOp &op, const FrShared &s, const FrPlace &c) {
    constexpr int KB = 11;
    const int H = a.H, dk = a.dk, d = a.d;
    float *part = reinterpret_cast<float *>(s.xs);
    float2 *ml = reinterpret_cast<float2 *>(s.red);
    const float scale = 1.0f / sqrtf((float)dk);
    const int i0 = c.lane * 4 < dk ? c.lane * 4 : 0;
    for (int task = blockIdx.x; task < a.B * H; task += gridDim.x) {
        const int b = task / H, h = task - b * H, T = a.enc_len[b];
        const size_t kb = ((size_t)a.enc_off[b] * H + (size_t)h * T) * dk + i0;
        const __half *khp = op.a_hi + kb, *klp = op.a_lo + kb, *vhp = khp + a.v_off, *vlp = klp + a.v_off;
        const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(op.q + (size_t)b * op.ldq + h * dk + i0));
        uint2 kh[KB], kl[KB], vh[KB], vl[KB];
        auto join = [&](uint2 x, uint2 y) {
            const float4 h4 = fr_unpack(x), l4 = fr_unpack(y);
            return make_float4(fmaf(l4.x, H16_LO_INV, h4.x), fmaf(l4.y, H16_LO_INV, h4.y), fmaf(l4.z, H16_LO_INV, h4.z), fmaf(l4.w, H16_LO_INV, h4.w));
        };
        fr_list<KB>(part, ml, c.warp, T, dk, c.lane,
                    [&](int j, int u) {
                        const int o = j * dk;
                        kh[u] = __ldg(reinterpret_cast<const uint2 *>(khp + o)); kl[u] = __ldg(reinterpret_cast<const uint2 *>(klp + o));
                        vh[u] = __ldg(reinterpret_cast<const uint2 *>(vhp + o)); vl[u] = __ldg(reinterpret_cast<const uint2 *>(vlp + o));
                    },
                    [&](int u) { return fr_dot(q4, join(kh[u], kl[u])) * scale; }, [&](int u) { return join(vh[u], vl[u]); });
        fr_sync();
        if (c.tid < dk) fr_context(op, part, ml, (size_t)b * d + h * dk, c.tid);
        fr_sync();
    }
}

template <bool AED, int TERMS>
__global__ void __launch_bounds__(FR_LAUNCH, 1)
fr_kernel(const __grid_constant__ FrArgs a) {
    extern __shared__ __align__(128) uint8_t fr_smem[];
    __shared__ uint64_t bars[2 * FR_STAGES];
    __shared__ int stop_flag;
    __shared__ float best_v[16];
    __shared__ int best_i[16];
    __shared__ FrOp ops[2];                                      // this operation and the next one
    FrShared s;
    s.ring = fr_smem;
    s.xs = s.ring + FR_STAGES * FR_PIECE;
    s.red = reinterpret_cast<float *>(s.xs + 2 * FR_XPLANE);
    s.vals = s.red + FR_RED_FLOATS;
    s.tab = reinterpret_cast<const FrWeights *>(s.vals + FR_VALS);
    s.full = bars; s.empty = bars + FR_STAGES; s.stop = &stop_flag; s.best_v = best_v; s.best_i = best_i;
    FrPlace c;
    c.tid = threadIdx.x; c.warp = threadIdx.x >> 5; c.lane = threadIdx.x & 31;
    c.ng = blockIdx.x / a.mtiles;
    c.row0 = (blockIdx.x % a.mtiles) * a.tile_rows;
    c.rows = a.M - c.row0 < a.tile_rows ? a.M - c.row0 : a.tile_rows;
    if (threadIdx.x == 0) {
        stop_flag = 0;
        for (int i = 0; i < FR_STAGES; i++) { mbar_init(&s.full[i], 1); mbar_init(&s.empty[i], FR_WARPS); }
        mbar_fence_init();
    }
    for (int i = threadIdx.x; i < a.n_gemms; i += FR_LAUNCH) const_cast<FrWeights *>(s.tab)[i] = static_cast<const FrWeights *>(a.weights)[i];
    for (int i = threadIdx.x; i < (int)(sizeof(FrOp) / 4); i += FR_LAUNCH) reinterpret_cast<int *>(&ops[0])[i] = reinterpret_cast<const int *>(a.ops)[i];
    __syncthreads();
    // registers move from the producer's warpgroup to the two that compute: 256 x 232 + 128 x 24 of the 384 x 168 launched
    if (c.warp >= FR_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        if (c.warp == FR_WARPS && c.lane == 0) fr_produce(a, s, c);
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
    unsigned it = 0, target = 0;
    const int rounds = AED ? a.positions + 1 : 1, start = AED ? 0 : *a.d_start;
    bool go = true;
    for (int p = 0; p < rounds && go; p++)
        for (int i = 0; i < a.n_ops && go; i++) {
            const FrOp &op = ops[i & 1];
            // the turn that opened this position counted the utterances that are done (all CTAs read it behind its barrier)
            if (AED && i == 1 && *reinterpret_cast<volatile int *>(a.st + 6 * a.B) >= a.B) { go = false; break; }
            {   // the next operation's description arrives meanwhile
                const int nx = i + 1 < a.n_ops ? i + 1 : 0;
                if (c.tid < (int)(sizeof(FrOp) / 16)) fr_cp16(smem_u32(&ops[(i + 1) & 1]) + c.tid * 16, reinterpret_cast<const uint8_t *>(a.ops + nx) + c.tid * 16);
                fr_cp_commit();
            }
            if (op.type == FR_GEMM) fr_gemm<AED, TERMS>(a, op, s, c, p, it);
            else if (op.type == FR_LN) {
                for (int m = blockIdx.x; m < a.M; m += gridDim.x) {
                    if (m != (int)blockIdx.x) fr_sync();
                    fr_rows<1, false, AED>(a, op, s, c, m, 1, true, p);
                }
            } else if (!AED && op.type == FR_STREAM_ATTN) fr_stream_attn(a, op, s, c, start);
            else if (AED && op.type == FR_AED_SELF) fr_aed_self(a, op, s, c, p);
            else if (AED && op.type == FR_AED_CROSS) fr_aed_cross(a, op, s, c);
            if (p + 1 == rounds && i + 1 == a.n_ops) break;
            fr_cp_wait();                                        // (the grid barrier begins with a block barrier)
            target += gridDim.x;
            go = fr_grid_sync(a, s, c, target);
        }
    fr_sync();
    if (c.tid == 0) *s.stop = 1;                                 // the producer may be waiting for room that nobody will make
}

// ------------------------------------------------------------------------------------------------------ host side
int fr_grid(int M, int tile_rows, int *mtiles, int *ngroups) {
    *mtiles = cdiv(M, tile_rows);
    *ngroups = device_sm_count() / *mtiles;
    return *ngroups >= 1 ? 0 : -1;
}

// The device table of a chain: the operations, then the weights of its contractions in order.
size_t fr_table_bytes(size_t n_ops) { return n_ops * (sizeof(FrOp) + sizeof(FrWeights)); }
std::vector<uint8_t> fr_table(const std::vector<FrOp> &ops) {
    std::vector<uint8_t> t(fr_table_bytes(ops.size()), 0);
    memcpy(t.data(), ops.data(), ops.size() * sizeof(FrOp));
    FrWeights *w = reinterpret_cast<FrWeights *>(t.data() + ops.size() * sizeof(FrOp));
    for (const FrOp &o : ops) if (o.type == FR_GEMM) { w->w = o.w; w->N = o.N; w->K = o.K; w++; }
    return t;
}

int fr_launch(FrArgs a, const std::vector<FrOp> &ops, const void *table, cudaStream_t st) {
    a.ops = static_cast<const FrOp *>(table);
    a.weights = a.ops + ops.size();
    a.n_ops = (int)ops.size();
    a.n_gemms = 0;
    for (const FrOp &o : ops) a.n_gemms += o.type == FR_GEMM;
    if (a.n_gemms > FR_MAX_GEMMS) { set_error("fr_launch: %d contractions in one chain", a.n_gemms); return -1; }
    if (a.positions > 0 && a.n_ops % 2) { set_error("fr_launch: an odd chain repeats out of step with its description slots"); return -1; }
    void (*kernel)(FrArgs) = a.positions > 0 ? (a.terms > 1 ? fr_kernel<true, 3> : fr_kernel<true, 1>) : (a.terms > 1 ? fr_kernel<false, 3> : fr_kernel<false, 1>);
    static PerDevice configured = {};
    int dev = 0;
    if (configured.below((size_t)FR_SMEM, &dev)) {
        for (void (*k)(FrArgs) : {fr_kernel<true, 3>, fr_kernel<true, 1>, fr_kernel<false, 3>, fr_kernel<false, 1>})
            MB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, FR_SMEM));
        configured.record(dev, (size_t)FR_SMEM);
    }
    MB_CUDA(cudaMemsetAsync(a.bar, 0, 2 * sizeof(unsigned), st));
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(a.mtiles * a.ngroups); lc.blockDim = dim3(FR_LAUNCH); lc.dynamicSmemBytes = FR_SMEM; lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;                   // the barriers need every CTA on an SM
    at[0].val.cooperative = 1;
    lc.attrs = at; lc.numAttrs = 1;
    MB_CUDA(cudaLaunchKernelEx(&lc, kernel, a));
    note_launch();
    return 0;
}

}  // namespace mb
