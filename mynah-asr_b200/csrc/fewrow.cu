// The few-row chains as one persistent kernel.
//
// A streaming step or an AED position is a few hundred dependent operations of at most 128 rows. As launches, chained and
// replayed from a graph, each of them costs 9-11 us (set-up, tensor-memory allocation, slice sums over a cluster, LayerNorm
// by the last warp to arrive) where its bytes would need one. Here one cooperative launch walks the whole chain; what
// separates two operations is a barrier over the CTAs of a row tile (about 1.6 us, the next weights asked for within it):
//   * a CTA keeps its place: a row tile of at most sixteen rows and every ngroups-th unit of eight weight rows. It sums a
//     unit over all of K itself (sixteen warps take 64-wide pieces of K, added in warp order), so nothing is exchanged
//     between CTAs inside an operation, and a row's bits do not depend on how many other rows there are;
//   * weights are the stored 8-bit blocks (1.06 bytes per parameter instead of 4 as operand planes) in fragment order; every
//     warp copies its pieces ahead into a ring of its own, through the barriers, so that HBM works while the chain waits;
//   * the products are mma.sync m16n8k16 on the integers themselves (exact in fp16) against the activations' (hi, lo)
//     planes, summed per 32-element block, then one f32 multiply-add per block with its scale: the quantised weight is
//     never rounded. (tcgen05 wants 128 rows on one side: a unit of eight weight rows per SM is what keeps all SMs busy
//     with N = 1024 and no exchange of partial sums.)
//   * the LayerNorms are computed where their result is staged, by every CTA. The conv module's middle sits in the epilogue
//     of the contraction before it.
// Measured: a step of 24 layers of d = 1024 takes 1.17 ms for one stream (2.74 as launches), 2.25 for 22, 3.7 for 64 with
// decoding (4.8), 4.85 for 120 (5.9); AED of the Canary shape (32 encoder layers, 4 decoder layers: 33 operations a position)
// takes 34 ms for one sentence of 10 s (180 positions), 44.5 for eight; 64 positions of the decoder alone 10.9 ms (19.3 as
// launches, with f32 weights), 13.3 for eight (20.1), 22.8 for 32 (25.1). An operation is 9.5 k cycles with one row, 11.2 to
// 11.4 k with eight and 15 to 16 k with sixteen, of which the barrier is 3 k.
// Values that other CTAs write are read past the L1 (ld.cg, cp.async.cg). All waits are bounded: one that runs out sets the
// status word and the abort flag, and every CTA leaves.
#include "fewrow.h"

#include <string.h>

#include "kernels.h"
#include "ln_row.cuh"

namespace mb {

static constexpr int FR_WARPS = 16, FR_THREADS = FR_WARPS * 32;
static constexpr int FR_SLAB = 1024;                     // K per staged slab and per piece of a unit: 64 for each warp
static constexpr int FR_PAIR_BYTES = 544;                // 64 k x 8 rows: 512 bytes of quants, 32 of scales
static constexpr int FR_AHEAD = 6;                       // pieces of weights a warp has asked for
static constexpr int FR_CT = 160;                        // floats of a warp's sums of two units and eight rows (fr_red)
static constexpr int FR_CONV_K = 9;                      // depthwise width with a register path
static constexpr int FR_LISTS = 16;                      // lists of keys of an attention
static constexpr int FR_XS = FR_SLAB + 32;               // halves per staged row: rows four 16-byte columns apart, no bank conflicts
static constexpr int FR_XPLANE = 32 * FR_XS * 2;         // bytes of one plane of 32 rows
static constexpr int FR_RED_FLOATS = FR_WARPS * 4 * FR_CT;
static_assert(16 * FR_XS * 2 >= 4 * FR_SLAB * 4, "LayerNorm vectors behind the rows of a tile");
static_assert(2 * FR_XPLANE >= FR_WARPS * FR_LISTS * 128 * 4, "lists of an attention per warp");
static_assert(FR_RED_FLOATS >= 8 * 8 * 32 * 4, "exchange of the LayerNorms' sums");

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
            q[8 * b + j] = (uint8_t)((row < n ? v : 0) + 128);
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
__device__ __forceinline__ void fr_sync() { __syncthreads(); }

// not volatile: the products of the four blocks of a piece are independent and may interleave
__device__ __forceinline__ void fr_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// four bytes q + 128 -> two half2 of q, exact: the byte under the exponent of 1024, minus 1152
__device__ __forceinline__ void fr_widen(uint32_t q, uint32_t &h0, uint32_t &h1) {
    const __half2 k = __halves2half2(__ushort_as_half(0xE480), __ushort_as_half(0xE480));       // -1152
    const uint32_t a = __byte_perm(q, 0x64646464u, 0x4140), b = __byte_perm(q, 0x64646464u, 0x4342);
    const __half2 x = __hadd2(*reinterpret_cast<const __half2 *>(&a), k), y = __hadd2(*reinterpret_cast<const __half2 *>(&b), k);
    h0 = *reinterpret_cast<const uint32_t *>(&x);
    h1 = *reinterpret_cast<const uint32_t *>(&y);
}
__device__ __forceinline__ void fr_cp16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fr_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void fr_cp_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void fr_cp_wait_but() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Shared memory by fixed offsets: nothing of it takes a register.
extern __shared__ __align__(128) uint8_t fr_smem[];
struct FrShared {
    static constexpr int RING = 0, XS = FR_AHEAD * FR_WARPS * FR_PAIR_BYTES, RED = XS + 2 * FR_XPLANE, VALS = RED + FR_RED_FLOATS * 4, OPS = VALS + FR_THREADS * 4,
                         BEST = OPS + 2 * (int)sizeof(FrOp), STOP = BEST + 128, END = STOP + 16;
    template <typename T> static __device__ __forceinline__ T *at(int o) { return reinterpret_cast<T *>(fr_smem + o); }
    static __device__ __forceinline__ uint8_t *ring(int warp, int slot) { return fr_smem + RING + (warp * FR_AHEAD + slot) * FR_PAIR_BYTES; }
    // [plane][32 rows]: two slabs of 16 rows, or all slabs of few rows one behind the other
    static __device__ __forceinline__ __half *x(int row, int plane) { return at<__half>(XS + plane * FR_XPLANE) + row * FR_XS; }
    static __device__ __forceinline__ float *red() { return at<float>(RED); }                   // partial sums per warp
    static __device__ __forceinline__ float *vals() { return at<float>(VALS); }                 // finished sums of a group
    static __device__ __forceinline__ FrOp &op(unsigned i) { return at<FrOp>(OPS)[i & 1]; }     // this operation and the next one
    static __device__ __forceinline__ float *best_v() { return at<float>(BEST); }               // running maximum per row (FR_EPI_ARGMAX)
    static __device__ __forceinline__ int *best_i() { return at<int>(BEST + 64); }
    static __device__ __forceinline__ volatile int *stop() { return at<int>(STOP); }            // a wait ran out
};
static_assert(FrShared::END <= 232448, "shared memory");
static constexpr int FR_SMEM = FrShared::END;

struct FrPlace {                          // the CTA's place
    int ng, mt, row0, rows;               // unit group, row tile, its first row and rows
    int tid, warp, lane;
};

// The LayerNorm vectors of a contraction, asked for ahead of it: behind the rows of its tile, where nothing else is then.
__device__ __forceinline__ float *fr_vectors() { return reinterpret_cast<float *>(FrShared::x(16, 0)); }
__device__ __forceinline__ void fr_ask_vectors(const FrOp &op, int tid, int n) {
    if (op.type != FR_GEMM || op.rows == FR_ROWS_PLANES) return;
    const bool two = op.rows == FR_ROWS_LN2 || op.rows == FR_ROWS_AED_NEXT;
    const uint32_t v = smem_u32(fr_vectors());
    for (int i = tid; i < op.K >> 2; i += n) {
        fr_cp16(v + 16 * i, op.ln_w + 4 * i);
        fr_cp16(v + 4 * FR_SLAB + 16 * i, op.ln_b + 4 * i);
        if (two) { fr_cp16(v + 8 * FR_SLAB + 16 * i, op.ln0_w + 4 * i); fr_cp16(v + 12 * FR_SLAB + 16 * i, op.ln0_b + 4 * i); }
    }
}

// ------------------------------------------------------------------------------------------------------ weights
// NB: eight-row halves of a row tile. Units whose sums a CTA holds at a time:
__host__ __device__ constexpr int fr_gu(int NB) { return 8 / NB; }

// A warp's way through the weights of a contraction: its 64 wide parts of this CTA's units, in groups of fr_gu units, in a group
// slab by slab, unit by unit. The next FR_AHEAD of them are on their way into a ring of the warp's own, the first ones since
// before the grid barrier: what comes from HBM travels while the chain waits for its latencies. One commit group per piece,
// empty ones behind the last. (A producer warp with bulk copies costs every warp a wait and an arrival per unit, 350 of 800
// cycles; in registers the pieces leave the LayerNorms too few.)
struct FrFeed {
    const uint8_t *base;                  // of slab 0 of the CTA's first unit, at the warp's part
    uint32_t ustep, sstep;                // bytes to the CTA's next unit, to the next slab
    int mine, slabs, first, sl, u;        // units and slabs; the next piece to ask for
    int slot;                             // where it goes: the place of the piece that is used next
};
template <int NB>
__device__ __forceinline__ void fr_ask(FrFeed &f, const FrPlace &c) {
    if (f.first < f.mine) {
        const uint8_t *p = f.base + (size_t)(f.first + f.u) * f.ustep + f.sl * f.sstep + c.lane * 16;
        const uint32_t to = smem_u32(FrShared::ring(c.warp, f.slot)) + c.lane * 16;
        fr_cp16(to, p);
        if (c.lane < 2) fr_cp16(to + 512, p + 512);
        if (++f.u >= fr_gu(NB) || f.first + f.u >= f.mine) {
            f.u = 0;
            if (++f.sl >= f.slabs) { f.sl = 0; f.first += fr_gu(NB); }
        }
    }
    fr_cp_commit();
    f.slot = f.slot + 1 == FR_AHEAD ? 0 : f.slot + 1;
}
template <int NB>
__device__ __forceinline__ void fr_open(const FrArgs &a, const FrOp &op, const FrPlace &c, FrFeed &f) {
    f.mine = f.first = f.sl = f.u = f.slot = 0;
    if (op.type != FR_GEMM) return;
    const int units = (op.N + 7) >> 3, ks = op.K < FR_SLAB ? op.K : FR_SLAB;
    f.slabs = op.K <= FR_SLAB ? 1 : op.K / FR_SLAB;
    f.sstep = (ks >> 6) * FR_PAIR_BYTES;
    f.ustep = a.ngroups * f.slabs * f.sstep;
    f.base = op.w + (size_t)c.ng * f.slabs * f.sstep + c.warp * FR_PAIR_BYTES;
    if (c.warp < (ks >> 6) && units > c.ng) f.mine = (units - c.ng + a.ngroups - 1) / a.ngroups;
#pragma unroll 1
    for (int i = 0; i < FR_AHEAD; i++) fr_ask<NB>(f, c);
}

// All CTAs of this row tile have come `target / ngroups` times (a row tile's chain never looks at another tile's rows).
// Meanwhile the next operation's LayerNorm vectors and first weights are asked for. False: a wait ran out here or elsewhere.
// (A word per CTA that one warp of every CTA watches, instead of one counter: 2.5 k cycles become 6 k, all read the same lines.)
template <int NB>
__device__ __forceinline__ bool fr_tile_sync(const FrArgs &a, const FrPlace &c, const FrOp &next, FrFeed &f, unsigned target) {
    fr_sync();
    unsigned *count = a.bar + 32 * (1 + c.mt);
    // the block barrier before and the release make the CTA's writes visible with the arrival, the acquire and the block
    // barrier behind it those of the others to all warps
    if (c.tid == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    fr_open<NB>(a, next, c, f);
    if (c.warp == 0) {
        if (c.lane == 0) {
            const long long t0 = clock64();
            unsigned v;
            for (int tries = 1;; tries++) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                if (v >= target) break;
                if (tries & 63) continue;
                if (*reinterpret_cast<volatile unsigned *>(a.bar) || clock64() - t0 > (1ll << 31)) {
                    atomicExch(a.bar, 1u);
                    atomicCAS(a.status, ST_OK, ST_TIMEOUT_EPILOGUE);
                    *FrShared::stop() = 1;
                    break;
                }
            }
        }
    } else {
        fr_ask_vectors(next, c.tid - 32, FR_THREADS - 32);
        fr_cp_commit();
    }
    fr_sync();
    return *FrShared::stop() == 0;
}

// --------------------------------------------------------------------------------------------------- LayerNorms
// LayerNorm of a row of at most 1024 by 8 / NC warps: warp `sub` of them holds the 128-wide chunks sub, sub + 8 / NC, .., a lane
// four columns of each. Sums in double of the differences from the row's first value x0 (ln_stats, ln_row.cuh: a large mean
// costs nothing), each lane over the chunks in order (the row's warps exchange them), then a butterfly: a row's bits do not
// depend on how many rows share the CTA. All warps call it. x0 becomes the first value of the result. (The subtraction takes
// 0.6 % of a step of one stream, 0.4 % of eight sentences: 143 and 14 LayerNorms one behind the other in a step or a position.)
template <int NC>
__device__ __forceinline__ void fr_ln(float4 (&v)[NC], float &x0, const float4 *w, const float4 *b, int n4, double rk, int row, int sub, int lane) {
    constexpr int WPR = 8 / NC;
    const double s = x0;
    double t = 0.0, q = 0.0;
    double2 *part = reinterpret_cast<double2 *>(FrShared::red()) + row * 8 * 32 + lane;
#pragma unroll
    for (int i = 0; i < NC; i++) {
        double x = v[i].x - s, y = v[i].y - s, z = v[i].z - s, u = v[i].w - s;
        if (lane + 32 * (sub + WPR * i) >= n4) x = y = z = u = 0.0;
        const double ct = (x + y) + (z + u), cq = fma(x, x, y * y) + fma(z, z, u * u);
        if (WPR > 1) part[(sub + WPR * i) * 32] = make_double2(ct, cq);
        else { t += ct; q += cq; }
    }
    if (WPR > 1) {
        fr_sync();
#pragma unroll
        for (int j = 0; j < 8; j++) { const double2 e = part[j * 32]; t += e.x; q += e.y; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { t += __shfl_xor_sync(0xffffffffu, t, o); q += __shfl_xor_sync(0xffffffffu, q, o); }
    // 1 / sqrt: the single precision value and one Newton step in double
    const double m = t * rk, ve = fma(-t, m, q) * rk + 1e-5, y = (double)rsqrtf((float)ve);
    const float mu = (float)(s + m), inv = (float)(y * fma(-0.5 * ve * y, y, 1.5));
    x0 = ((x0 - mu) * inv) * w[0].x + b[0].x;
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const int at = lane + 32 * (sub + WPR * i);
        if (at >= n4) continue;
        const float4 ww = w[at], bb = b[at];
        v[i] = make_float4(((v[i].x - mu) * inv) * ww.x + bb.x, ((v[i].y - mu) * inv) * ww.y + bb.y,
                           ((v[i].z - mu) * inv) * ww.z + bb.z, ((v[i].w - mu) * inv) * ww.w + bb.w);
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
        if (fin) st[2 * B + b] = 1;
    }
    return cur;
}

// The rows of the tile through the contraction's LayerNorms into X, 8 / NC warps to a row; every unit group for itself. Group 0 keeps
// LN2's rows and an AED row's books.
template <bool AED, int NC>
__device__ __forceinline__ void fr_rows(const FrArgs &a, const FrOp &op, const FrPlace &c, int p) {
    const int K = op.K, n4 = K >> 2, r = c.warp / (8 / NC), sub = c.warp % (8 / NC), m = c.row0 + r;
    const bool on = r < c.rows;
    const float4 *vec = reinterpret_cast<const float4 *>(fr_vectors());
    float4 v[NC];
    float x0 = 0.f;
    if (on) {
        const float *x = op.x + (size_t)m * K, *pe = nullptr;
        if (AED && op.rows == FR_ROWS_AED_NEXT) {
            x = a.emb + (size_t)fr_aed_turn(a, c.lane, m, p, c.ng == 0 && sub == 0) * K;
            pe = a.pos + (size_t)(p < a.max_seq ? p : a.max_seq - 1) * K;
        }
        x0 = __ldcg(x);
#pragma unroll
        for (int i = 0; i < NC; i++) {
            const int at = c.lane + 32 * (sub + 8 / NC * i);
            v[i] = at < n4 ? __ldcg(reinterpret_cast<const float4 *>(x) + at) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (AED && pe) {
            x0 += __ldg(pe);
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const int at = c.lane + 32 * (sub + 8 / NC * i);
                if (at >= n4) continue;
                const float4 y = __ldg(reinterpret_cast<const float4 *>(pe) + at);
                v[i] = make_float4(v[i].x + y.x, v[i].y + y.y, v[i].z + y.z, v[i].w + y.w);
            }
        }
    }
    fr_cp_wait();
    fr_sync();                                                   // the vectors are everybody's
    if (!on) { for (int i = 0; i < NC; i++) v[i] = make_float4(0.f, 0.f, 0.f, 0.f); }
    if (op.rows == FR_ROWS_LN2 || (AED && op.rows == FR_ROWS_AED_NEXT)) {
        fr_ln(v, x0, vec + 2 * (FR_SLAB / 4), vec + 3 * (FR_SLAB / 4), n4, a.inv_d, r, sub, c.lane);
        if (NC < 8) fr_sync();                                   // the sums have been read
        if (c.ng == 0 && on) {
#pragma unroll
            for (int i = 0; i < NC; i++)
                if (c.lane + 32 * (sub + 8 / NC * i) < n4) reinterpret_cast<float4 *>(op.x_copy + (size_t)m * K)[c.lane + 32 * (sub + 8 / NC * i)] = v[i];
        }
    }
    fr_ln(v, x0, vec, vec + FR_SLAB / 4, n4, a.inv_d, r, sub, c.lane);
    if (!on) return;
    bool fits = true;
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const int at = c.lane + 32 * (sub + 8 / NC * i);
        if (at >= n4) continue;
        if (!AED && op.rows == FR_ROWS_LN_SILU) v[i] = make_float4(silu_f(v[i].x), silu_f(v[i].y), silu_f(v[i].z), silu_f(v[i].w));
        __align__(8) __half h[4], l[4];
        fits &= split_h16(v[i].x, h[0], l[0]); fits &= split_h16(v[i].y, h[1], l[1]);
        fits &= split_h16(v[i].z, h[2], l[2]); fits &= split_h16(v[i].w, h[3], l[3]);
        *reinterpret_cast<uint2 *>(FrShared::x(r, 0) + 4 * at) = *reinterpret_cast<const uint2 *>(h);
        *reinterpret_cast<uint2 *>(FrShared::x(r, 1) + 4 * at) = *reinterpret_cast<const uint2 *>(l);
    }
    if (!fits) atomicCAS(a.status, ST_OK, ST_RANGE);
}

// --------------------------------------------------------------------------------------------------- contraction
// slabs `sl`, .. `sl + n - 1` of the tile's planes to rows `at` on, one behind the other (asynchronous). A warp takes a row.
__device__ __forceinline__ void fr_stage_planes(const FrOp &op, const FrPlace &c, int sl, int n, int ks, int at, int planes) {
    for (int i = c.warp; i < n * c.rows * planes; i += FR_WARPS) {
        const int j = planes == 2 ? i >> 1 : i, k = n == 1 ? 0 : j / c.rows, r = j - k * c.rows;
        const __half *src = (planes == 2 && (i & 1) ? op.a_lo : op.a_hi) + (size_t)(c.row0 + r) * op.K + (size_t)(sl + k) * FR_SLAB;
        const uint32_t dst = smem_u32(FrShared::x(at + j, planes == 2 ? i & 1 : 0));
#pragma unroll
        for (int col = c.lane * 8; col < FR_SLAB; col += 256) if (col < ks) fr_cp16(dst + col * 2, src + col);
    }
    fr_cp_commit();
}

// A thread's output of a group of units: unit slot, row of the tile, column of the unit (columns side by side).
struct FrOut {
    int u, row, col, n;                   // n: column of the contraction
    bool on;
    float bias, res;                      // asked for under the products
};
template <int NB>
__device__ __forceinline__ FrOut fr_out(const FrArgs &a, const FrOp &op, const FrPlace &c, int first, int nu, bool glu) {
    FrOut o;
    o.u = c.tid / (64 * NB); o.row = (c.tid >> 3) & (8 * NB - 1); o.col = c.tid & 7;
    const int unit = c.ng + (first + o.u) * a.ngroups;
    o.n = !glu ? unit * 8 + o.col : o.col < 4 ? unit * 4 + o.col : op.N / 2 + unit * 4 + o.col - 4;
    o.on = o.u < nu && o.row < c.rows && o.n < op.N;
    o.bias = o.on && op.bias ? __ldg(op.bias + o.n) : 0.f;
    o.res = o.on && op.epi == FR_EPI_RESID ? __ldcg(op.res + (size_t)(c.row0 + o.row) * op.ldo + o.n) : 0.f;
    return o;
}
// A warp's sums: per two units and eight rows a block of FR_CT floats, in it (column g of both units, rows 2 t and 2 t + 1) at
// 20 g + 4 t: [unit][row]. Steps of 20 keep the columns of a row in different banks.
__device__ __forceinline__ float *fr_red(int warp, int block) { return FrShared::red() + (warp * 4 + block) * FR_CT; }

// np: warps that have a part of the sums; they are added in warp order
template <bool AED, int NB>
__device__ __forceinline__ void fr_epilogue(const FrArgs &a, const FrOp &op, const FrPlace &c, int first, int nu, int mine, int np, const FrOut &o) {
    float v = 0.f;
    if (o.on) {
        const float *red = fr_red(0, (o.u >> 1) * NB + (o.row >> 3)) + 20 * o.col + ((o.row & 7) >> 1) * 4 + (o.u & 1) * 2 + (o.row & 1);
        if (np == FR_WARPS) {
#pragma unroll
            for (int w = 0; w < FR_WARPS; w++) v += red[w * 4 * FR_CT];
        } else {
            for (int w = 0; w < np; w++) v += red[w * 4 * FR_CT];
        }
        v += o.bias;
    }
    if (op.epi >= FR_EPI_GLU_CONV) {
        FrShared::vals()[c.tid] = v;                             // [unit][row][column]
        fr_sync();
        if (AED) {
            const int row = c.warp;                              // a warp per row
            if (row >= 8 * NB) return;
            float bv = -3.0e38f;
            int bi = 0x7fffffff;
            for (int i = c.lane; i < nu * 8; i += 32) {
                const int n = (c.ng + (first + (i >> 3)) * a.ngroups) * 8 + (i & 7);
                const float x = FrShared::vals()[((i >> 3) * 8 * NB + row) * 8 + (i & 7)];
                if (n < op.N && (x > bv || (x == bv && n < bi))) { bv = x; bi = n; }
            }
#pragma unroll
            for (int q = 16; q > 0; q >>= 1) {
                const float x = __shfl_xor_sync(0xffffffffu, bv, q);
                const int k = __shfl_xor_sync(0xffffffffu, bi, q);
                if (x > bv || (x == bv && k < bi)) { bv = x; bi = k; }
            }
            if (c.lane == 0) {
                if (first == 0 || bv > FrShared::best_v()[row] || (bv == FrShared::best_v()[row] && bi < FrShared::best_i()[row])) { FrShared::best_v()[row] = bv; FrShared::best_i()[row] = bi; }
                if (first + nu >= mine && row < c.rows) {
                    a.cand_v[(size_t)(c.row0 + row) * a.ngroups + c.ng] = FrShared::best_v()[row];
                    a.cand_i[(size_t)(c.row0 + row) * a.ngroups + c.ng] = FrShared::best_i()[row];
                }
            }
            return;
        }
        // GLU rows behind the cached ones of their stream, the depthwise taps, the cache moved on
        const int Q = a.Q, ns = c.rows / Q, k = op.conv_k, d = a.d;
        for (int i = c.tid; i < nu * ns * 4; i += FR_THREADS) {
            const int j = i & 3, sl = (i >> 2) % ns, u = (i >> 2) / ns, ch = (c.ng + (first + u) * a.ngroups) * 4 + j, stream = c.row0 / Q + sl;
            float *cc = op.conv_cache + (size_t)stream * (k - 1) * d + ch;
            const float *val = FrShared::vals() + (u * NB * 8 + sl * Q) * 8 + j, *w = op.dw_w + (size_t)ch * k;
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
    if (!o.on) return;
    const int m = c.row0 + o.row;
    bool fits = true;
    if (op.act == ACT_SILU) v = silu_f(v);
    else if (op.act == ACT_RELU) v = fmaxf(v, 0.0f);
    if (op.epi == FR_EPI_PLANES) {
        __half h, l;
        fits = split_h16(v, h, l);
        op.o_hi[(size_t)m * op.N + o.n] = h;
        op.o_lo[(size_t)m * op.N + o.n] = l;
    } else if (op.epi == FR_EPI_RESID) {
        op.out[(size_t)m * op.ldo + o.n] = o.res + op.alpha * v;
    } else if (op.epi == FR_EPI_QKV && o.n >= op.n_split) {
        const int e = o.n - op.n_split, half_n = (op.N - op.n_split) / 2;
        __half h, l;
        fits = split_h16(v, h, l);
        (e < half_n ? op.o_hi : op.o_lo)[(size_t)m * half_n + (e < half_n ? e : e - half_n)] = h;
    } else {
        op.out[(size_t)m * op.ldo + o.n] = v;
    }
    if (!fits) atomicCAS(a.status, ST_OK, ST_RANGE);
}

// A warp's 64-wide parts of two units (BOTH; else one) and NB times eight rows: acc += ... The weights are the 16-row operand of
// m16n8k16 (unit 0 above unit 1), X the 8-column one, so that up to eight rows cost half of what sixteen do.
template <int TERMS, int NB, bool BOTH>
__device__ __forceinline__ void fr_pair(const uint8_t *p0, const uint8_t *p1, int lane, const uint4 (&xh)[2][NB], const uint4 (&xl)[2][NB], float (&acc)[NB][4]) {
    const uint4 q0 = *reinterpret_cast<const uint4 *>(p0 + lane * 16), q1 = BOTH ? *reinterpret_cast<const uint4 *>(p1 + lane * 16) : make_uint4(0, 0, 0, 0);
    const __half *s0 = reinterpret_cast<const __half *>(p0 + 512) + (lane >> 3) * 4 + ((lane >> 2) & 1), *s1 = reinterpret_cast<const __half *>(p1 + 512) + (lane >> 3) * 4 + ((lane >> 2) & 1);
#pragma unroll
    for (int b = 0; b < 2; b++) {
        uint32_t w[4], v[4] = {0, 0, 0, 0};
        fr_widen(b ? q0.z : q0.x, w[0], w[1]);
        fr_widen(b ? q0.w : q0.y, w[2], w[3]);
        if (BOTH) { fr_widen(b ? q1.z : q1.x, v[0], v[1]); fr_widen(b ? q1.w : q1.y, v[2], v[3]); }
        float ch[NB][4], cl[NB][4];
#pragma unroll
        for (int n = 0; n < NB; n++) {
#pragma unroll
            for (int i = 0; i < 4; i++) ch[n][i] = cl[n][i] = 0.f;
            fr_mma(ch[n], w[0], v[0], w[1], v[1], xh[b][n].x, xh[b][n].y);
            if (TERMS > 1) fr_mma(cl[n], w[0], v[0], w[1], v[1], xl[b][n].x, xl[b][n].y);
        }
#pragma unroll
        for (int n = 0; n < NB; n++) {
            fr_mma(ch[n], w[2], v[2], w[3], v[3], xh[b][n].z, xh[b][n].w);
            if (TERMS > 1) fr_mma(cl[n], w[2], v[2], w[3], v[3], xl[b][n].z, xl[b][n].w);
        }
        const float d0 = __half2float(s0[b * 2]), d1 = BOTH ? __half2float(s1[b * 2]) : 0.f;
#pragma unroll
        for (int n = 0; n < NB; n++)
#pragma unroll
            for (int i = 0; i < (BOTH ? 4 : 2); i++) acc[n][i] = fmaf(i < 2 ? d0 : d1, TERMS > 1 ? fmaf(cl[n][i], H16_LO_INV, ch[n][i]) : ch[n][i], acc[n][i]);
    }
}

// One slab of a group of nu units, two at a time: the rows' fragments stay in registers for all of them; the sums of units wait
// in shared memory for their next slab. The loop is not unrolled: sixteen warps hide the latencies, and what bounds it is the
// instructions issued.
template <int TERMS, int NB>
__device__ __forceinline__ void fr_slab(const FrPlace &c, FrFeed &f, int xrow, int nu, bool more) {
    const int g = c.lane >> 2, t = c.lane & 3;
    uint4 xh[2][NB], xl[2][NB];                                  // [block][rows g, g + 8]
#pragma unroll
    for (int n = 0; n < NB; n++) {
        const int r = xrow + (g + 8 * n < c.rows ? g + 8 * n : 0);       // a row that the tile does not have is the first one again; its sums are never stored
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int at = c.warp * 64 + b * 32 + 8 * t;
            xh[b][n] = *reinterpret_cast<const uint4 *>(FrShared::x(r, 0) + at);
            if (TERMS > 1) xl[b][n] = *reinterpret_cast<const uint4 *>(FrShared::x(r, 1) + at);
        }
    }
    float *sums = fr_red(c.warp, 0) + 20 * g + 4 * t;
#pragma unroll 1
    for (int u = 0; u < nu; u += 2, sums += NB * FR_CT) {
        float acc[NB][4];
#pragma unroll
        for (int n = 0; n < NB; n++) {
            acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
            if (more) { const float4 v = *reinterpret_cast<const float4 *>(sums + n * FR_CT); acc[n][0] = v.x; acc[n][1] = v.y; acc[n][2] = v.z; acc[n][3] = v.w; }
        }
        fr_cp_wait_but<FR_AHEAD - 2>();
        __syncwarp();
        const uint8_t *p0 = FrShared::ring(c.warp, f.slot), *p1 = FrShared::ring(c.warp, f.slot + 1 == FR_AHEAD ? 0 : f.slot + 1);
        const bool both = u + 1 < nu;
        if (both) fr_pair<TERMS, NB, true>(p0, p1, c.lane, xh, xl, acc);
        else fr_pair<TERMS, NB, false>(p0, p0, c.lane, xh, xl, acc);
#pragma unroll
        for (int n = 0; n < NB; n++) *reinterpret_cast<float4 *>(sums + n * FR_CT) = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
        __syncwarp();                                            // all lanes have read the pieces
        fr_ask<NB>(f, c);
        if (both) fr_ask<NB>(f, c);
    }
}

// What the attention behind this contraction will read of the caches and the position keys, on its way to the L2 meanwhile.
__device__ __forceinline__ void fr_stream_prefetch(const FrArgs &a, const FrOp &op, const FrPlace &c) {
    const int tasks = c.rows / a.Q * a.H, K = a.valid + a.Q;
    for (int task = c.ng + c.warp * a.ngroups; task < tasks; task += FR_WARPS * a.ngroups) {
        const size_t base = ((size_t)(c.row0 / a.Q) * a.H + task) * a.left * a.dk;
        const int h = task % a.H, bytes = a.left * a.dk * 2;
        for (int i = c.lane * 128; i < bytes; i += 32 * 128) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t *>(op.kc + base) + i));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t *>(op.vc + base) + i));
        }
        if (c.row0 == 0 && task < a.H)                           // once for all streams
            for (int j = c.lane; j < K; j += 32) {
                const uint8_t *p = reinterpret_cast<const uint8_t *>(op.rk + (size_t)j * op.ldrk + h * a.dk);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(p + a.dk * 2 - 2));
            }
    }
}

// One contraction over this CTA's rows and units.
template <bool AED, int TERMS, int NB>
__device__ __forceinline__ void fr_gemm(const FrArgs &a, const FrOp &op, const FrPlace &c, int p, FrFeed &f) {
    const int units = (op.N + 7) >> 3, mine = units > c.ng ? (units - c.ng + a.ngroups - 1) / a.ngroups : 0;
    const int ks = op.K < FR_SLAB ? op.K : FR_SLAB, slabs = op.K <= FR_SLAB ? 1 : op.K / FR_SLAB, np = ks >> 6, planes = TERMS > 1 ? 2 : 1;
    if (AED && op.epi == FR_EPI_ARGMAX && mine == 0 && c.tid < c.rows) {
        a.cand_v[(size_t)(c.row0 + c.tid) * a.ngroups + c.ng] = -3.0e38f;
        a.cand_i[(size_t)(c.row0 + c.tid) * a.ngroups + c.ng] = 0x7fffffff;
    }
    // few rows: all slabs are asked for at once, and once; else two slabs in turn, again for every group of units
    const bool from_planes = op.rows == FR_ROWS_PLANES, all = !from_planes || c.rows * slabs <= 32;
    if (mine == 0 && (from_planes || c.ng != 0)) return;         // (group 0 keeps rows and books even where no unit is its own)
    if (!from_planes) {                                          // (8 / NC warps to a row)
        if (NB > 1) fr_rows<AED, 8>(a, op, c, p);
        else if (c.rows <= 2) fr_rows<AED, 1>(a, op, c, p);
        else if (c.rows <= 4) fr_rows<AED, 2>(a, op, c, p);
        else fr_rows<AED, 4>(a, op, c, p);
    }
    if (from_planes && all) fr_stage_planes(op, c, 0, slabs, ks, 0, planes);
    if (!AED && op.epi == FR_EPI_QKV) fr_stream_prefetch(a, op, c);
    constexpr int GU = fr_gu(NB);
    for (int first = 0; first < mine; first += GU) {
        const int nu = mine - first < GU ? mine - first : GU;
        if (!all) {
            if (first) fr_sync();
            fr_stage_planes(op, c, 0, 1, ks, 0, planes);
        }
        const FrOut o = fr_out<NB>(a, op, c, first, nu, !AED && op.epi == FR_EPI_GLU_CONV);
        if (all && first == 0) { fr_cp_wait(); fr_sync(); }
        for (int sl = 0; sl < slabs; sl++) {
            if (!all) {
                // (a slab's rows were asked for before the pieces of the slab before it were used: nu groups ago)
                if (sl == 0) fr_cp_wait();
                else if (nu == GU) fr_cp_wait_but<GU>();
                else fr_cp_wait_but<1>();
                fr_sync();
                if (sl + 1 < slabs) fr_stage_planes(op, c, sl + 1, 1, ks, ((sl + 1) & 1) * 16, planes);
            }
            if (c.warp < np) fr_slab<TERMS, NB>(c, f, from_planes ? (all ? sl * c.rows : (sl & 1) * 16) : 0, nu, sl > 0);
        }
        fr_sync();
        fr_epilogue<AED, NB>(a, op, c, first, nu, mine, np, o);
        if (first + GU < mine) fr_sync();                     // the sums are read before the next group writes its own
    }
}

// ---------------------------------------------------------------------------------------------------- attentions
// One query over n keys, in FR_LISTS lists: list w holds the keys w, w + FR_LISTS, ... A warp walks a list in rounds of KB
// keys: all key and value rows of a round are asked for at once (one round covers a list of the usual 71 streaming keys), the
// scores stay in its lanes, the softmax is a running maximum per list. A lane owns four columns; dk is a multiple of 4 up to
// 128. The lists meet in fr_context in a fixed order: the bits are the same whether sixteen warps take one list each or one
// warp takes all.
bool fr_attn_fits(int dk) { return dk % 4 == 0 && dk <= 128; }

struct FrTask {                           // a warp's share of a round of (query group, head) tasks
    int wpt;                              // warps per task
    int slot, sub;                        // task of the round, warp in it
    float *part;                          // [FR_LISTS][128] sums of the task
    float2 *ml;                           // [FR_LISTS] running maximum and sum of weights
};
// as many warps per task as leaves the CTA's tasks one round where they fit into one
__device__ __forceinline__ FrTask fr_task(const FrArgs &a, const FrPlace &c, int tasks) {
    FrTask t;
    const int mine = (tasks + a.ngroups - 1) / a.ngroups;
    t.wpt = mine <= 1 ? 16 : mine <= 2 ? 8 : mine <= 4 ? 4 : mine <= 8 ? 2 : 1;
    t.slot = c.warp / t.wpt; t.sub = c.warp - t.slot * t.wpt;
    t.part = reinterpret_cast<float *>(FrShared::x(0, 0)) + t.slot * FR_LISTS * 128;
    t.ml = reinterpret_cast<float2 *>(FrShared::red()) + t.slot * FR_LISTS;
    return t;
}

// load(j, u) fetches key and value of key j into slot u, score(u) is the lane's part of the dot product, value(u) its columns
template <int KB, typename FL, typename FS, typename FV>
__device__ __forceinline__ void fr_list(const FrTask &k, int list, int n, int dk, int lane, FL load, FS score, FV value) {
    const bool on = lane * 4 < dk;
    float m = -INFINITY, l = 0.f;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j0 = list; j0 < n; j0 += KB * FR_LISTS) {
#pragma unroll
        for (int u = 0; u < KB; u++) load(j0 + FR_LISTS * u < n ? j0 + FR_LISTS * u : j0, u);
        float sc[KB], mx = m;
#pragma unroll
        for (int u = 0; u < KB; u++) sc[u] = on ? score(u) : 0.f;
#pragma unroll
        for (int o2 = 16; o2 > 0; o2 >>= 1)
#pragma unroll
            for (int u = 0; u < KB; u++) sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o2);
#pragma unroll
        for (int u = 0; u < KB; u++) { if (j0 + FR_LISTS * u >= n) sc[u] = -INFINITY; mx = fmaxf(mx, sc[u]); }
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
    if (on) *reinterpret_cast<float4 *>(k.part + list * 128 + lane * 4) = o;
    if (lane == 0) k.ml[list] = make_float2(m, l);
}
// the task's lists into its context row
__device__ __forceinline__ void fr_context(const FrOp &op, const FrTask &k, size_t out, int dk, int lane) {
    const float2 e = k.ml[lane % FR_LISTS];
    float mx = e.x;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float f = expf(e.x - mx);                              // an empty list: exp(-inf) = 0
    float sum = f * e.y;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    for (int i0 = k.sub * 32; i0 < dk; i0 += 32 * k.wpt) {
        const int i = i0 + lane;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < FR_LISTS; w++) v = fmaf(__shfl_sync(0xffffffffu, f, w), k.part[w * 128 + i], v);
        if (i >= dk) continue;
        __half hi, lo;
        split_h16(v / sum, hi, lo);
        op.o_hi[out + i] = hi;
        op.o_lo[out + i] = lo;
    }
}
__device__ __forceinline__ float4 fr_unpack(uint2 a) {
    const float2 x = __half22float2(*reinterpret_cast<const __half2 *>(&a.x)), y = __half22float2(*reinterpret_cast<const __half2 *>(&a.y));
    return make_float4(x.x, x.y, y.x, y.y);
}
__device__ __forceinline__ uint2 fr_ld8(const __half *p) { return __ldcg(reinterpret_cast<const uint2 *>(p)); }
__device__ __forceinline__ float fr_dot(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }

// score(t, j) = ((q_t + u) . k_j + (q_t + v) . rk[K - 1 - valid - t + j]) / sqrt(dk) over [cached frames ; chunk]; afterwards the
// chunk's k / v rows go to their ring slots (update_kv_cache, src/encoder.c:763-776): a (stream, head) is read by its own task alone.
__device__ __forceinline__ void fr_stream_attn(const FrArgs &a, const FrOp &op, const FrPlace &c, int start) {
    constexpr int KB = 5;
    const int H = a.H, dk = a.dk, d = a.d, Q = a.Q, left = a.left, valid = a.valid, K = valid + Q, tasks = c.rows / Q * H;
    const FrTask k = fr_task(a, c, tasks);
    const float scale = 1.0f / sqrtf((float)dk);
    const int i0 = c.lane * 4 < dk ? c.lane * 4 : 0;
    for (int base = c.ng; base < tasks; base += FR_WARPS / k.wpt * a.ngroups) {
        const int task = base + k.slot * a.ngroups, st = c.row0 / Q + task / H, h = task % H;
        const bool on = task < tasks;
        const size_t cbase = ((size_t)st * H + h) * left * dk, nbase = (size_t)st * Q * d + h * dk;
        for (int t = 0; t < Q; t++) {
            const size_t row = (size_t)st * Q + t;
            if (on) {
                const __half *rk = op.rk + (size_t)(K - 1 - valid - t) * op.ldrk + h * dk + i0;
                const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(op.q + row * op.ldq + h * dk + i0));
                const float4 bu = __ldg(reinterpret_cast<const float4 *>(op.bias_u + h * dk + i0)), bv = __ldg(reinterpret_cast<const float4 *>(op.bias_v + h * dk + i0));
                const float4 qu = make_float4(q4.x + bu.x, q4.y + bu.y, q4.z + bu.z, q4.w + bu.w), qv = make_float4(q4.x + bv.x, q4.y + bv.y, q4.z + bv.z, q4.w + bv.w);
                uint2 kk[KB], rr[KB], vv[KB];
                for (int list = k.sub; list < FR_LISTS; list += k.wpt)
                    fr_list<KB>(k, list, K, dk, c.lane,
                                [&](int j, int u) {
                                    int x = start + j;
                                    if (x >= left) x -= left;
                                    const size_t o = j < valid ? cbase + (size_t)x * dk + i0 : nbase + (size_t)(j - valid) * d + i0;
                                    kk[u] = fr_ld8((j < valid ? op.kc : op.kn) + o);
                                    rr[u] = fr_ld8(rk + (size_t)j * op.ldrk);
                                    vv[u] = fr_ld8((j < valid ? op.vc : op.vn) + o);
                                },
                                [&](int u) { return (fr_dot(qu, fr_unpack(kk[u])) + fr_dot(qv, fr_unpack(rr[u]))) * scale; },
                                [&](int u) { return fr_unpack(vv[u]); });
            }
            fr_sync();
            if (on) fr_context(op, k, row * d + h * dk, dk, c.lane);
            if (t + 1 < Q || base + FR_WARPS / k.wpt * a.ngroups < tasks) fr_sync();
        }
        if (on)
            for (int i = k.sub * 32 + c.lane; i < Q * dk; i += 32 * k.wpt) {
                const int t = i / dk, e = i - t * dk;
                int x = start + valid + t;
                while (x >= left) x -= left;
                op.kc[cbase + (size_t)x * dk + e] = __ldcg(op.kn + nbase + (size_t)t * d + e);
                op.vc[cbase + (size_t)x * dk + e] = __ldcg(op.vn + nbase + (size_t)t * d + e);
            }
    }
}

// One query per utterance over its own past (src/decoder_aed.c:186-197), f32 cache [B][max_len][d].
__device__ __forceinline__ void fr_aed_self(const FrArgs &a, const FrOp &op, const FrPlace &c, int p) {
    constexpr int KB = 4;
    const int H = a.H, dk = a.dk, d = a.d, tasks = c.rows * H;
    const FrTask k = fr_task(a, c, tasks);
    const float scale = 1.0f / sqrtf((float)dk);
    const int i0 = c.lane * 4 < dk ? c.lane * 4 : 0;
    for (int base = c.ng; base < tasks; base += FR_WARPS / k.wpt * a.ngroups) {
        const int task = base + k.slot * a.ngroups, b = c.row0 + task / H, h = task % H;
        const bool on = task < tasks;
        const float *row = op.q + (size_t)b * op.ldq + h * dk;
        float *Kc = op.ck + (size_t)b * a.max_len * d + h * dk, *Vc = op.cv + (size_t)b * a.max_len * d + h * dk;
        if (on) {
            const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(row + i0));
            float4 kk[KB], vv[KB];
            for (int list = k.sub; list < FR_LISTS; list += k.wpt)
                fr_list<KB>(k, list, p + 1, dk, c.lane,
                            [&](int j, int u) {                  // this position's row straight from the projection
                                kk[u] = __ldcg(reinterpret_cast<const float4 *>(j < p ? Kc + (size_t)j * d + i0 : row + d + i0));
                                vv[u] = __ldcg(reinterpret_cast<const float4 *>(j < p ? Vc + (size_t)j * d + i0 : row + 2 * d + i0));
                            },
                            [&](int u) { return fr_dot(q4, kk[u]) * scale; }, [&](int u) { return vv[u]; });
        }
        fr_sync();
        if (on) {
            for (int i = k.sub * 32 + c.lane; i < dk; i += 32 * k.wpt) {
                Kc[(size_t)p * d + i] = __ldcg(row + d + i);
                Vc[(size_t)p * d + i] = __ldcg(row + 2 * d + i);
            }
            fr_context(op, k, (size_t)b * d + h * dk, dk, c.lane);
        }
        if (base + FR_WARPS / k.wpt * a.ngroups < tasks) fr_sync();
    }
}

// One query per utterance over its projected encoder frames (src/decoder_aed.c:199-202), (hi, lo) planes by (utterance, head).
__device__ __forceinline__ void fr_aed_cross(const FrArgs &a, const FrOp &op, const FrPlace &c) {
    constexpr int KB = 4;
    const int H = a.H, dk = a.dk, d = a.d, tasks = c.rows * H;
    const FrTask k = fr_task(a, c, tasks);
    const float scale = 1.0f / sqrtf((float)dk);
    const int i0 = c.lane * 4 < dk ? c.lane * 4 : 0;
    for (int base = c.ng; base < tasks; base += FR_WARPS / k.wpt * a.ngroups) {
        const int task = base + k.slot * a.ngroups, b = c.row0 + task / H, h = task % H;
        const bool on = task < tasks;
        if (on) {
            const int T = a.enc_len[b];
            const size_t kb = ((size_t)a.enc_off[b] * H + (size_t)h * T) * dk + i0;
            const __half *khp = op.a_hi + kb, *klp = op.a_lo + kb, *vhp = khp + a.v_off, *vlp = klp + a.v_off;
            const float4 q4 = __ldcg(reinterpret_cast<const float4 *>(op.q + (size_t)b * op.ldq + h * dk + i0));
            uint2 kh[KB], kl[KB], vh[KB], vl[KB];
            auto join = [&](uint2 x, uint2 y) {
                const float4 h4 = fr_unpack(x), l4 = fr_unpack(y);
                return make_float4(fmaf(l4.x, H16_LO_INV, h4.x), fmaf(l4.y, H16_LO_INV, h4.y), fmaf(l4.z, H16_LO_INV, h4.z), fmaf(l4.w, H16_LO_INV, h4.w));
            };
            for (int list = k.sub; list < FR_LISTS; list += k.wpt)
                fr_list<KB>(k, list, T, dk, c.lane,
                            [&](int j, int u) {
                                const int o = j * dk;
                                kh[u] = __ldg(reinterpret_cast<const uint2 *>(khp + o)); kl[u] = __ldg(reinterpret_cast<const uint2 *>(klp + o));
                                vh[u] = __ldg(reinterpret_cast<const uint2 *>(vhp + o)); vl[u] = __ldg(reinterpret_cast<const uint2 *>(vlp + o));
                            },
                            [&](int u) { return fr_dot(q4, join(kh[u], kl[u])) * scale; }, [&](int u) { return join(vh[u], vl[u]); });
        }
        fr_sync();
        if (on) fr_context(op, k, (size_t)b * d + h * dk, dk, c.lane);
        if (base + FR_WARPS / k.wpt * a.ngroups < tasks) fr_sync();
    }
}

template <bool AED, int TERMS, int NB>
__global__ void __launch_bounds__(FR_THREADS, 1)
fr_kernel(const __grid_constant__ FrArgs a) {
    FrPlace c;
    c.tid = threadIdx.x; c.warp = threadIdx.x >> 5; c.lane = threadIdx.x & 31;
    c.ng = blockIdx.x / a.mtiles; c.mt = blockIdx.x % a.mtiles;
    c.row0 = c.mt * a.tile_rows;
    c.rows = a.M - c.row0 < a.tile_rows ? a.M - c.row0 : a.tile_rows;
    if (threadIdx.x == 0) *FrShared::stop() = 0;
    for (int i = threadIdx.x; i < (int)(sizeof(FrOp) / 4); i += FR_THREADS) reinterpret_cast<int *>(&FrShared::op(0))[i] = reinterpret_cast<const int *>(a.ops)[i];
    __syncthreads();
    FrFeed f;
    fr_open<NB>(a, FrShared::op(0), c, f);
    fr_ask_vectors(FrShared::op(0), c.tid, FR_THREADS);
    fr_cp_commit();
    unsigned turn = 0;
    const int rounds = AED ? a.positions + 1 : 1, start = AED ? 0 : *a.d_start;
    bool go = true;
    for (int p = 0; p < rounds && go; p++)
        for (int i = 0; i < a.n_ops && go; i++) {
            const FrOp &op = FrShared::op(turn), &next = FrShared::op(turn + 1);
            // the turn that opened this position marked the rows that are done (all CTAs of the tile read it behind the barrier)
            if (AED && i == 1) {
                bool done = true;
                for (int r = 0; r < c.rows; r++) done &= __ldcg(a.st + 2 * a.B + c.row0 + r) != 0;
                if (done) { go = false; break; }
            }
            {   // the next operation's description arrives meanwhile
                const int nx = i + 1 < a.n_ops ? i + 1 : 0;
                if (c.tid < (int)(sizeof(FrOp) / 16)) fr_cp16(smem_u32(&next) + c.tid * 16, reinterpret_cast<const uint8_t *>(a.ops + nx) + c.tid * 16);
                fr_cp_commit();
            }
            if (op.type == FR_GEMM) fr_gemm<AED, TERMS, NB>(a, op, c, p, f);
            else if (!AED) fr_stream_attn(a, op, c, start);
            else if (op.type == FR_AED_SELF) fr_aed_self(a, op, c, p);
            else fr_aed_cross(a, op, c);
            if (p + 1 == rounds && i + 1 == a.n_ops) break;
            fr_cp_wait();                                        // (the barrier begins with a block barrier)
            turn++;
            go = fr_tile_sync<NB>(a, c, next, f, turn * a.ngroups);
        }
    fr_cp_wait();
}

// ------------------------------------------------------------------------------------------------------ host side
int fr_grid(int M, int tile_rows, int *mtiles, int *ngroups) {
    *mtiles = cdiv(M, tile_rows);
    *ngroups = device_sm_count() / *mtiles;
    return *ngroups >= 1 ? 0 : -1;
}

// The device table of a chain
size_t fr_table_bytes(size_t n_ops) { return n_ops * sizeof(FrOp); }
std::vector<uint8_t> fr_table(const std::vector<FrOp> &ops) {
    const uint8_t *p = reinterpret_cast<const uint8_t *>(ops.data());
    return std::vector<uint8_t>(p, p + fr_table_bytes(ops.size()));
}

int fr_launch(FrArgs a, const std::vector<FrOp> &ops, const void *table, cudaStream_t st) {
    a.ops = static_cast<const FrOp *>(table);
    a.n_ops = (int)ops.size();
    a.inv_d = 1.0 / a.d;
    const int pick = (a.positions > 0) * 4 + (a.terms > 1) * 2 + (a.tile_rows > 8 && a.M > 8);    // eight rows or fewer: one half
    void (*const kernels[8])(FrArgs) = {fr_kernel<false, 1, 1>, fr_kernel<false, 1, 2>, fr_kernel<false, 3, 1>, fr_kernel<false, 3, 2>,
                                        fr_kernel<true, 1, 1>, fr_kernel<true, 1, 2>, fr_kernel<true, 3, 1>, fr_kernel<true, 3, 2>};
    static PerDevice configured = {};
    int dev = 0;
    if (configured.below((size_t)FR_SMEM, &dev)) {
        for (void (*k)(FrArgs) : kernels) MB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, FR_SMEM));
        configured.record(dev, (size_t)FR_SMEM);
    }
    MB_CUDA(cudaMemsetAsync(a.bar, 0, FR_BAR_WORDS * sizeof(unsigned), st));
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(a.mtiles * a.ngroups); lc.blockDim = dim3(FR_THREADS); lc.dynamicSmemBytes = FR_SMEM; lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;                   // the barriers need every CTA on an SM
    at[0].val.cooperative = 1;
    lc.attrs = at; lc.numAttrs = 1;
    MB_CUDA(cudaLaunchKernelEx(&lc, kernels[pick], a));
    note_launch();
    return 0;
}

}  // namespace mb
