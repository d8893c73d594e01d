// Voice activity and offline segment planning with the audio resident on the device.
//
// The reference plans the segments of a long file on the host before anything reaches the encoder: a Silero-style
// network gives one speech probability per 32 ms frame (mynah_asr_vad_feed, src/vad.c:316-385), a hysteresis turns
// the probabilities into padded speech spans (mynah_asr_vad_speech_spans, src/vad.c:417-492), the spans — widened
// and merged — become segments, and anything longer than the model's limit is cut at the 20 ms window of least
// energy (plan_segments_vad, plan_segments, find_split_point, src/mynah_asr.c:1177-1323). Frame by frame on one
// core this serialises in front of the path; here the audio is uploaded once and
//
//   * vad_encode_kernel runs everything of the network that does not depend on the recurrent state for ALL frames
//     at once (one CTA per frame): lookbehind | frame | reflect pad -> STFT as a product with the basis -> magnitude
//     -> the conv + ReLU blocks -> the LSTM's input contribution b_ih + b_hh + W_ih x;
//     (vad_encode16_kernel for the geometry of the published models, vad_encode_kernel for any other);
//   * vad_lstm_kernel walks the frames in order with one cluster of eight CTAs that hold W_hh in registers and exchange
//     the state through distributed shared memory; vad_head_kernel (ReLU -> 1x1 conv -> sigmoid) then gives the
//     probabilities of all frames at once;
//   * window_energy_kernel forms the double-precision sum of squares of every candidate 20 ms window of a search
//     range, one thread per window, in the reference's summation order (so the minimum falls on the same window);
//   * the decisions that are integer / double logic over those numbers — hysteresis, padding, widening, merging,
//     cutting — run on the host exactly as the reference states them.
#include <math.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "../../include/mynah_b200.h"
#include "kernels.h"

using namespace mb;

namespace {

constexpr int VAD_MAX_ENC = 8;

struct VadDev {
    int frame, context, pad, n_fft, hop, n_bins, stft_frames, hidden, n_enc;
    int cin[VAD_MAX_ENC], cout[VAD_MAX_ENC], k[VAD_MAX_ENC], stride[VAD_MAX_ENC], pl[VAD_MAX_ENC], pr[VAD_MAX_ENC];
    const float *basis, *enc_w[VAD_MAX_ENC], *enc_b[VAD_MAX_ENC], *w_ih, *w_hh, *b_ih, *b_hh, *head_w;
    float head_b;
    int act_max;                       // floats of the larger activation buffer
    // the published geometry: weights with the output row fastest (vad_encode16_kernel), else null
    const float *basis_t, *basis_ny, *enc_t[4], *w_ih_t;
};

__device__ __forceinline__ int conv_len(int t_in, int k, int stride, int pl, int pr) { return (t_in + pl + pr - k) / stride + 1; }

// One CTA per frame. Shared memory: buf [context + frame + pad] | spec [2 n_bins stft_frames] | act0 | act1.
__global__ void __launch_bounds__(256)
vad_encode_kernel(const VadDev v, const float *__restrict__ audio, long long n_samples, int frame0, float *__restrict__ xz) {
    extern __shared__ float sm[];
    const int C = v.context, F = v.frame, P = v.pad, N = C + F, T0 = v.stft_frames, B = v.n_bins;
    float *buf = sm, *spec = buf + N + P, *act0 = spec + 2 * B * T0, *act1 = act0 + v.act_max;
    const long long f = blockIdx.x, base = (frame0 + f) * F;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const long long s = base - C + i;        // the lookbehind is the tail of the previous frame (zeros before the signal)
        buf[i] = (s >= 0 && s < n_samples) ? audio[s] : 0.0f;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < P; j += blockDim.x) buf[N + j] = buf[N - 2 - j];       // reflect pad on the right
    __syncthreads();
    // STFT as windows x basis (vad.c:330-336), then the magnitude
    for (int o = threadIdx.x; o < 2 * B * T0; o += blockDim.x) {
        const int r = o / T0, t = o % T0;
        const float *br = v.basis + (size_t)r * v.n_fft, *w = buf + t * v.hop;
        float acc = 0.0f;
        for (int k = 0; k < v.n_fft; k++) acc = fmaf(br[k], w[k], acc);
        spec[o] = acc;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < B * T0; o += blockDim.x) {
        const float re = spec[o], im = spec[o + B * T0];
        act0[o] = sqrtf(re * re + im * im);
    }
    __syncthreads();
    float *in = act0, *out = act1;
    int t_in = T0;
    for (int l = 0; l < v.n_enc; l++) {
        const int t_out = conv_len(t_in, v.k[l], v.stride[l], v.pl[l], v.pr[l]), ck = v.cin[l] * v.k[l];
        for (int o = threadIdx.x; o < v.cout[l] * t_out; o += blockDim.x) {
            const int co = o / t_out, t = o % t_out;
            const float *w = v.enc_w[l] + (size_t)co * ck;
            float acc = 0.0f;
            for (int ci = 0; ci < v.cin[l]; ci++)
                for (int kk = 0; kk < v.k[l]; kk++) {
                    const int s = t * v.stride[l] - v.pl[l] + kk;
                    if (s >= 0 && s < t_in) acc = fmaf(w[ci * v.k[l] + kk], in[ci * t_in + s], acc);
                }
            const float x = acc + v.enc_b[l][co];
            out[o] = x > 0.0f ? x : 0.0f;
        }
        __syncthreads();
        float *sw = in; in = out; out = sw;
        t_in = t_out;
    }
    // the LSTM's input contribution for this frame: b_ih + b_hh + W_ih x (vad.c:357-359)
    const int H = v.hidden;
    for (int r = threadIdx.x; r < 4 * H; r += blockDim.x) {
        const float *w = v.w_ih + (size_t)r * H;
        float acc = 0.0f;
        for (int j = 0; j < H; j++) acc = fmaf(w[j], in[j], acc);
        xz[(size_t)f * 4 * H + r] = (v.b_ih[r] + v.b_hh[r]) + acc;
    }
}

// The same for the published geometry (512-sample frames behind 64 samples of context, 256-point windows every 128
// samples, four blocks of three taps with strides 1 2 2 1 and 128 64 64 128 channels), sixteen frames per CTA.
// One frame per CTA reads every weight (0.9 MB) once per frame, one scalar at a time: 7.9 ms for five minutes of audio.
// Here a lane owns output rows and a warp two frames: weights come in whole lines, with the output row fastest, and feed
// all columns of the warp from a register; inputs are 16-byte broadcasts. Bound by the f32 FMA rate: 1.3 ms in pieces of
// 64 CTAs under the recurrence, 0.17 at full rate. Every sum runs in the order of vad_encode_kernel, so the bits are the same.
constexpr int VE_F = 16, VE_N = 576, VE_BUF = VE_N + 64 + 4, VE_THREADS = 256;
constexpr int VE_MAG = 129 * 4 + 4;            // floats of one frame's magnitudes [bin][window], padded
constexpr int VE_C0 = 128 * 4 + 4, VE_C1 = 64 * 2 + 4, VE_C2 = 64 + 4, VE_C3 = 128 + 4;
constexpr int VE_SMEM = VE_F * (VE_BUF + VE_MAG + VE_C0) * 4;

__global__ void __launch_bounds__(VE_THREADS, 2)
vad_encode16_kernel(const VadDev v, const float *__restrict__ audio, long long n_samples, int frame0, int frames, float *__restrict__ xz) {
    extern __shared__ __align__(16) float sm[];
    float *buf = sm, *mag = buf + VE_F * VE_BUF, *c0 = mag + VE_F * VE_MAG, *c1 = buf, *c2 = c1 + VE_F * VE_C1, *c3 = c2 + VE_F * VE_C2;
    const int f0 = frame0 + blockIdx.x * VE_F, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < VE_F * VE_N; i += VE_THREADS) {
        const int f = i / VE_N, j = i % VE_N;
        const long long s = (long long)(f0 + f) * 512 - 64 + j;
        buf[f * VE_BUF + j] = (s >= 0 && s < n_samples) ? audio[s] : 0.0f;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < VE_F * 64; i += VE_THREADS) {
        const int f = i / 64, j = i % 64;
        buf[f * VE_BUF + VE_N + j] = buf[f * VE_BUF + VE_N - 2 - j];
    }
    __syncthreads();
    const int fa = 2 * warp;                                    // this warp's frames: fa, fa + 1
    {   // bins 0..127: re and im rows of four bins per lane, eight windows
        float re[4][8], im[4][8];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int c = 0; c < 8; c++) re[i][c] = im[i][c] = 0.0f;
        const float *w = v.basis_t + lane;
#pragma unroll 1
        for (int k = 0; k < 256; k += 4) {
            float4 x[8];
#pragma unroll
            for (int c = 0; c < 8; c++) x[c] = *reinterpret_cast<const float4 *>(buf + (fa + (c >> 2)) * VE_BUF + (c & 3) * 128 + k);
#pragma unroll
            for (int kk = 0; kk < 4; kk++) {
                float wr[4], wi[4];
#pragma unroll
                for (int i = 0; i < 4; i++) { wr[i] = __ldg(w + (k + kk) * 256 + 32 * i); wi[i] = __ldg(w + (k + kk) * 256 + 128 + 32 * i); }
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const float xv = kk == 0 ? x[c].x : kk == 1 ? x[c].y : kk == 2 ? x[c].z : x[c].w;
#pragma unroll
                    for (int i = 0; i < 4; i++) { re[i][c] = fmaf(wr[i], xv, re[i][c]); im[i][c] = fmaf(wi[i], xv, im[i][c]); }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float m[4];
#pragma unroll
                for (int t = 0; t < 4; t++) m[t] = sqrtf(re[i][4 * h + t] * re[i][4 * h + t] + im[i][4 * h + t] * im[i][4 * h + t]);
                *reinterpret_cast<float4 *>(mag + (fa + h) * VE_MAG + (lane + 32 * i) * 4) = make_float4(m[0], m[1], m[2], m[3]);
            }
        // bin 128: a lane per window of this warp
        if (lane < 8) {
            const float *x = buf + (fa + (lane >> 2)) * VE_BUF + (lane & 3) * 128;
            float r = 0.0f, q = 0.0f;
            for (int k = 0; k < 256; k++) { r = fmaf(__ldg(v.basis_ny + k), x[k], r); q = fmaf(__ldg(v.basis_ny + 256 + k), x[k], q); }
            mag[(fa + (lane >> 2)) * VE_MAG + 128 * 4 + (lane & 3)] = sqrtf(r * r + q * q);
        }
    }
    __syncwarp();                                               // from here on a warp reads only what it wrote itself
    {   // block 0: 129 -> 128 channels, four steps, taps t-1, t, t+1
        float acc[4][8];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int c = 0; c < 8; c++) acc[i][c] = 0.0f;
        const float *w = v.enc_t[0] + lane;
#pragma unroll 1
        for (int ci = 0; ci < 129; ci++) {
            float x[2][4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float4 q = *reinterpret_cast<const float4 *>(mag + (fa + h) * VE_MAG + ci * 4);
                x[h][0] = q.x; x[h][1] = q.y; x[h][2] = q.z; x[h][3] = q.w;
            }
#pragma unroll
            for (int kk = 0; kk < 3; kk++) {
                float wv[4];
#pragma unroll
                for (int i = 0; i < 4; i++) wv[i] = __ldg(w + (ci * 3 + kk) * 128 + 32 * i);
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    const int s = (c & 3) - 1 + kk;
                    if (s < 0 || s > 3) continue;
#pragma unroll
                    for (int i = 0; i < 4; i++) acc[i][c] = fmaf(wv[i], x[c >> 2][s], acc[i][c]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float b = v.enc_b[0][lane + 32 * i];
#pragma unroll
            for (int h = 0; h < 2; h++)
                *reinterpret_cast<float4 *>(c0 + (fa + h) * VE_C0 + (lane + 32 * i) * 4) =
                    make_float4(fmaxf(acc[i][4 * h] + b, 0.0f), fmaxf(acc[i][4 * h + 1] + b, 0.0f), fmaxf(acc[i][4 * h + 2] + b, 0.0f), fmaxf(acc[i][4 * h + 3] + b, 0.0f));
        }
    }
    __syncthreads();                                            // c1..c3 lie over the samples
    {   // block 1: 128 -> 64, steps 0 and 1 at 2 t - 1 + kk
        float acc[2][2][2];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) acc[i][h][0] = acc[i][h][1] = 0.0f;
        const float *w = v.enc_t[1] + lane;
#pragma unroll 2
        for (int ci = 0; ci < 128; ci++) {
            float x[2][4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float4 q = *reinterpret_cast<const float4 *>(c0 + (fa + h) * VE_C0 + ci * 4);
                x[h][0] = q.x; x[h][1] = q.y; x[h][2] = q.z; x[h][3] = q.w;
            }
#pragma unroll
            for (int kk = 0; kk < 3; kk++) {
                const float w0 = __ldg(w + (ci * 3 + kk) * 64), w1 = __ldg(w + (ci * 3 + kk) * 64 + 32);
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    const int s = 2 * t - 1 + kk;
                    if (s < 0) continue;
#pragma unroll
                    for (int h = 0; h < 2; h++) { acc[0][h][t] = fmaf(w0, x[h][s], acc[0][h][t]); acc[1][h][t] = fmaf(w1, x[h][s], acc[1][h][t]); }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float b = v.enc_b[1][lane + 32 * i];
#pragma unroll
            for (int h = 0; h < 2; h++)
                *reinterpret_cast<float2 *>(c1 + (fa + h) * VE_C1 + (lane + 32 * i) * 2) = make_float2(fmaxf(acc[i][h][0] + b, 0.0f), fmaxf(acc[i][h][1] + b, 0.0f));
        }
    }
    __syncwarp();
    {   // block 2: 64 -> 64, one step: taps 1 and 2 fall on steps 0 and 1
        float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        const float *w = v.enc_t[2] + lane;
#pragma unroll 4
        for (int ci = 0; ci < 64; ci++) {
            const float2 xa = *reinterpret_cast<const float2 *>(c1 + fa * VE_C1 + ci * 2), xb = *reinterpret_cast<const float2 *>(c1 + (fa + 1) * VE_C1 + ci * 2);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float w1 = __ldg(w + (ci * 3 + 1) * 64 + 32 * i), w2 = __ldg(w + (ci * 3 + 2) * 64 + 32 * i);
                acc[i][0] = fmaf(w2, xa.y, fmaf(w1, xa.x, acc[i][0]));
                acc[i][1] = fmaf(w2, xb.y, fmaf(w1, xb.x, acc[i][1]));
            }
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float b = v.enc_b[2][lane + 32 * i];
            c2[fa * VE_C2 + lane + 32 * i] = fmaxf(acc[i][0] + b, 0.0f);
            c2[(fa + 1) * VE_C2 + lane + 32 * i] = fmaxf(acc[i][1] + b, 0.0f);
        }
    }
    __syncwarp();
    {   // block 3: 64 -> 128, one step, the middle tap
        float acc[4][2];
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i][0] = acc[i][1] = 0.0f;
        const float *w = v.enc_t[3] + lane;
#pragma unroll 4
        for (int ci = 0; ci < 64; ci++) {
            const float xa = c2[fa * VE_C2 + ci], xb = c2[(fa + 1) * VE_C2 + ci];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float wv = __ldg(w + (ci * 3 + 1) * 128 + 32 * i);
                acc[i][0] = fmaf(wv, xa, acc[i][0]);
                acc[i][1] = fmaf(wv, xb, acc[i][1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float b = v.enc_b[3][lane + 32 * i];
            c3[fa * VE_C3 + lane + 32 * i] = fmaxf(acc[i][0] + b, 0.0f);
            c3[(fa + 1) * VE_C3 + lane + 32 * i] = fmaxf(acc[i][1] + b, 0.0f);
        }
    }
    __syncthreads();
    {   // the LSTM's input contribution: a warp takes 64 of the 512 rows for all sixteen frames
        float acc[2][VE_F];
#pragma unroll
        for (int f = 0; f < VE_F; f++) acc[0][f] = acc[1][f] = 0.0f;
        const int r = warp * 64 + lane;
        const float *w = v.w_ih_t + r;
#pragma unroll 1
        for (int j = 0; j < 128; j += 4) {
            float wv[4][2];
#pragma unroll
            for (int q = 0; q < 4; q++) { wv[q][0] = __ldg(w + (j + q) * 512); wv[q][1] = __ldg(w + (j + q) * 512 + 32); }
#pragma unroll
            for (int f = 0; f < VE_F; f++) {
                const float4 x = *reinterpret_cast<const float4 *>(c3 + f * VE_C3 + j);
#pragma unroll
                for (int i = 0; i < 2; i++) acc[i][f] = fmaf(wv[3][i], x.w, fmaf(wv[2][i], x.z, fmaf(wv[1][i], x.y, fmaf(wv[0][i], x.x, acc[i][f]))));
            }
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float b = v.b_ih[r + 32 * i] + v.b_hh[r + 32 * i];
#pragma unroll
            for (int f = 0; f < VE_F; f++) if (f0 + f < frames) xz[(size_t)(f0 + f - frame0) * 512 + r + 32 * i] = b + acc[i][f];
        }
    }
}

__device__ __forceinline__ float vad_sigmoid(float x) {       // mynah_asr_sigmoid (src/qmat.h:31-35)
    if (x >= 0.0f) return 1.0f / (1.0f + expf(-x));
    const float e = expf(x);
    return e / (1.0f + e);
}

// sigmoid(x) or tanh(x) without a branch: one exponential, one reciprocal. tanh is (1 - e) / (1 + e) with e = exp(-2 |x|), and
// below 0.55, where 1 - e cancels, the fifth convergent of its continued fraction (relative error 3e-9 there).
__device__ __forceinline__ float vl_gate(float x, bool is_tanh) {
    const float ax = fabsf(x), e = expf(is_tanh ? -2.0f * ax : -ax), x2 = x * x;
    const bool small = is_tanh && ax < 0.55f;
    float num = is_tanh ? copysignf(1.0f - e, x) : x >= 0.0f ? 1.0f : e;
    num = small ? x * fmaf(x2, x2 + 105.0f, 945.0f) : num;
    const float den = small ? fmaf(x2, fmaf(x2, 15.0f, 420.0f), 945.0f) : 1.0f + e;
    return num * __frcp_rn(den);
}

// The recurrence, frames [f0, f1): z = xz[f] + W_hh h, gates i f g o. A step is a chain of latencies, so everything is
// laid out to shorten it (0.49 us a frame, 950 cycles: 270 of waiting for the last frame's values, 269 of product and exchange,
// 411 of gates and sending; 2.55 us with one CTA that read h and part of W_hh from shared memory, waited at three
// block barriers and had one thread add up the head's 128 terms):
//   * a cluster of eight CTAs, sixteen hidden units each; eight lanes share a unit, a lane holds 16 columns of the
//     unit's four gate rows in registers (64 weights) and reads its 16 values of h in four 16-byte loads;
//   * the four sums are reduced by a halving exchange that leaves each lane pair with one gate, the pairs apply their
//     non-linearities side by side, four shuffles bring the gates together, and all eight lanes of a unit go on with
//     the same c and h: no barrier between the product and the new state;
//   * lane k sends the unit's h to CTA k (st.async), whose mbarrier completes when all 128 values of the frame have
//     arrived (readers that poll (value, frame number) pairs instead need 0.56 us a frame, against 0.49). Two h buffers suffice: frame f + 2 is sent only after every value of f + 1 has come, that is after every
//     warp of the cluster has read f.
// Waits are bounded; one that runs out sets the status word and the cluster unwinds together.
constexpr int VL_CTAS = 8, VL_THREADS = 128, VL_H = 128;

__device__ __forceinline__ void vl_send(uint32_t addr, float value, uint32_t bar, int cta) {
    asm volatile(
        "{\n\t.reg .b32 ra, rb;\n\t"
        "mapa.shared::cluster.u32 ra, %0, %3;\n\t"
        "mapa.shared::cluster.u32 rb, %2, %3;\n\t"
        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [ra], %1, [rb];\n\t}"
        ::"r"(addr), "r"(__float_as_uint(value)), "r"(bar), "r"(cta)
        : "memory");
}
__device__ __forceinline__ void vl_cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(VL_CTAS, 1, 1) __launch_bounds__(VL_THREADS, 1)
vad_lstm_kernel(const VadDev v, const float *__restrict__ xz, int f0, int f1, float *__restrict__ hist, float *__restrict__ c_state, int *status) {
    __shared__ __align__(16) float h[2][VL_H + 8 * 4];            // eight slices of 16, four floats apart: no bank conflicts
    __shared__ uint64_t bar[2];
    const int lane = threadIdx.x & 31, part = lane & 7, u = blockIdx.x * 16 + (threadIdx.x >> 3);
    float w[4][16];
#pragma unroll
    for (int g = 0; g < 4; g++)
#pragma unroll
        for (int j = 0; j < 16; j++) w[g][j] = v.w_hh[(size_t)(g * VL_H + u) * VL_H + part * 16 + j];
    for (int i = threadIdx.x; i < VL_H; i += VL_THREADS) h[(f0 & 1) ^ 1][(i >> 4) * 20 + (i & 15)] = f0 ? hist[(size_t)(f0 - 1) * VL_H + i] : 0.0f;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; b++) { mbar_init(&bar[b], 1); }
        mbar_fence_init();
        for (int b = 0; b < 2; b++) mbar_expect_tx(&bar[b], VL_H * 4);
    }
    float c = f0 ? c_state[u] : 0.0f;
    __syncthreads();
    vl_cluster_sync();
    const int gate = ((part >> 2) & 1) * 2 + ((part >> 1) & 1);   // 0 i, 1 f, 2 g, 3 o
    const float *xp = xz + (size_t)gate * VL_H + u;       // xz: rows of frames f0, f0 + 1, ..
    const uint32_t dst = smem_u32(&h[0][(u >> 4) * 20 + (u & 15)]), dbar = smem_u32(&bar[0]);
    constexpr int AHEAD = 4;                                      // input contributions asked for this many frames early
    float xq[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; i++) xq[i] = f0 + i < f1 ? xp[(size_t)i * 4 * VL_H] : 0.0f;
    bool ok = true;
    for (int fb = f0; fb < f1 && ok; fb += AHEAD) {
#pragma unroll
        for (int q = 0; q < AHEAD; q++) {
            const int f = fb + q;
            if (f >= f1 || !ok) break;
            const int n = f - f0, buf = (f & 1) ^ 1;              // h of frame f - 1
            if (n > 0) {
                // the buffer's barrier: its k-th completion is the k-th frame of that parity
                ok = __all_sync(0xffffffffu, mbar_wait(&bar[buf], (uint32_t)(((n - 1) >> 1) & 1)));
                if (!ok) break;
                if (threadIdx.x == 0) mbar_expect_tx(&bar[buf], VL_H * 4);
            }
            const float x0 = xq[q];
            if (f + AHEAD < f1) xq[q] = xp[(size_t)(n + AHEAD) * 4 * VL_H];
            float s[4][2];
#pragma unroll
            for (int g = 0; g < 4; g++) s[g][0] = s[g][1] = 0.0f;
            const float4 *hp = reinterpret_cast<const float4 *>(&h[buf][part * 20]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 hv = hp[j];
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    s[g][0] = fmaf(w[g][4 * j], hv.x, s[g][0]); s[g][1] = fmaf(w[g][4 * j + 1], hv.y, s[g][1]);
                    s[g][0] = fmaf(w[g][4 * j + 2], hv.z, s[g][0]); s[g][1] = fmaf(w[g][4 * j + 3], hv.w, s[g][1]);
                }
            }
            // halving exchange: lane bit 2 picks gates {i, f} or {g, o}, bit 1 one of the two, bit 0 adds the last halves
            const float t0 = s[0][0] + s[0][1], t1 = s[1][0] + s[1][1], t2 = s[2][0] + s[2][1], t3 = s[3][0] + s[3][1];
            const bool hi2 = part & 4, hi1 = part & 2;
            float a = (hi2 ? t2 : t0) + __shfl_xor_sync(0xffffffffu, hi2 ? t0 : t2, 4);
            float b = (hi2 ? t3 : t1) + __shfl_xor_sync(0xffffffffu, hi2 ? t1 : t3, 4);
            float z = (hi1 ? b : a) + __shfl_xor_sync(0xffffffffu, hi1 ? a : b, 2);
            z += __shfl_xor_sync(0xffffffffu, z, 1);
            z += x0;
            const float y = vl_gate(z, gate == 2);
            const int base = lane & 24;
            const float ig = __shfl_sync(0xffffffffu, y, base), fg = __shfl_sync(0xffffffffu, y, base + 2), gg = __shfl_sync(0xffffffffu, y, base + 4),
                        og = __shfl_sync(0xffffffffu, y, base + 6);
            c = fg * c + ig * gg;
            const float hn = og * vl_gate(c, true);
            vl_send(dst + (uint32_t)((f & 1) * sizeof(h[0])), hn, dbar + (uint32_t)((f & 1) * 8), part);
            if (part == 0) hist[(size_t)f * VL_H + u] = hn;
        }
    }
    // the last frame's values (and the one before, where a wait ran out) are still on their way into this CTA
    if (ok && f1 > f0) ok = mbar_wait(&bar[(f1 - 1) & 1], (uint32_t)(((f1 - 1 - f0) >> 1) & 1));
    if (!ok && lane == 0) atomicExch(status, ST_TIMEOUT_EPILOGUE);
    if (part == 0) c_state[u] = c;
    __syncthreads();
    vl_cluster_sync();
}

// probability of every frame: head over ReLU(h), a warp per frame
__global__ void __launch_bounds__(256)
vad_head_kernel(const VadDev v, const float *__restrict__ hist, int frames, float *__restrict__ probs) {
    const int f = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (f >= frames) return;
    float a = 0.0f;
#pragma unroll
    for (int j = 0; j < VL_H / 32; j++) a = fmaf(v.head_w[lane + 32 * j], fmaxf(hist[(size_t)f * VL_H + lane + 32 * j], 0.0f), a);
    a = warp_sum(a);
    if (lane == 0) probs[f] = vad_sigmoid(v.head_b + a);
}

// e[j] = sum of squares (double) of the `win` samples from lo + j hop, added in order (find_split_point, src/mynah_asr.c:1183-1189)
__global__ void window_energy_kernel(const float *__restrict__ s, long long lo, int win, int hop, int n_windows, double *__restrict__ e) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_windows) return;
    const float *p = s + lo + (long long)j * hop;
    double acc = 0.0;
    for (int i = 0; i < win; i++) { const double x = p[i]; acc += x * x; }
    e[j] = acc;
}

}  // namespace

namespace {
// A device buffer with its own capacity: one that could not be grown has none, whatever became of the others.
template <typename T>
struct KeptBuffer {
    T *p = nullptr;
    size_t cap = 0;                                                             // in elements
    bool grow(size_t need) {
        if (need <= cap) return true;
        drop();
        if (cudaMalloc((void **)&p, need * sizeof(T)) != cudaSuccess) { cudaGetLastError(); p = nullptr; set_error("device allocation failed"); return false; }
        cap = need;
        return true;
    }
    void drop() { if (p) cudaFree(p); p = nullptr; cap = 0; }
    KeptBuffer() = default;
    KeptBuffer(const KeptBuffer &) = delete;
    KeptBuffer &operator=(const KeptBuffer &) = delete;
    ~KeptBuffer() { drop(); }
};

// Device buffers of one handle (or one call without a handle), kept from call to call and grown when needed. When a call
// ends, audio above KEEP bytes is given back, and so are the LSTM states above a quarter of that (512 bytes per frame of 512
// samples: both lines lie at a signal of 70 minutes) with the probabilities. xz and energy (20 s) have a size of their own.
struct VadBuffers {
    static constexpr size_t KEEP = 256u << 20;
    KeptBuffer<float> audio, xz, hist, probs;                                   // xz: two pieces; hist [frames][128]
    KeptBuffer<double> energy;
    void end_call() {
        if (audio.cap * sizeof(float) > KEEP) audio.drop();
        if (hist.cap * sizeof(float) > KEEP / 4) { hist.drop(); probs.drop(); }
    }
};
}  // namespace

struct mynah_b200_vad {
    mynah_b200_vad_config cfg;
    VadDev d;
    std::vector<void *> owned;
    cudaStream_t stream = nullptr, copy = nullptr;
    cudaEvent_t encoded = nullptr, walked[2] = {nullptr, nullptr};
    size_t smem = 0;
    float *c_state = nullptr;
    int *status = nullptr;
    VadBuffers buf;
    std::mutex mu;                       // calls on one handle share the buffers and run one after the other
};

namespace {

constexpr int VAD_CHUNK = 1024;          // frames per piece of the copy -> encode -> recurrence pipeline; the first is a quarter

float *vad_upload(mynah_b200_vad *v, const float *src, size_t n) {
    float *p = nullptr;
    if (!src || cudaMalloc((void **)&p, n * sizeof(float)) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    v->owned.push_back(p);
    if (cudaMemcpy(p, src, n * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
    return p;
}
// w [rows, cols] with the row index fastest
float *vad_upload_t(mynah_b200_vad *v, const float *w, int rows, int cols) {
    std::vector<float> t((size_t)rows * cols);
    for (int r = 0; r < rows; r++) for (int c = 0; c < cols; c++) t[(size_t)c * rows + r] = w[(size_t)r * cols + c];
    return vad_upload(v, t.data(), t.size());
}

bool vad_published_geometry(const VadDev &d) {
    static const int cout[4] = {128, 64, 64, 128}, stride[4] = {1, 2, 2, 1};
    bool ok = d.frame == 512 && d.context == 64 && d.pad == 64 && d.n_fft == 256 && d.hop == 128 && d.n_bins == 129 && d.n_enc == 4;
    for (int i = 0; i < 4 && ok; i++) ok = d.cout[i] == cout[i] && d.k[i] == 3 && d.stride[i] == stride[i] && d.pl[i] == 1 && d.pr[i] == 1;
    return ok;
}

// Host signal -> v->buf.audio and its speech probabilities. The recurrence sets the pace, so the signal goes up in pieces
// on a second stream, where each piece is encoded too while the one before it is walked.
int vad_run(mynah_b200_vad *v, const float *samples, size_t n, std::vector<float> &probs) {
    const int F = v->d.frame, frames = (int)((n + F - 1) / F);
    VadBuffers &b = v->buf;
    probs.assign((size_t)frames, 0.f);
    if (!b.audio.grow(n ? n : 1)) return -1;
    if (frames == 0) return 0;
    const size_t nxz = (size_t)VAD_CHUNK * 4 * VL_H;
    if (!b.hist.grow((size_t)frames * VL_H) || !b.probs.grow((size_t)frames) || !b.xz.grow(2 * nxz)) return -1;
    cudaError_t e = cudaMemsetAsync(v->status, 0, sizeof(int), v->stream);
    for (int f = 0, i = 0; f < frames && e == cudaSuccess; i++) {
        const int end = f == 0 ? (frames < VAD_CHUNK / 4 ? frames : VAD_CHUNK / 4) : (frames - f < VAD_CHUNK ? frames : f + VAD_CHUNK);
        const size_t s0 = (size_t)f * F, s1 = (size_t)end * F < n ? (size_t)end * F : n;
        float *xz = b.xz.p + (i & 1) * nxz;
        e = cudaMemcpyAsync(b.audio.p + s0, samples + s0, (s1 - s0) * sizeof(float), cudaMemcpyHostToDevice, v->copy);
        if (e == cudaSuccess && i >= 2) e = cudaStreamWaitEvent(v->copy, v->walked[i & 1], 0);
        if (e != cudaSuccess) break;
        // samples past s1 are not on the device yet, and no frame before `end` reads them
        if (v->d.basis_t) vad_encode16_kernel<<<cdiv(end - f, VE_F), VE_THREADS, VE_SMEM, v->copy>>>(v->d, b.audio.p, (long long)s1, f, end, xz);
        else vad_encode_kernel<<<end - f, 256, v->smem, v->copy>>>(v->d, b.audio.p, (long long)s1, f, xz);
        e = cudaEventRecord(v->encoded, v->copy);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(v->stream, v->encoded, 0);
        if (e != cudaSuccess) break;
        vad_lstm_kernel<<<VL_CTAS, VL_THREADS, 0, v->stream>>>(v->d, xz, f, end, b.hist.p, v->c_state, v->status);
        note_launch(2);
        e = cudaEventRecord(v->walked[i & 1], v->stream);
        f = end;
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    int st = 0;
    if (e == cudaSuccess) {
        vad_head_kernel<<<cdiv(frames, 8), 256, 0, v->stream>>>(v->d, b.hist.p, frames, b.probs.p);
        note_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(probs.data(), b.probs.p, (size_t)frames * sizeof(float), cudaMemcpyDeviceToHost, v->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&st, v->status, sizeof(int), cudaMemcpyDeviceToHost, v->stream);
    const cudaError_t es = cudaStreamSynchronize(v->stream);
    cudaStreamSynchronize(v->copy);
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) { set_error("vad: %s", cudaGetErrorString(e)); return -1; }
    if (st) { set_error("vad: a bounded wait inside the recurrence ran out (code %d)", st); return -1; }
    return frames;
}

struct Span { long long t0, t1; };

// mynah_asr_vad_seg_feed / _finish / mynah_asr_vad_pad_spans (src/vad.c:417-474) over a probability vector
std::vector<Span> spans_from_probs(const mynah_b200_vad_config &c, const std::vector<float> &probs, long long n_samples) {
    const double sr = 16000.0;
    auto ms = [&](int v) { return sr * (double)v / 1000.0; };
    std::vector<Span> out;
    bool trig = false;
    long long start = 0, temp_end = -1;
    for (size_t i = 0; i < probs.size(); i++) {
        const long long cur = (long long)c.frame_samples * (long long)i;
        const double p = (double)probs[i];
        if (p >= c.threshold) {
            temp_end = -1;
            if (!trig) { trig = true; start = cur; }
            continue;
        }
        if (p < c.neg_threshold && trig) {
            if (temp_end < 0) temp_end = cur;
            if ((double)(cur - temp_end) < ms(c.min_silence_ms)) continue;
            const long long end = temp_end;
            trig = false; temp_end = -1;
            if ((double)(end - start) > ms(c.min_speech_ms)) out.push_back(Span{start, end});
        }
    }
    if (trig && (double)(n_samples - start) > ms(c.min_speech_ms)) out.push_back(Span{start, n_samples});
    const long long pad = (long long)(sr * (double)c.speech_pad_ms / 1000.0);
    const int n = (int)out.size();
    for (int i = 0; i < n; i++) {
        if (i == 0) out[0].t0 = out[0].t0 - pad > 0 ? out[0].t0 - pad : 0;
        if (i != n - 1) {
            const long long gap = out[i + 1].t0 - out[i].t1;
            if (gap < 2 * pad) {
                out[i].t1 += gap / 2;
                const long long s1 = out[i + 1].t0 - gap / 2;
                out[i + 1].t0 = s1 > 0 ? s1 : 0;
            } else {
                out[i].t1 = out[i].t1 + pad < n_samples ? out[i].t1 + pad : n_samples;
                const long long s1 = out[i + 1].t0 - pad;
                out[i + 1].t0 = s1 > 0 ? s1 : 0;
            }
        } else {
            out[i].t1 = out[i].t1 + pad < n_samples ? out[i].t1 + pad : n_samples;
        }
    }
    return out;
}

// find_split_point (src/mynah_asr.c:1178-1192) on the resident signal: -1 on a device error
long long split_point_dev(VadBuffers &b, long long lo, long long hi, int sr, cudaStream_t st, std::vector<double> &host) {
    const int win = sr / 50, hop = win / 2;
    if (hop <= 0 || lo + win > hi) return hi;
    const int nw = (int)((hi - win - lo) / hop) + 1;
    if (!b.energy.grow((size_t)nw)) return -1;
    window_energy_kernel<<<cdiv(nw, 128), 128, 0, st>>>(b.audio.p, lo, win, hop, nw, b.energy.p);
    note_launch();
    host.resize((size_t)nw);
    cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) err = cudaMemcpyAsync(host.data(), b.energy.p, (size_t)nw * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (err == cudaSuccess) err = cudaStreamSynchronize(st);
    if (err != cudaSuccess) { set_error("plan_segments: %s", cudaGetErrorString(err)); return -1; }
    double best = 1e300;
    long long pos = hi;
    for (int j = 0; j < nw; j++) if (host[(size_t)j] < best) { best = host[(size_t)j]; pos = lo + (long long)j * hop + win / 2; }
    return pos;
}

}  // namespace

extern "C" {

mynah_b200_vad *mynah_b200_vad_new(const mynah_b200_vad_config *c, const float *basis, const float *const *enc_w,
                                   const float *const *enc_b, const float *w_ih, const float *w_hh, const float *b_ih,
                                   const float *b_hh, const float *head_w, float head_b) {
    if (!mynah_b200_available()) { set_error("vad: no sm_100 CUDA device available"); return nullptr; }
    if (!c || !basis || !enc_w || !enc_b || !w_ih || !w_hh || !b_ih || !b_hh || !head_w) { set_error("vad_new: bad argument"); return nullptr; }
    if (c->n_enc < 1 || c->n_enc > VAD_MAX_ENC || c->lstm_hidden != 128 || c->frame_samples <= 0 || c->n_fft <= 0 || c->hop_length <= 0) {
        set_error("vad_new: unsupported geometry (1..%d encoder blocks, LSTM width 128)", VAD_MAX_ENC); return nullptr;
    }
    mynah_b200_vad *v = new mynah_b200_vad();
    v->cfg = *c;
    VadDev &d = v->d;
    memset(&d, 0, sizeof(d));
    d.frame = c->frame_samples; d.context = c->context_samples; d.pad = c->reflect_pad; d.n_fft = c->n_fft; d.hop = c->hop_length;
    d.n_bins = c->n_bins; d.hidden = c->lstm_hidden; d.n_enc = c->n_enc; d.head_b = head_b;
    d.stft_frames = (d.context + d.frame + d.pad - d.n_fft) / d.hop + 1;
    int t = d.stft_frames, cin = d.n_bins, act_max = d.n_bins * d.stft_frames;
    bool ok = d.stft_frames >= 1 && d.pad + 2 <= d.context + d.frame;
    d.basis = vad_upload(v, basis, (size_t)2 * d.n_bins * d.n_fft);
    ok = ok && d.basis;
    for (int i = 0; i < d.n_enc && ok; i++) {
        d.cin[i] = cin; d.cout[i] = c->enc_channels[i]; d.k[i] = c->enc_kernels[i]; d.stride[i] = c->enc_strides[i];
        d.pl[i] = c->enc_pads[2 * i]; d.pr[i] = c->enc_pads[2 * i + 1];
        if (d.cout[i] <= 0 || d.k[i] <= 0 || d.stride[i] <= 0) { ok = false; break; }
        t = (t + d.pl[i] + d.pr[i] - d.k[i]) / d.stride[i] + 1;
        if (t < 1) { ok = false; break; }
        if (d.cout[i] * t > act_max) act_max = d.cout[i] * t;
        d.enc_w[i] = vad_upload(v, enc_w[i], (size_t)d.cout[i] * cin * d.k[i]);
        d.enc_b[i] = vad_upload(v, enc_b[i], (size_t)d.cout[i]);
        ok = d.enc_w[i] && d.enc_b[i];
        cin = d.cout[i];
    }
    // the encoder must collapse to one timestep of the LSTM's width (vad.c:214-239)
    ok = ok && t == 1 && cin == d.hidden;
    const size_t H = (size_t)d.hidden;
    if (ok) {
        d.w_ih = vad_upload(v, w_ih, 4 * H * H); d.w_hh = vad_upload(v, w_hh, 4 * H * H);
        d.b_ih = vad_upload(v, b_ih, 4 * H); d.b_hh = vad_upload(v, b_hh, 4 * H); d.head_w = vad_upload(v, head_w, H);
        ok = d.w_ih && d.w_hh && d.b_ih && d.b_hh && d.head_w;
    }
    d.act_max = act_max;
    v->smem = ((size_t)d.context + d.frame + d.pad + 2 * (size_t)d.n_bins * d.stft_frames + 2 * (size_t)act_max) * sizeof(float);
    if (ok && v->smem > 200 * 1024) ok = false;
    if (ok && vad_published_geometry(d)) {
        std::vector<float> bt((size_t)256 * 256), ny(512);
        for (int k = 0; k < 256; k++) {
            for (int r = 0; r < 128; r++) { bt[(size_t)k * 256 + r] = basis[(size_t)r * 256 + k]; bt[(size_t)k * 256 + 128 + r] = basis[(size_t)(129 + r) * 256 + k]; }
            ny[k] = basis[(size_t)128 * 256 + k]; ny[256 + k] = basis[(size_t)257 * 256 + k];
        }
        d.basis_ny = vad_upload(v, ny.data(), ny.size());
        for (int i = 0; i < 4 && ok; i++) ok = (d.enc_t[i] = vad_upload_t(v, enc_w[i], d.cout[i], d.cin[i] * 3)) != nullptr;
        d.w_ih_t = vad_upload_t(v, w_ih, 512, 128);
        d.basis_t = vad_upload(v, bt.data(), bt.size());
        ok = ok && d.basis_ny && d.w_ih_t && d.basis_t;
        if (ok && cudaFuncSetAttribute(vad_encode16_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, VE_SMEM) != cudaSuccess) ok = false;
    }
    if (ok && (cudaStreamCreateWithFlags(&v->stream, cudaStreamNonBlocking) != cudaSuccess || cudaStreamCreateWithFlags(&v->copy, cudaStreamNonBlocking) != cudaSuccess ||
               cudaEventCreateWithFlags(&v->encoded, cudaEventDisableTiming) != cudaSuccess)) ok = false;
    for (int i = 0; i < 2 && ok; i++) ok = cudaEventCreateWithFlags(&v->walked[i], cudaEventDisableTiming) == cudaSuccess;
    if (ok) {
        std::vector<float> zero(VL_H + 1, 0.f);
        v->c_state = vad_upload(v, zero.data(), VL_H);
        v->status = reinterpret_cast<int *>(vad_upload(v, zero.data(), 1));
        ok = v->c_state && v->status;
    }
    if (ok && v->smem > 48 * 1024 && cudaFuncSetAttribute(vad_encode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)v->smem) != cudaSuccess) ok = false;
    cudaDeviceSynchronize();
    if (!ok) { set_error("vad_new: the tensors contradict the geometry, or a device call failed"); mynah_b200_vad_free(v); return nullptr; }
    return v;
}

void mynah_b200_vad_free(mynah_b200_vad *v) {
    if (!v) return;
    for (void *p : v->owned) cudaFree(p);
    if (v->encoded) cudaEventDestroy(v->encoded);
    for (cudaEvent_t e : v->walked) if (e) cudaEventDestroy(e);
    if (v->copy) cudaStreamDestroy(v->copy);
    if (v->stream) cudaStreamDestroy(v->stream);
    delete v;
}

int mynah_b200_vad_frame_samples(const mynah_b200_vad *v) { return v ? v->d.frame : 0; }

int mynah_b200_vad_probs(mynah_b200_vad *v, const float *samples, size_t n, float *probs, int cap) {
    if (!v || (!samples && n) || !probs) { set_error("vad_probs: bad argument"); return -1; }
    std::lock_guard<std::mutex> lk(v->mu);
    std::vector<float> p;
    const int frames = vad_run(v, samples, n, p);
    v->buf.end_call();
    if (frames < 0) return -1;
    if (frames > cap) { set_error("vad_probs: %d frames, room for %d", frames, cap); return -1; }
    memcpy(probs, p.data(), (size_t)frames * sizeof(float));
    return frames;
}

int mynah_b200_vad_speech_spans(mynah_b200_vad *v, const float *samples, size_t n, long long *spans, int cap) {
    if (!v || (!samples && n) || !spans || cap < 0) { set_error("vad_speech_spans: bad argument"); return -1; }
    std::lock_guard<std::mutex> lk(v->mu);
    std::vector<float> p;
    const int frames = vad_run(v, samples, n, p);
    v->buf.end_call();
    if (frames < 0) return -1;
    const std::vector<Span> sp = spans_from_probs(v->cfg, p, (long long)n);
    if ((int)sp.size() > cap) { set_error("vad_speech_spans: more than %d spans", cap); return -1; }
    for (size_t i = 0; i < sp.size(); i++) { spans[2 * i] = sp[i].t0; spans[2 * i + 1] = sp[i].t1; }
    return (int)sp.size();
}

int mynah_b200_plan_segments(mynah_b200_vad *v, const float *samples, size_t n_samples, int sample_rate, double seg_sec,
                             long long *segs, int cap) {
    if ((!samples && n_samples) || !segs || cap < 1 || sample_rate <= 0 || seg_sec <= 0) { set_error("plan_segments: bad argument"); return -1; }
    if (!mynah_b200_available()) { set_error("plan_segments: no sm_100 device"); return -1; }
    cudaStream_t st = v ? v->stream : nullptr;
    VadBuffers own;                                 // of a call without a network
    VadBuffers &buf = v ? v->buf : own;
    std::unique_lock<std::mutex> lk;
    if (v) lk = std::unique_lock<std::mutex>(v->mu);
    const long long n = (long long)n_samples, sr = sample_rate, seg_max = (long long)(seg_sec * (double)sample_rate);
    std::vector<Span> ranges;                       // what gets cut: the whole signal, or the widened and merged speech spans
    bool vad_plan = false;
    if (v && n > 0) {
        std::vector<float> p;
        if (vad_run(v, samples, n_samples, p) >= 0) {
            std::vector<Span> sp = spans_from_probs(v->cfg, p, n);
            const long long ctx = (long long)(0.6 * (double)sample_rate);      // MYNAH_ASR_VAD_CONTEXT_SEC (src/mynah_asr.c:67-68)
            for (Span &s : sp) { s.t0 = s.t0 > ctx ? s.t0 - ctx : 0; s.t1 = s.t1 + ctx < n ? s.t1 + ctx : n; }
            for (const Span &s : sp) {
                if (!ranges.empty() && s.t0 <= ranges.back().t1) { if (s.t1 > ranges.back().t1) ranges.back().t1 = s.t1; }
                else ranges.push_back(s);
            }
            vad_plan = true;
        }
    }
    if (!vad_plan) {
        ranges.assign(1, Span{0, n});
        if (!buf.audio.grow(n_samples ? n_samples : 1)) return -1;
        if (n && (cudaMemcpyAsync(buf.audio.p, samples, n_samples * sizeof(float), cudaMemcpyHostToDevice, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess)) {
            cudaGetLastError(); set_error("H2D copy failed"); buf.end_call(); return -1;
        }
    }
    std::vector<long long> out;
    std::vector<double> scratch;
    int rc = 0;
    for (const Span &r : ranges) {
        long long cur = r.t0;
        while (cur < r.t1 && rc == 0) {
            long long end = r.t1;
            if (r.t1 - cur > seg_max + seg_max / 10) {                         // +10 %: no split for a small overrun
                const long long hi = cur + seg_max;
                long long lo = seg_max > 20 * sr ? hi - 20 * sr : cur + sr;    // the last 20 s of the window, at least 1 s in
                if (lo <= cur) lo = cur + 1;
                end = split_point_dev(buf, lo, hi, sample_rate, st, scratch);
                if (end < 0) { rc = -1; break; }
                if (vad_plan && (end <= cur || end > r.t1)) end = hi;
            }
            if (end <= cur) end = cur + 1;
            out.push_back(cur); out.push_back(end - cur);
            cur = end;
        }
    }
    buf.end_call();
    if (rc) return -1;
    if (out.empty()) { out.push_back(0); out.push_back(0); }                  // nothing to decode: one empty segment
    const int k = (int)(out.size() / 2);
    if (k > cap) { set_error("plan_segments: %d segments, room for %d", k, cap); return -1; }
    memcpy(segs, out.data(), out.size() * sizeof(long long));
    return k;
}

}  // extern "C"
