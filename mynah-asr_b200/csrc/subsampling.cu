// dw-striding 8x subsampling front-end (the reference's conv2d_s2 /
// mynah_asr_subsampling_forward, src/subsampling.c:107-269), channel-last on device.
//
// The reference keeps activations channel-major [C, T, F] and runs the pointwise
// 1x1 convs as [C,C] x [C,S] GEMMs. Here activations are [T, F, C] so that
//   * the 3x3 stride-2 convs read and write 256 consecutive channels per (t, f)
//     (coalesced), and
//   * each pointwise conv is a plain row-major contraction [S, C] x [C, C]^T on the
//     tensor cores, its epilogue applying bias + ReLU, and the last one emits the
//     [T', F'*C] operand of the output linear directly (the linear's columns are
//     permuted once at load time from the reference's channel-major flatten
//     c*F'+f to f*C+c).
// Zero padding: causal (2 left, 1 right) or symmetric (1, 1) on both axes.
#include "kernels.h"
#include "model.h"

namespace mb {

// stage 0: full conv 1 -> C, 3x3, stride 2, + bias + ReLU.   feats [T,F] -> out [To,Fo,C]
__global__ void __launch_bounds__(256)
conv_in_kernel(const float *__restrict__ x, const float *__restrict__ w, const float *__restrict__ b,
               float *__restrict__ out, int T, int F, int C, int To, int Fo, int pl) {
    const size_t total = (size_t)To * Fo * C;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % C);
        const int fo = (int)((i / C) % Fo);
        const int to = (int)(i / ((size_t)C * Fo));
        float acc = 0.0f;
#pragma unroll
        for (int dt = 0; dt < 3; dt++) {
            const int t = to * 2 - pl + dt;
            if (t < 0 || t >= T) continue;
#pragma unroll
            for (int df = 0; df < 3; df++) {
                const int f = fo * 2 - pl + df;
                if (f < 0 || f >= F) continue;
                acc += w[c * 9 + dt * 3 + df] * x[(size_t)t * F + f];
            }
        }
        out[i] = fmaxf(acc + b[c], 0.0f);
    }
}

int conv_in_relu(const float *feats, const float *w, const float *b, float *out, int T, int F, int C, int To, int Fo,
                 int pl, cudaStream_t st) {
    const size_t total = (size_t)To * Fo * C;
    if (total == 0) return 0;
    const unsigned blocks = (unsigned)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    conv_in_kernel<<<blocks, 256, 0, st>>>(feats, w, b, out, T, F, C, To, Fo, pl);
    MB_CUDA(cudaGetLastError());
    return 0;
}

// stage 0 fused into the first depthwise conv: the [T1, F1, C] activation of stage 0 (the
// largest tensor of the whole model: 196 MB for 60 s of audio) is never materialised.
// Every stage-1 output needs a 3x3 patch of stage-0 outputs, i.e. a 7x7 patch of the
// input; a CTA stages the input rows it needs in shared memory (read by all channels as
// broadcasts, fetched as 16-byte pieces into registers) and one thread per channel recomputes the
// nine stage-0 values in registers.
// Stage-0 positions outside [0,T1) x [0,F1) are the depthwise conv's own zero padding.
static constexpr int FUSE_F2 = 32;     // stage-1 frequency positions of a patch

// the utterance of a group that packed frame `row` of stage 1 (or 2) belongs to
__device__ __forceinline__ int front_find(const FrontItem *__restrict__ items, int n, int row, bool stage2) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((stage2 ? items[mid].off3 : items[mid].off2) <= row) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(256)
conv_in_dw_kernel(const FrontItem *__restrict__ items, int n_items, int rows2, const float *__restrict__ w0, const float *__restrict__ b0,
                  const float *__restrict__ w1, const float *__restrict__ b1, __half *__restrict__ hi,
                  __half *__restrict__ lo, int F, int C, int F1, int F2, int pl) {
    __shared__ __align__(16) float patch[7][4 * FUSE_F2 + 4];
    // A block walks rows with its channels' weights in registers: their loads (36 bytes between lanes) cost more than eight
    // outputs. Along a row the window slides: the first column of stage-0 values is the last one of the output before.
    // 60 s of audio, 256 channels: 125 us with a block per row and eight columns, 98 so; 63 multiply-adds per output are 22.
    const int c = blockIdx.y * 256 + threadIdx.x;
    const bool on = c < C;
    float k0[9], k1[9];
#pragma unroll
    for (int i = 0; i < 9; i++) { k0[i] = on ? w0[c * 9 + i] : 0.f; k1[i] = on ? w1[c * 9 + i] : 0.f; }
    const float bias0 = on ? b0[c] : 0.f, bias1 = on ? b1[c] : 0.f;
    const int pw = 4 * FUSE_F2 + 3;
    for (int row = blockIdx.x; row < rows2; row += gridDim.x) {
        const FrontItem &item = items[front_find(items, n_items, row, false)];
        const float *__restrict__ x = item.feats;
        const int T = item.t_mel, T1 = item.T1, t2 = row - item.off2;
        // stage-0 rows 2*t2 - pl + {0,1,2} need input rows 2*(that) - pl + {0,1,2}
        const int trow0 = 2 * (2 * t2 - pl) - pl;       // first input row of the patch
        for (int f2base = 0; f2base < F2; f2base += FUSE_F2) {
            const int fcol0 = 2 * (2 * f2base - pl) - pl;       // first input column of the patch
            __syncthreads();                            // the patch before has been read
            for (int i = threadIdx.x; i < 7 * pw; i += 256) {
                const int r = i / pw, q = i - r * pw, t = trow0 + r, f = fcol0 + q;
                patch[r][q] = (t >= 0 && t < T && f >= 0 && f < F) ? x[(size_t)t * F + f] : 0.0f;
            }
            __syncthreads();
            if (!on) continue;
            // columns 4 j .. 4 j + 3 of the window, as 16-byte broadcast loads; the next four become them
            float4 left[7];
#pragma unroll
            for (int r = 0; r < 7; r++) left[r] = *reinterpret_cast<const float4 *>(&patch[r][0]);
            float edge[3];                              // stage-0 values of column f1 = 2 f2 - pl, by dt
            auto stage0 = [&](const float (&in)[7][8], int dt, int df) {
                float v = 0.0f;
#pragma unroll
                for (int a = 0; a < 3; a++)
#pragma unroll
                    for (int b = 0; b < 3; b++) v += k0[a * 3 + b] * in[2 * dt + a][2 * df + b];
                return fmaxf(v + bias0, 0.0f);
            };
            const int last = F2 - f2base < FUSE_F2 ? F2 - f2base : FUSE_F2;
            for (int j = 0; j < last; j++) {
                const int f2 = f2base + j;
                float in[7][8];
#pragma unroll
                for (int r = 0; r < 7; r++) {
                    const float4 h4 = *reinterpret_cast<const float4 *>(&patch[r][4 * j + 4]);
                    in[r][0] = left[r].x; in[r][1] = left[r].y; in[r][2] = left[r].z; in[r][3] = left[r].w;
                    in[r][4] = h4.x; in[r][5] = h4.y; in[r][6] = h4.z; in[r][7] = h4.w;
                    left[r] = h4;
                }
                if (j == 0) {
#pragma unroll
                    for (int dt = 0; dt < 3; dt++) edge[dt] = stage0(in, dt, 0);
                }
                const int f1 = 2 * f2 - pl;
                float acc = 0.0f;
#pragma unroll
                for (int dt = 0; dt < 3; dt++) {
                    const int t1 = 2 * t2 - pl + dt;
                    if (t1 < 0 || t1 >= T1) continue;
                    if (f1 >= 0) acc += k1[dt * 3] * edge[dt];
                    if (f1 + 1 < F1) acc += k1[dt * 3 + 1] * stage0(in, dt, 1);
                    edge[dt] = stage0(in, dt, 2);
                    if (f1 + 2 < F1) acc += k1[dt * 3 + 2] * edge[dt];
                }
                __half h, l;
                split_h16(bias1 + acc, h, l);
                const size_t o = ((size_t)row * F2 + f2) * C + c;
                hi[o] = h;
                lo[o] = l;
            }
        }
    }
}

int conv_in_dw_fused(const FrontItem *items, int n_items, int rows2, const float *w0, const float *b0, const float *w1, const float *b1,
                     H16 out, int F, int C, int F1, int F2, int pl, cudaStream_t st) {
    if (rows2 <= 0 || F2 <= 0) return 0;
    const int per = cdiv(C, 256), room = 3 * device_sm_count() / per;
    dim3 grid(rows2 < room || room < 1 ? rows2 : room, per);
    conv_in_dw_kernel<<<grid, 256, 0, st>>>(items, n_items, rows2, w0, b0, w1, b1, out.hi, out.lo, F, C, F1, F2, pl);
    MB_CUDA(cudaGetLastError());
    return 0;
}

// stages 1-2: depthwise 3x3 stride 2 + bias.   x [T,F,C] f32 -> (hi,lo) [To*Fo, C]
__global__ void __launch_bounds__(256)
dw3x3_kernel(const FrontItem *__restrict__ items, int n_items, int rows3, const float *__restrict__ x_all, const float *__restrict__ w,
             const float *__restrict__ b, __half *__restrict__ hi, __half *__restrict__ lo, int F, int C, int Fo, int pl) {
    // a thread keeps its channel and the channel's weights (36 bytes between lanes) for all the outputs of the block
    const int c = blockIdx.y * 256 + threadIdx.x, total = rows3 * Fo;
    if (c >= C) return;
    float k[9];
#pragma unroll
    for (int i = 0; i < 9; i++) k[i] = w[c * 9 + i];
    const float bias = b[c];
    for (int o = blockIdx.x; o < total; o += gridDim.x) {
        const int row = o / Fo, fo = o - row * Fo;
        const FrontItem &item = items[front_find(items, n_items, row, true)];
        const int to = row - item.off3, T = item.T2;
        const float *x = x_all + (size_t)item.off2 * F * C;
        float acc = 0.0f;
#pragma unroll
        for (int dt = 0; dt < 3; dt++) {
            const int t = to * 2 - pl + dt;
            if (t < 0 || t >= T) continue;
#pragma unroll
            for (int df = 0; df < 3; df++) {
                const int f = fo * 2 - pl + df;
                if (f < 0 || f >= F) continue;
                acc += k[dt * 3 + df] * x[((size_t)t * F + f) * C + c];
            }
        }
        __half h, l;
        split_h16(bias + acc, h, l);
        hi[(size_t)o * C + c] = h;
        lo[(size_t)o * C + c] = l;
    }
}

int dwconv3x3_s2(const FrontItem *items, int n_items, int rows3, const float *x, const float *w, const float *b, H16 out, int F, int C,
                 int Fo, int pl, cudaStream_t st) {
    if (rows3 <= 0 || Fo <= 0) return 0;
    const int per = cdiv(C, 256), total = rows3 * Fo, room = 8 * device_sm_count() / per;      // eight blocks of 256 to an SM
    dw3x3_kernel<<<dim3(total < room || room < 1 ? total : room, per), 256, 0, st>>>(items, n_items, rows3, x, w, b, out.hi, out.lo, F, C, Fo, pl);
    MB_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace mb
