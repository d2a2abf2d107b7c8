// fx_learned.cu -- training of the learned smoother's network (new; no reference counterpart):
// parameters, the per-sample forward and backward pass, the deterministic batch gradient, Adam,
// and the packing of the trained weights into the inference kernel's MMA operand fragments.
// The network, the loss and the sample layout are described in fx_learned.cuh.
//
// Training runs on the CUDA cores in FP32 with the network's own rounding: weights and hidden
// activations rounded to BF16 exactly as the tensor-core inference kernel rounds them, so a
// trained network computes in training what it computes when applied.  A block takes whole samples
// and one reduction kernel adds the blocks' partial gradients in block order, so a gradient is
// bitwise reproducible.
//
// A sample is 3.9 million fused multiply-adds, which the FP32 units bound (a block's operands stay in
// shared memory); a thread computing one output, or one parameter's gradient, at a time loads two
// operands for each and ran at 0.09 of the FP32 rate (2.43 ms for 2048 samples).  So every phase
// is tiled in registers: the convolutions compute 8 (or 7) points of a row x 4 channels per thread,
// the weight gradients 8 output channels x 3 taps of a row per thread over a share of the rows.
// Activations lie point by point with their channels adjacent, padded so that the lanes of a warp
// (4 channel groups x 8 rows, or 16 channels) fall in distinct banks: 0.57 ms, 0.39 of the FP32 rate
// (0.59 ms with the call around it), with 18 warps per SM and the gradient sums spilled between phases.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>

#include "fx_learned.cuh"

using namespace fx;
using namespace fx::lsm;

namespace {

constexpr int kTrThreads = 288;
constexpr int kMaxPartBlocks = 1024;

// shared-memory layout of the training kernel (floats)
constexpr int kStr1 = 18;                      // a1: floats per point (16 channels; 8-byte aligned groups)
constexpr int kStr2 = 20;                      // a2: floats per point (16-byte aligned groups)
constexpr int kPad2 = kP2 + 4;                 // a2: points per row, two zero columns on each side
constexpr int kSmA1 = kP1 * kP1 * kStr1;       // a1, later the gradient at a1's pre-activation
constexpr int kSmA2 = kP2 * kPad2 * kStr2;     // a2, later the gradient at a2's pre-activation
constexpr int kSmC = kP3 * kP3;                // 361: network output c; and as many: dL/dc
constexpr int kSmG = kT * kT;                  // 256: dL/d(Hc), then 256: the whole-error part of dL/dc
constexpr int kSmR = kNCo * kNCo;              // 81: R c, later P^T dL/d(Hc)
constexpr int kSmW1 = kIn * 9 * kC;            // [ci][tap][co]
constexpr int kSmW2 = kC * 9 * kC;             // [ci][tap][co], and as many [co][tap][ci]
constexpr int kSmW3 = 9 * kC;                  // [tap][ci]
constexpr int kSmInHalf = (kInLen + 5) / 2;    // BF16 inputs, and what the last row's tile reads past them
constexpr int kSmTrainWords = kSmA1 + kSmA2 + kSmW1 + 2 * kSmW2 + kSmW3 + 2 * kC + 4 + 2 * (kSmC + 3) + 2 * kSmG +
                              (kSmR + 3) + 32 + kSmInHalf;
constexpr int kSmTrain = kSmTrainWords * 4;
static_assert(2 * (kSmTrain + 1024) <= 228 * 1024, "two blocks per SM");
// parts of the block that share a parameter's gradient: rows of the layer's output
constexpr int kRg1 = 16, kRg2 = 3, kRg3 = 6, kRgB = kTrThreads / kC;
static_assert(kRg2 * kSmW2 + kRg1 * kSmW1 + kRg3 * kSmW3 + 2 * kTrThreads + kTrThreads <= kSmA1 + kSmA2,
              "the final sums fit the activations' space");

// R at coarse point (I, J) of a field over the output region [-1, 17]^2 (index offset 1)
__device__ __forceinline__ float fw19(const float *f, int I, int J) {
    const int y = 2 * I + 1, x = 2 * J + 1;
    const float *c = f + y * kP3 + x;
    const float e = (c[-kP3] + c[kP3]) + (c[-1] + c[1]);
    const float d = (c[-kP3 - 1] + c[-kP3 + 1]) + (c[kP3 - 1] + c[kP3 + 1]);
    return (4.f * c[0] + (2.f * e + d)) * 0.0625f;
}

// bilinear interpolation of the coarse values Rc at loss point (py, px)
__device__ __forceinline__ float bil9(const float *Rc, int py, int px) {
    const int I = py >> 1, J = px >> 1;
    const float *r = Rc + I * kNCo + J;
    const bool oy = py & 1, ox = px & 1;
    if (!oy && !ox) return r[0];
    if (oy && !ox) return 0.5f * (r[0] + r[kNCo]);
    if (!oy && ox) return 0.5f * (r[0] + r[1]);
    return 0.25f * ((r[0] + r[kNCo]) + (r[1] + r[kNCo + 1]));
}

// One block per group of samples: forward, loss and backward of each, gradients accumulated in
// registers over the block's samples; writes part[block][p] and part[block][kNParams] = the block's
// summed loss.
__global__ void __launch_bounds__(kTrThreads, 2) k_lsm_train(const float *__restrict__ wq,
                                                             const __nv_bfloat16 *__restrict__ in_all,
                                                             const float *__restrict__ tgt_all,
                                                             const float *__restrict__ norm_all,
                                                             const int *__restrict__ idx, int count, float lambda,
                                                             float *__restrict__ part) {
    extern __shared__ __align__(16) float tsm[];
    float *S_a2 = tsm;  // 16-byte aligned groups first
    float *S_w1 = S_a2 + kSmA2;
    float *S_w2f = S_w1 + kSmW1;  // [ci][tap][co]
    float *S_w2b = S_w2f + kSmW2;  // [co][tap][ci]
    float *S_w3 = S_w2b + kSmW2;
    float *S_b1 = S_w3 + kSmW3;
    float *S_b2 = S_b1 + kC;
    float *S_b3 = S_b2 + kC;
    float *S_a1 = S_b3 + 4;
    float *S_c = S_a1 + kSmA1;
    float *S_gc = S_c + kSmC + 3;
    float *S_gh = S_gc + kSmC + 3;
    float *S_ge = S_gh + kSmG;
    float *S_r = S_ge + kSmG;
    float *S_red = S_r + kSmR + 3;
    __nv_bfloat16 *S_in = reinterpret_cast<__nv_bfloat16 *>(S_red + 32);
    const int tid = threadIdx.x;
    for (int p = tid; p < kSmW1; p += kTrThreads) {
        const int co = p % kC, t = p / kC;
        S_w1[p] = wq[w1(co, t / 9, t % 9)];
    }
    for (int p = tid; p < kSmW2; p += kTrThreads) {
        const int lo = p % kC, t = p / kC;
        S_w2f[p] = wq[w2(lo, t / 9, t % 9)];
        S_w2b[p] = wq[w2(t / 9, lo, t % 9)];
    }
    for (int p = tid; p < kSmW3; p += kTrThreads) S_w3[p] = wq[w3(p % kC, p / kC)];
    if (tid < kC) {
        S_b1[tid] = wq[kOffB1 + tid];
        S_b2[tid] = wq[kOffB2 + tid];
    }
    if (tid == 0) S_b3[0] = wq[kOffB3];
    for (int p = tid; p < kSmA2; p += kTrThreads) S_a2[p] = 0.f;  // the zero columns stay zero
    for (int p = tid; p < 2 * kSmInHalf; p += kTrThreads) S_in[p] = __float2bfloat16_rn(0.f);

    // tiles of the convolutions: 4 channels (cg) of 8 or 7 points of a row
    const int cg = tid & 3, trow1 = (tid >> 2) % kP1, tx1 = (tid >> 2) / kP1 * 8;
    const int trow2 = (tid >> 2) % kP2, tx2 = (tid >> 2) / kP2 * 7;
    const bool on1 = tid < 4 * kP1 * 3, on2 = tid < 4 * kP2 * 3;
    // tiles of the weight gradients: 8 output channels x 3 taps of filter row ky, one input channel
    const int g2ci = tid % kC, g2ky = tid / kC % 3, g2h = tid / 48 % 2, g2r = tid / 96;
    const int g1t = tid % 18, g1ci = g1t % 3, g1ky = g1t / 3 % 3, g1h = g1t / 9, g1r = tid / 18;
    const int g3ci = tid % kC, g3ky = tid / kC % 3, g3r = tid / 48;
    const int bco = tid % kC, bgr = tid / kC;
    float acc2[8][3] = {}, acc1[8][3] = {}, acc3[3] = {}, accb1 = 0.f, accb2 = 0.f, accb3 = 0.f;
    float loss_acc = 0.f;
    __syncthreads();

    for (int sidx = blockIdx.x; sidx < count; sidx += gridDim.x) {
        const int s = idx[sidx];
        const __nv_bfloat16 *in = in_all + (size_t)s * kInLen;
        const float *tgt = tgt_all + (size_t)s * kTgtLen;  // tH [256], tE [256]
        const float nrm = norm_all[2 * s] + lambda * norm_all[2 * s + 1];
        const float inv_n = nrm > 0.f ? 1.f / nrm : 0.f;
        for (int k = tid; k < kInLen; k += kTrThreads) S_in[k] = in[k];
        __syncthreads();
        // ---- forward: every output accumulates over (ci, tap) from its bias
        if (on1) {  // a1 = bf16(relu(conv1 + b1))
            float z[8][4];
#pragma unroll
            for (int p = 0; p < 8; p++)
#pragma unroll
                for (int c = 0; c < 4; c++) z[p][c] = S_b1[cg * 4 + c];
#pragma unroll
            for (int ci = 0; ci < kIn; ci++)
#pragma unroll
                for (int ky = 0; ky < 3; ky++) {
                    const __nv_bfloat16 *a = S_in + ci * kPin * kPin + (trow1 + ky) * kPin + tx1;
                    float v[10];
#pragma unroll
                    for (int j = 0; j < 10; j++) v[j] = __bfloat162float(a[j]);
#pragma unroll
                    for (int kx = 0; kx < 3; kx++) {
                        const float4 w = *reinterpret_cast<const float4 *>(S_w1 + (ci * 9 + ky * 3 + kx) * kC + cg * 4);
#pragma unroll
                        for (int p = 0; p < 8; p++) {
                            z[p][0] = fmaf(w.x, v[p + kx], z[p][0]);
                            z[p][1] = fmaf(w.y, v[p + kx], z[p][1]);
                            z[p][2] = fmaf(w.z, v[p + kx], z[p][2]);
                            z[p][3] = fmaf(w.w, v[p + kx], z[p][3]);
                        }
                    }
                }
#pragma unroll
            for (int p = 0; p < 8; p++)
                if (tx1 + p < kP1) {
                    float2 *o = reinterpret_cast<float2 *>(S_a1 + (trow1 * kP1 + tx1 + p) * kStr1 + cg * 4);
                    o[0] = make_float2(bf16r(fmaxf(z[p][0], 0.f)), bf16r(fmaxf(z[p][1], 0.f)));
                    o[1] = make_float2(bf16r(fmaxf(z[p][2], 0.f)), bf16r(fmaxf(z[p][3], 0.f)));
                }
        }
        __syncthreads();
        if (on2) {  // a2 = bf16(relu(conv2 + b2))
            float z[7][4];
#pragma unroll
            for (int p = 0; p < 7; p++)
#pragma unroll
                for (int c = 0; c < 4; c++) z[p][c] = S_b2[cg * 4 + c];
#pragma unroll 2
            for (int ci = 0; ci < kC; ci++)
#pragma unroll
                for (int ky = 0; ky < 3; ky++) {
                    const float *a = S_a1 + ((trow2 + ky) * kP1 + tx2) * kStr1 + ci;
                    float v[9];
#pragma unroll
                    for (int j = 0; j < 9; j++) v[j] = a[j * kStr1];
#pragma unroll
                    for (int kx = 0; kx < 3; kx++) {
                        const float4 w = *reinterpret_cast<const float4 *>(S_w2f + (ci * 9 + ky * 3 + kx) * kC + cg * 4);
#pragma unroll
                        for (int p = 0; p < 7; p++) {
                            z[p][0] = fmaf(w.x, v[p + kx], z[p][0]);
                            z[p][1] = fmaf(w.y, v[p + kx], z[p][1]);
                            z[p][2] = fmaf(w.z, v[p + kx], z[p][2]);
                            z[p][3] = fmaf(w.w, v[p + kx], z[p][3]);
                        }
                    }
                }
#pragma unroll
            for (int p = 0; p < 7; p++)
                *reinterpret_cast<float4 *>(S_a2 + (trow2 * kPad2 + tx2 + p + 2) * kStr2 + cg * 4) =
                    make_float4(bf16r(fmaxf(z[p][0], 0.f)), bf16r(fmaxf(z[p][1], 0.f)), bf16r(fmaxf(z[p][2], 0.f)),
                                bf16r(fmaxf(z[p][3], 0.f)));
        }
        __syncthreads();
        for (int o = tid; o < kP3 * kP3; o += kTrThreads) {  // c = conv3 + b3
            const int y = o / kP3, x = o - y * kP3;
            float z = S_b3[0];
            for (int ci = 0; ci < kC; ci += 4) {
                float4 a[9], w[9];
#pragma unroll
                for (int tap = 0; tap < 9; tap++) {
                    a[tap] = *reinterpret_cast<const float4 *>(S_a2 + ((y + tap / 3) * kPad2 + x + tap % 3 + 2) * kStr2 + ci);
                    w[tap] = *reinterpret_cast<const float4 *>(S_w3 + tap * kC + ci);
                }
#pragma unroll
                for (int tap = 0; tap < 9; tap++) z = fmaf(w[tap].x, a[tap].x, z);
#pragma unroll
                for (int tap = 0; tap < 9; tap++) z = fmaf(w[tap].y, a[tap].y, z);
#pragma unroll
                for (int tap = 0; tap < 9; tap++) z = fmaf(w[tap].z, a[tap].z, z);
#pragma unroll
                for (int tap = 0; tap < 9; tap++) z = fmaf(w[tap].w, a[tap].w, z);
            }
            S_c[o] = z;
        }
        __syncthreads();
        for (int o = tid; o < kSmR; o += kTrThreads) S_r[o] = fw19(S_c, o / kNCo, o % kNCo);
        __syncthreads();
        // ---- loss; dL/d(Hc) = -2 (tH - Hc) / n and the whole-error part -2 lambda (tE - c) / n
        float lsum = 0.f;
        for (int o = tid; o < kT * kT; o += kTrThreads) {
            const int py = o / kT, px = o - py * kT;
            const float cv = S_c[(py + 1) * kP3 + px + 1];
            const float u = tgt[o] - (cv - bil9(S_r, py, px));
            const float w = tgt[kT * kT + o] - cv;
            lsum = fmaf(u, u, lsum);
            lsum = fmaf(lambda * w, w, lsum);
            S_gh[o] = -2.f * u * inv_n;
            S_ge[o] = -2.f * lambda * w * inv_n;
        }
        // block sum of lsum: warp shuffles, then the warp partials (the barrier also publishes
        // S_gh and ends the previous sample's reads of S_red)
        for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, off);
        __syncthreads();
        if ((tid & 31) == 0) S_red[tid >> 5] = lsum;
        __syncthreads();
        if (tid == 0) {
            float t = 0.f;
            for (int w = 0; w < kTrThreads / 32; w++) t += S_red[w];
            loss_acc += t * inv_n;
        }
        // ---- backward through H = I - P R: dL/dc = g - R^T P^T g (g on the loss region)
        for (int o = tid; o < kSmR; o += kTrThreads) {  // (P^T g) at coarse (I, J)
            const int I = o / kNCo, J = o - I * kNCo;
            float acc = 0.f;
            for (int dy = -1; dy <= 1; dy++)
                for (int dx = -1; dx <= 1; dx++) {
                    const int py = 2 * I + dy, px = 2 * J + dx;
                    if (py < 0 || px < 0 || py >= kT || px >= kT) continue;
                    const float wgt = (dy == 0 ? 1.f : 0.5f) * (dx == 0 ? 1.f : 0.5f);
                    acc = fmaf(wgt, S_gh[py * kT + px], acc);
                }
            S_r[o] = acc;
        }
        __syncthreads();
        for (int o = tid; o < kP3 * kP3; o += kTrThreads) {  // dL/dc over [-1, 17]^2
            const int y = o / kP3, x = o - y * kP3;
            const int ly = y - 1, lx = x - 1;  // loss coordinates
            float g = (ly >= 0 && lx >= 0 && ly < kT && lx < kT) ? S_gh[ly * kT + lx] + S_ge[ly * kT + lx] : 0.f;
            for (int I = (ly - 1 + 1) >> 1; I <= (ly + 1) >> 1; I++) {
                if (I < 0 || I >= kNCo || 2 * I < ly - 1 || 2 * I > ly + 1) continue;
                for (int J = (lx - 1 + 1) >> 1; J <= (lx + 1) >> 1; J++) {
                    if (J < 0 || J >= kNCo || 2 * J < lx - 1 || 2 * J > lx + 1) continue;
                    const float wr = (2 * I == ly ? 2.f : 1.f) * (2 * J == lx ? 2.f : 1.f) * 0.0625f;
                    g = fmaf(-wr, S_r[I * kNCo + J], g);
                }
            }
            S_gc[o] = g;
            accb3 += g;  // db3
        }
        __syncthreads();
        // ---- conv3: dW3, then dL/dz2 in place of a2
        {
            float t[3] = {};
            for (int y = g3r; y < kP3; y += kRg3) {
                const float *a = S_a2 + ((y + g3ky) * kPad2 + 2) * kStr2 + g3ci;
                float a0 = a[0], a1 = a[kStr2];
#pragma unroll 4
                for (int x = 0; x < kP3; x++) {
                    const float a2 = a[(x + 2) * kStr2], g = S_gc[y * kP3 + x];
                    t[0] = fmaf(g, a0, t[0]);
                    t[1] = fmaf(g, a1, t[1]);
                    t[2] = fmaf(g, a2, t[2]);
                    a0 = a1;
                    a1 = a2;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; k++) acc3[k] += t[k];
        }
        __syncthreads();
        for (int o = tid; o < kP2 * kP2; o += kTrThreads) {
            const int y = o / kP2, x = o - y * kP2;
            float g[9];
#pragma unroll
            for (int tap = 0; tap < 9; tap++) {
                const int cy = y - tap / 3, cx = x - tap % 3;
                g[tap] = (cy < 0 || cx < 0 || cy >= kP3 || cx >= kP3) ? 0.f : S_gc[cy * kP3 + cx];
            }
            float4 *a = reinterpret_cast<float4 *>(S_a2 + (y * kPad2 + x + 2) * kStr2);
#pragma unroll
            for (int q = 0; q < kC / 4; q++) {
                float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int tap = 0; tap < 9; tap++) {
                    const float4 w = *reinterpret_cast<const float4 *>(S_w3 + tap * kC + 4 * q);
                    z.x = fmaf(w.x, g[tap], z.x);
                    z.y = fmaf(w.y, g[tap], z.y);
                    z.z = fmaf(w.z, g[tap], z.z);
                    z.w = fmaf(w.w, g[tap], z.w);
                }
                const float4 v = a[q];  // ReLU mask from a2 itself
                a[q] = make_float4(v.x > 0.f ? z.x : 0.f, v.y > 0.f ? z.y : 0.f, v.z > 0.f ? z.z : 0.f,
                                   v.w > 0.f ? z.w : 0.f);
            }
        }
        __syncthreads();
        // ---- conv2: dW2, db2, then dL/dz1 in place of a1
        {
            float t[8][3] = {};
            for (int y = 7 * g2r; y < 7 * g2r + 7; y++) {
                const float *a = S_a1 + (y + g2ky) * kP1 * kStr1 + g2ci;
                const float *gz = S_a2 + (y * kPad2 + 2) * kStr2 + 8 * g2h;
                float a0 = a[0], a1 = a[kStr1];
#pragma unroll 3
                for (int x = 0; x < kP2; x++) {
                    const float a2 = a[(x + 2) * kStr1];
                    const float4 lo = *reinterpret_cast<const float4 *>(gz + x * kStr2);
                    const float4 hi = *reinterpret_cast<const float4 *>(gz + x * kStr2 + 4);
                    const float g[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        t[c][0] = fmaf(g[c], a0, t[c][0]);
                        t[c][1] = fmaf(g[c], a1, t[c][1]);
                        t[c][2] = fmaf(g[c], a2, t[c][2]);
                    }
                    a0 = a1;
                    a1 = a2;
                }
            }
#pragma unroll
            for (int c = 0; c < 8; c++)
#pragma unroll
                for (int k = 0; k < 3; k++) acc2[c][k] += t[c][k];
            float b = 0.f;
            for (int o = bgr; o < kP2 * kP2; o += kRgB) b += S_a2[(o / kP2 * kPad2 + o % kP2 + 2) * kStr2 + bco];
            accb2 += b;
        }
        __syncthreads();
        if (on1) {  // dL/dz1 of 4 input channels (cg) of 8 points: transposed filters over the padded rows
            float z[8][4] = {};
#pragma unroll 2
            for (int co = 0; co < kC; co++)
#pragma unroll
                for (int ky = 0; ky < 3; ky++) {
                    const int zy = trow1 - ky;
                    if (zy < 0 || zy >= kP2) continue;
                    const float *gz = S_a2 + (zy * kPad2 + tx1) * kStr2 + co;
                    float v[10];
#pragma unroll
                    for (int j = 0; j < 10; j++) v[j] = gz[j * kStr2];  // v[j]: point tx1 + j - 2
#pragma unroll
                    for (int kx = 0; kx < 3; kx++) {
                        const float4 w = *reinterpret_cast<const float4 *>(S_w2b + (co * 9 + ky * 3 + kx) * kC + cg * 4);
#pragma unroll
                        for (int p = 0; p < 8; p++) {
                            z[p][0] = fmaf(w.x, v[p + 2 - kx], z[p][0]);
                            z[p][1] = fmaf(w.y, v[p + 2 - kx], z[p][1]);
                            z[p][2] = fmaf(w.z, v[p + 2 - kx], z[p][2]);
                            z[p][3] = fmaf(w.w, v[p + 2 - kx], z[p][3]);
                        }
                    }
                }
#pragma unroll
            for (int p = 0; p < 8; p++)
                if (tx1 + p < kP1) {
                    float2 *o = reinterpret_cast<float2 *>(S_a1 + (trow1 * kP1 + tx1 + p) * kStr1 + cg * 4);
                    const float2 u = o[0], v = o[1];
                    o[0] = make_float2(u.x > 0.f ? z[p][0] : 0.f, u.y > 0.f ? z[p][1] : 0.f);
                    o[1] = make_float2(v.x > 0.f ? z[p][2] : 0.f, v.y > 0.f ? z[p][3] : 0.f);
                }
        }
        __syncthreads();
        // ---- conv1: dW1, db1
        {
            float t[8][3] = {};
            for (int y = g1r; y < kP1; y += kRg1) {
                const __nv_bfloat16 *a = S_in + g1ci * kPin * kPin + (y + g1ky) * kPin;
                const float *gz = S_a1 + y * kP1 * kStr1 + 8 * g1h;
                float a0 = __bfloat162float(a[0]), a1 = __bfloat162float(a[1]);
                for (int x = 0; x < kP1; x++) {
                    const float a2 = __bfloat162float(a[x + 2]);
                    const float2 *gp = reinterpret_cast<const float2 *>(gz + x * kStr1);
                    const float2 g01 = gp[0], g23 = gp[1], g45 = gp[2], g67 = gp[3];
                    const float g[8] = {g01.x, g01.y, g23.x, g23.y, g45.x, g45.y, g67.x, g67.y};
#pragma unroll
                    for (int c = 0; c < 8; c++) {
                        t[c][0] = fmaf(g[c], a0, t[c][0]);
                        t[c][1] = fmaf(g[c], a1, t[c][1]);
                        t[c][2] = fmaf(g[c], a2, t[c][2]);
                    }
                    a0 = a1;
                    a1 = a2;
                }
            }
#pragma unroll
            for (int c = 0; c < 8; c++)
#pragma unroll
                for (int k = 0; k < 3; k++) acc1[c][k] += t[c][k];
            float b = 0.f;
            for (int o = bgr; o < kP1 * kP1; o += kRgB) b += S_a1[o * kStr1 + bco];
            accb1 += b;
        }
        __syncthreads();
    }
    // ---- the parts of each parameter's gradient, added in a fixed order
    float *T2 = tsm, *T1 = T2 + kRg2 * kSmW2, *T3 = T1 + kRg1 * kSmW1, *TB = T3 + kRg3 * kSmW3;
    static_assert(kSmA2 + kSmW1 + 2 * kSmW2 + kSmW3 + 2 * kC + 4 + kSmA1 >=
                      kRg2 * kSmW2 + kRg1 * kSmW1 + kRg3 * kSmW3 + 3 * kTrThreads, "final sums");
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            T2[g2r * kSmW2 + ((8 * g2h + c) * kC + g2ci) * 9 + 3 * g2ky + k] = acc2[c][k];
            T1[g1r * kSmW1 + ((8 * g1h + c) * kIn + g1ci) * 9 + 3 * g1ky + k] = acc1[c][k];
        }
#pragma unroll
    for (int k = 0; k < 3; k++) T3[g3r * kSmW3 + g3ci * 9 + 3 * g3ky + k] = acc3[k];
    TB[tid] = accb1;
    TB[kTrThreads + tid] = accb2;
    TB[2 * kTrThreads + tid] = accb3;
    __syncthreads();
    float *out = part + (size_t)blockIdx.x * (kNParams + 1);
    for (int p = tid; p < kNParams; p += kTrThreads) {
        float g = 0.f;
        if (p < kOffB1)
            for (int r = 0; r < kRg1; r++) g += T1[r * kSmW1 + p - kOffW1];
        else if (p < kOffW2)
            for (int r = 0; r < kRgB; r++) g += TB[r * kC + p - kOffB1];
        else if (p < kOffB2)
            for (int r = 0; r < kRg2; r++) g += T2[r * kSmW2 + p - kOffW2];
        else if (p < kOffW3)
            for (int r = 0; r < kRgB; r++) g += TB[kTrThreads + r * kC + p - kOffB2];
        else if (p < kOffB3)
            for (int r = 0; r < kRg3; r++) g += T3[r * kSmW3 + p - kOffW3];
        else
            for (int r = 0; r < kTrThreads; r++) g += TB[2 * kTrThreads + r];
        out[p] = g;
    }
    if (tid == 0) out[kNParams] = loss_acc;
}

// grad[p] = sum over blocks of part[b][p], in block order (p = kNParams: the loss)
__global__ void k_lsm_reduce(const float *__restrict__ part, int nblocks, float *__restrict__ grad) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > kNParams) return;
    float s = 0.f;
    for (int b = 0; b < nblocks; b++) s += part[(size_t)b * (kNParams + 1) + p];
    grad[p] = s;
}

// Adam (Kingma & Ba 2015) on the mean gradient grad / batch, with bias correction.
__global__ void k_lsm_adam(float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
                           const float *__restrict__ grad, float inv_batch, float lr, float b1, float b2, float eps,
                           float c1, float c2) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kNParams) return;
    const float g = grad[p] * inv_batch;
    const float mm = b1 * m[p] + (1.f - b1) * g;
    const float vv = b2 * v[p] + (1.f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    w[p] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

__device__ __forceinline__ bool is_bias(int p) {
    return (p >= kOffB1 && p < kOffW2) || (p >= kOffB2 && p < kOffW3) || p == kOffB3;
}

// wq = the parameters as the network uses them; frag = the MMA B-operand fragments (see
// fx_learned.cuh).  Fragment element (k, n) of lane l: k = 2 (l % 4) + {0, 1} (+ 8 for the second
// register), n = l / 4.
__global__ void k_lsm_pack(const float *__restrict__ w, float *__restrict__ wq, uint32_t *__restrict__ frag) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < kNParams) wq[t] = is_bias(t) ? w[t] : __bfloat162float(__float2bfloat16_rn(w[t]));
    if (t >= kFragWords) return;
    auto r = [&](int p) { return w[p]; };
    float lo = 0.f, hi = 0.f;
    if (t < kFrag1) {  // conv1: [ks][nh][lane][reg], k = tap * 4 + ch (ch 3 and k >= 36 are zero)
        const int reg = t & 1, lane = (t >> 1) & 31, nh = (t >> 6) & 1, ks = t >> 7;
        const int k = ks * 16 + reg * 8 + (lane & 3) * 2, co = nh * 8 + (lane >> 2);
        auto b1 = [&](int kk) {
            const int tap = kk >> 2, ch = kk & 3;
            return (tap < 9 && ch < kIn) ? r(w1(co, ch, tap)) : 0.f;
        };
        lo = b1(k);
        hi = b1(k + 1);
    } else if (t < kFrag1 + kFrag2) {  // conv2: [tap][nh][lane][reg], k = ci
        const int u = t - kFrag1;
        const int reg = u & 1, lane = (u >> 1) & 31, nh = (u >> 6) & 1, tap = u >> 7;
        const int ci = reg * 8 + (lane & 3) * 2, co = nh * 8 + (lane >> 2);
        lo = r(w2(co, ci, tap));
        hi = r(w2(co, ci + 1, tap));
    } else {  // conv3: [tap][lane][reg], k = ci, only n = 0 nonzero
        const int u = t - kFrag1 - kFrag2;
        const int reg = u & 1, lane = (u >> 1) & 31, tap = u >> 6;
        const int ci = reg * 8 + (lane & 3) * 2;
        if ((lane >> 2) == 0) {
            lo = r(w3(ci, tap));
            hi = r(w3(ci + 1, tap));
        }
    }
    frag[t] = pack_bf16x2(lo, hi);
}

}  // namespace

int fx_lsm::pack() {
    const int n = kFragWords > kNParams ? kFragWords : kNParams;
    k_lsm_pack<<<(n + 255) / 256, 256, 0, ctx->stream>>>(d_w, d_wq, d_frag);
    return check_launch(ctx, "lsm_pack");
}

namespace fx {

// The summed gradient and loss of the samples h_idx[0..count) -> m->d_grad (asynchronous).
int lsm_batch_grad(fx_lsm *m, const fx_lsm_data *d, const int *h_idx, size_t count, float lambda) {
    fx_ctx *ctx = m->ctx;
    if (count == 0) return fail(FX_ERR_INVALID_ARGUMENT, "empty batch");
    for (size_t i = 0; i < count; i++)
        if (h_idx[i] < 0 || (size_t)h_idx[i] >= d->count)
            return fail(FX_ERR_INVALID_ARGUMENT, "sample index out of range");
    if (count > m->idx_cap) {
        if (m->d_idx) cudaFreeAsync(m->d_idx, ctx->stream);
        m->d_idx = nullptr;
        FX_CUDA(cudaMallocAsync(&m->d_idx, count * sizeof(int), ctx->stream));
        m->idx_cap = count;
    }
    FX_CUDA(cudaMemcpyAsync(m->d_idx, h_idx, count * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    const int blocks = (int)std::min<size_t>(count, (size_t)m->part_blocks);
    timing_pre(ctx, "lsm_train");
    k_lsm_train<<<blocks, kTrThreads, kSmTrain, ctx->stream>>>(m->d_wq, d->d_in, d->d_tgt, d->d_norm, m->d_idx,
                                                               (int)count, lambda, m->d_part);
    timing_post(ctx, (double)count);
    FX_TRY(check_launch(ctx, "lsm_train"));
    k_lsm_reduce<<<(kNParams + 1 + 255) / 256, 256, 0, ctx->stream>>>(m->d_part, blocks, m->d_grad);
    return check_launch(ctx, "lsm_reduce");
}

}  // namespace fx

extern "C" {

int fx_lsm_param_count(size_t *n) {
    if (!n) return fail(FX_ERR_INVALID_ARGUMENT, "null out");
    *n = kNParams;
    return FX_OK;
}

int fx_lsm_destroy(fx_lsm *m) {
    if (!m) return FX_OK;
    cudaSetDevice(m->ctx->device);
    cudaStreamSynchronize(m->ctx->stream);
    for (void *p : {(void *)m->d_w, (void *)m->d_wq, (void *)m->d_frag, (void *)m->d_m, (void *)m->d_v,
                    (void *)m->d_part, (void *)m->d_grad, (void *)m->d_idx})
        if (p) cudaFree(p);
    delete m;
    return FX_OK;
}

int fx_lsm_create(fx_ctx *ctx, unsigned long long seed, fx_lsm **out) {
    if (!ctx || !out) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    static bool attr_set[64] = {};
    if (ctx->device >= 0 && ctx->device < 64 && !attr_set[ctx->device]) {
        FX_CUDA(cudaFuncSetAttribute(k_lsm_train, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmTrain));
        attr_set[ctx->device] = true;
    }
    fx_lsm *m = new fx_lsm();
    m->ctx = ctx;
    int occ = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_lsm_train, kTrThreads, kSmTrain) != cudaSuccess || occ < 1)
        occ = 1;
    m->part_blocks = std::min(kMaxPartBlocks, occ * ctx->num_sms);
    const size_t P = kNParams;
    if (cudaMalloc(&m->d_w, P * 4) != cudaSuccess || cudaMalloc(&m->d_wq, P * 4) != cudaSuccess ||
        cudaMalloc(&m->d_frag, kFragWords * 4) != cudaSuccess || cudaMalloc(&m->d_m, P * 4) != cudaSuccess ||
        cudaMalloc(&m->d_v, P * 4) != cudaSuccess || cudaMalloc(&m->d_grad, (P + 1) * 4) != cudaSuccess ||
        cudaMalloc(&m->d_part, (size_t)m->part_blocks * (P + 1) * 4) != cudaSuccess) {
        (void)cudaGetLastError();
        fx_lsm_destroy(m);
        return fail(FX_ERR_BACKEND, "learned smoother: allocation failed");
    }
    // He-normal initialisation of W1 and W2 (std sqrt(2 / fan_in)), zero biases, and a zero last
    // layer, so that the untrained smoother is the weighted-Jacobi step
    std::vector<float> h(P, 0.f);
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.f, 1.f);
    const float s1 = std::sqrt(2.f / (kIn * 9)), s2 = std::sqrt(2.f / (kC * 9));
    for (int p = kOffW1; p < kOffB1; p++) h[p] = s1 * nd(rng);
    for (int p = kOffW2; p < kOffB2; p++) h[p] = s2 * nd(rng);
    int st = FX_OK;
    if (cudaMemcpyAsync(m->d_w, h.data(), P * 4, cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
        cudaMemsetAsync(m->d_m, 0, P * 4, ctx->stream) != cudaSuccess ||
        cudaMemsetAsync(m->d_v, 0, P * 4, ctx->stream) != cudaSuccess ||
        cudaStreamSynchronize(ctx->stream) != cudaSuccess)
        st = fail(FX_ERR_BACKEND, "learned smoother: initialisation failed");
    if (st == FX_OK) st = m->pack();
    if (st != FX_OK) {
        fx_lsm_destroy(m);
        return st;
    }
    *out = m;
    return FX_OK;
}

int fx_lsm_get_params(fx_lsm *m, float *dst, size_t n) {
    if (!m || !dst) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    if (n != (size_t)kNParams) return fail(FX_ERR_DIMENSION_MISMATCH, "parameter count is " + std::to_string(kNParams));
    FX_CUDA(cudaMemcpyAsync(dst, m->d_w, n * 4, cudaMemcpyDeviceToHost, m->ctx->stream));
    FX_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return FX_OK;
}

int fx_lsm_set_params(fx_lsm *m, const float *src, size_t n) {
    if (!m || !src) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    if (n != (size_t)kNParams) return fail(FX_ERR_DIMENSION_MISMATCH, "parameter count is " + std::to_string(kNParams));
    FX_CUDA(cudaMemcpyAsync(m->d_w, src, n * 4, cudaMemcpyHostToDevice, m->ctx->stream));
    FX_CUDA(cudaMemsetAsync(m->d_m, 0, n * 4, m->ctx->stream));
    FX_CUDA(cudaMemsetAsync(m->d_v, 0, n * 4, m->ctx->stream));
    m->adam_t = 0;
    FX_TRY(m->pack());
    FX_CUDA(cudaStreamSynchronize(m->ctx->stream));
    return FX_OK;
}

int fx_lsm_data_create(fx_ctx *ctx, size_t capacity, fx_lsm_data **out) {
    if (!ctx || !out) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    if (capacity == 0 || capacity > ((size_t)1 << 24)) return fail(FX_ERR_INVALID_ARGUMENT, "capacity out of range");
    fx_lsm_data *d = new fx_lsm_data();
    d->ctx = ctx;
    d->cap = capacity;
    if (cudaMalloc(&d->d_in, capacity * kInLen * sizeof(__nv_bfloat16)) != cudaSuccess ||
        cudaMalloc(&d->d_tgt, capacity * kTgtLen * 4) != cudaSuccess ||
        cudaMalloc(&d->d_norm, capacity * 2 * 4) != cudaSuccess) {
        (void)cudaGetLastError();
        if (d->d_in) cudaFree(d->d_in);
        if (d->d_tgt) cudaFree(d->d_tgt);
        if (d->d_norm) cudaFree(d->d_norm);
        delete d;
        return fail(FX_ERR_BACKEND, "learned smoother samples: allocation failed");
    }
    *out = d;
    return FX_OK;
}

int fx_lsm_data_destroy(fx_lsm_data *d) {
    if (!d) return FX_OK;
    cudaSetDevice(d->ctx->device);
    cudaStreamSynchronize(d->ctx->stream);
    cudaFree(d->d_in);
    cudaFree(d->d_tgt);
    cudaFree(d->d_norm);
    delete d;
    return FX_OK;
}

int fx_lsm_data_size(const fx_lsm_data *d, size_t *n) {
    if (!d || !n) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    *n = d->count;
    return FX_OK;
}

int fx_lsm_data_get(const fx_lsm_data *d, size_t index, float *inputs, float *target, float *norm) {
    if (!d || !inputs || !target || !norm) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    if (index >= d->count) return fail(FX_ERR_INVALID_ARGUMENT, "sample index out of range");
    std::vector<__nv_bfloat16> b(kInLen);
    cudaStream_t s = d->ctx->stream;
    FX_CUDA(cudaMemcpyAsync(b.data(), d->d_in + index * kInLen, kInLen * 2, cudaMemcpyDeviceToHost, s));
    FX_CUDA(cudaMemcpyAsync(target, d->d_tgt + index * kTgtLen, kTgtLen * 4, cudaMemcpyDeviceToHost, s));
    FX_CUDA(cudaMemcpyAsync(norm, d->d_norm + 2 * index, 8, cudaMemcpyDeviceToHost, s));
    FX_CUDA(cudaStreamSynchronize(s));
    for (int k = 0; k < kInLen; k++) {  // BF16 -> FP32 is exact: the high half of the word
        uint16_t u;
        std::memcpy(&u, &b[k], 2);
        const uint32_t w = (uint32_t)u << 16;
        std::memcpy(&inputs[k], &w, 4);
    }
    return FX_OK;
}

int fx_lsm_loss_grad(fx_lsm *m, const fx_lsm_data *d, const size_t *indices, size_t count, double lambda,
                     double *loss, float *grad) {
    if (!m || !d || !indices || !loss) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    if (d->ctx->device != m->ctx->device) return fail(FX_ERR_INVALID_ARGUMENT, "samples on another device");
    std::vector<int> idx(count);
    for (size_t i = 0; i < count; i++) {
        if (indices[i] >= d->count) return fail(FX_ERR_INVALID_ARGUMENT, "sample index out of range");
        idx[i] = (int)indices[i];
    }
    if (!(lambda >= 0.0)) return fail(FX_ERR_INVALID_ARGUMENT, "lambda must be non-negative");
    FX_TRY(lsm_batch_grad(m, d, idx.data(), count, (float)lambda));
    std::vector<float> g(kNParams + 1);
    FX_CUDA(cudaMemcpyAsync(g.data(), m->d_grad, (kNParams + 1) * 4, cudaMemcpyDeviceToHost, m->ctx->stream));
    FX_CUDA(cudaStreamSynchronize(m->ctx->stream));
    *loss = (double)g[kNParams] / (double)count;
    if (grad)
        for (int p = 0; p < kNParams; p++) grad[p] = g[p] / (float)count;
    return FX_OK;
}

int fx_lsm_train(fx_lsm *m, const fx_lsm_data *d, size_t epochs, size_t batch, double lr, double lambda,
                 unsigned long long seed, double *epoch_loss) {
    FX_RANGE("fx_lsm_train");
    if (!m || !d) return fail(FX_ERR_INVALID_ARGUMENT, "null argument");
    if (!(lambda >= 0.0)) return fail(FX_ERR_INVALID_ARGUMENT, "lambda must be non-negative");
    if (d->count == 0 || batch == 0) return fail(FX_ERR_INVALID_ARGUMENT, "no samples or zero batch");
    if (!(lr > 0.0)) return fail(FX_ERR_INVALID_ARGUMENT, "learning rate must be positive");
    fx_ctx *ctx = m->ctx;
    batch = std::min(batch, d->count);
    const size_t steps = d->count / batch;
    std::vector<int> order(d->count);
    for (size_t i = 0; i < d->count; i++) order[i] = (int)i;
    std::mt19937_64 rng(seed);
    // the per-step losses stay on the device until the end of each epoch
    float *d_losses = nullptr;
    FX_CUDA(cudaMallocAsync(&d_losses, steps * sizeof(float), ctx->stream));
    std::vector<float> h_losses(steps);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    int st = FX_OK;
    for (size_t e = 0; e < epochs && st == FX_OK; e++) {
        std::shuffle(order.begin(), order.end(), rng);
        for (size_t k = 0; k < steps && st == FX_OK; k++) {
            st = lsm_batch_grad(m, d, order.data() + k * batch, batch, (float)lambda);
            if (st != FX_OK) break;
            m->adam_t++;
            const float c1 = 1.f - (float)std::pow((double)b1, (double)m->adam_t);
            const float c2 = 1.f - (float)std::pow((double)b2, (double)m->adam_t);
            k_lsm_adam<<<(kNParams + 255) / 256, 256, 0, ctx->stream>>>(m->d_w, m->d_m, m->d_v, m->d_grad,
                                                                        1.f / (float)batch, (float)lr, b1, b2, eps, c1, c2);
            st = check_launch(ctx, "lsm_adam");
            if (st == FX_OK) st = m->pack();
            if (st == FX_OK && cudaMemcpyAsync(d_losses + k, m->d_grad + kNParams, 4, cudaMemcpyDeviceToDevice,
                                               ctx->stream) != cudaSuccess)
                st = fail(FX_ERR_BACKEND, "learned smoother: loss copy failed");
        }
        if (st == FX_OK && epoch_loss) {
            if (cudaMemcpyAsync(h_losses.data(), d_losses, steps * 4, cudaMemcpyDeviceToHost, ctx->stream) !=
                    cudaSuccess ||
                cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
                st = fail(FX_ERR_BACKEND, "learned smoother: loss read failed");
                break;
            }
            double s = 0.0;
            for (float v : h_losses) s += v;
            epoch_loss[e] = s / (double)(steps * batch);  // mean per-sample loss over the epoch (before each step)
        }
    }
    cudaFreeAsync(d_losses, ctx->stream);
    if (st == FX_OK) FX_CUDA(cudaStreamSynchronize(ctx->stream));
    return st;
}

}  // extern "C"
