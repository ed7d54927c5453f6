// warmstart_cnn.cu -- training and inference kernels of the warm-start
// network: a 4-level convolutional encoder/decoder that maps per-problem
// feature maps (dirty images and the gridded uv density) to a positive,
// unit-flux start image for CG.
//
// The reference has no learned component; these kernels serve the
// library's warm-start extension only. Layout: activations float NCHW
// [B][C][H][W]; 3x3 weights [Cout][Cin][3][3] as bf16 (the layer's working
// copy of an FP32 master), FP32 accumulation everywhere, FP64 for the
// per-image normalisation and loss sums. All reductions are deterministic
// (per-block partials summed in a fixed order, no floating-point atomics).
//
//   k_conv3       3x3 convolution, zero padding: bias, optional residual add,
//                 optional ReLU. With `flip` it is the data-gradient of a
//                 convolution (transposed, flipped taps; input channels =
//                 the forward's output channels), optionally accumulating.
//   k_conv3_wgrad per-slice partials of dW[co][ci][tap] and db[co]
//   k_reduce_slices  fixed-order sum of those partials
//   k_relu_mask   g *= (y > 0)
//   k_pool2 / k_pool2_bwd / k_up2 / k_up2_bwd   2x2 average pool, nearest upsample
//   k_head / k_head_bwd  1x1 conv -> softplus -> divide by the image sum
//   k_mse         per-image squared error (absolute or relative), gradient
//   k_adam        Adam step on FP32 masters, bf16 working copy
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "gpair_b200.h"

#define CV_CI 8    // input channels per shared-memory chunk
#define NTAP 9

// out[b][co][y][x] = act(bias[co] + skip + sum_ci,tap w * in[b][ci][y+dy][x+dx])
// flip: in = dL/d(out) of a forward conv with weights w[Cin][Cout][3][3]
// (here Cin/Cout are the forward's Cout/Cin), taps mirrored.
//
// A thread makes 4 pixels of a row x CT output channels: per input channel 6
// shared loads of its 3 x 6 inputs and 9 of its weights (CT contiguous values
// each, the same for every pixel group) feed 36 CT FMAs. (One pixel x 16
// channels with scalar weight loads, one load per FMA, was bound by shared
// memory: 64^2, 16 images, 16 -> 16 channels 28.5 us, 8^2, 128 -> 128 112 us;
// now 21 and 33.) Every output sums its products in the order of input channel,
// then tap. A block's tile is 4 TW4 x TH pixels and CB channels.
template <int TW4, int TH, int CB, int CT>
__global__ void __launch_bounds__(TW4 *TH *(CB / CT)) k_conv3(const float *__restrict__ in,
                                                              const __nv_bfloat16 *__restrict__ w,
                                                              const float *__restrict__ bias,
                                                              const float *__restrict__ skip, float *__restrict__ out,
                                                              int Cin, int Cout, int H, int W, int relu, int flip,
                                                              int accumulate)
{
    constexpr int TW = 4 * TW4, LD = TW + 4, NT = TW4 * TH * (CB / CT);
    __shared__ __align__(16) float xs[CV_CI][TH + 2][LD];
    __shared__ __align__(16) float ws[CV_CI][NTAP][CB];
    const int tiles_x = (W + TW - 1) / TW;
    const int tx0 = (blockIdx.x % tiles_x) * TW, ty0 = (blockIdx.x / tiles_x) * TH;
    const int co0 = blockIdx.y * CB, b = blockIdx.z;
    const int gx = threadIdx.x % TW4, gy = (threadIdx.x / TW4) % TH, og = threadIdx.x / (TW4 * TH);
    const float *inb = in + (size_t)b * Cin * H * W;
    float acc[CT][4];
#pragma unroll
    for (int o = 0; o < CT; o++)
#pragma unroll
        for (int p = 0; p < 4; p++) acc[o][p] = 0.f;
    // the next chunk's inputs and weights wait in registers while this one is computed
    constexpr int XT = CV_CI * (TH + 2) * (TW + 2), XR = (XT + NT - 1) / NT, WT = CB * CV_CI * NTAP, WR = (WT + NT - 1) / NT;
    float xr[XR];
    __nv_bfloat16 wr[WR];
    auto load = [&](int ci0) {
        // input tile with a one-pixel halo, zero outside the image
#pragma unroll
        for (int j = 0; j < XR; j++) {
            const int i = j * NT + threadIdx.x;
            const int c = i / ((TH + 2) * (TW + 2)), r = i % ((TH + 2) * (TW + 2));
            const int yy = ty0 - 1 + r / (TW + 2), xx = tx0 - 1 + r % (TW + 2);
            const bool ok = i < XT && ci0 + c < Cin && yy >= 0 && yy < H && xx >= 0 && xx < W;
            xr[j] = ok ? __ldg(&inb[((size_t)(ci0 + c) * H + yy) * W + xx]) : 0.f;
        }
        // weights in their memory order: [co][ci][tap], or [ci][co][tap] of the mirrored layer
#pragma unroll
        for (int j = 0; j < WR; j++) {
            const int i = j * NT + threadIdx.x;
            const int o = flip ? (i / NTAP) % CB : i / (CV_CI * NTAP), c = flip ? i / (CB * NTAP) : (i / NTAP) % CV_CI;
            const int k = i % NTAP;
            const bool ok = i < WT && co0 + o < Cout && ci0 + c < Cin;
            const size_t at = flip ? ((size_t)(ci0 + c) * Cout + co0 + o) * NTAP + k
                                   : ((size_t)(co0 + o) * Cin + ci0 + c) * NTAP + k;
            wr[j] = ok ? w[at] : __float2bfloat16_rn(0.f);
        }
    };
    load(0);
    for (int ci0 = 0; ci0 < Cin; ci0 += CV_CI) {
        const int nc = min(CV_CI, Cin - ci0);
#pragma unroll
        for (int j = 0; j < XR; j++) {
            const int i = j * NT + threadIdx.x;
            const int c = i / ((TH + 2) * (TW + 2)), r = i % ((TH + 2) * (TW + 2));
            if (i < XT) xs[c][r / (TW + 2)][r % (TW + 2)] = xr[j];
        }
#pragma unroll
        for (int j = 0; j < WR; j++) {
            const int i = j * NT + threadIdx.x;
            const int o = flip ? (i / NTAP) % CB : i / (CV_CI * NTAP), c = flip ? i / (CB * NTAP) : (i / NTAP) % CV_CI;
            const int k = flip ? NTAP - 1 - i % NTAP : i % NTAP;
            if (i < WT) ws[c][k][o] = __bfloat162float(wr[j]);
        }
        __syncthreads();
        if (ci0 + CV_CI < Cin) load(ci0 + CV_CI);
#pragma unroll(CT <= 2 ? 4 : 1)
        for (int c = 0; c < nc; c++) {
            float v[3][6];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float *row = &xs[c][gy + r][4 * gx];
                *reinterpret_cast<float4 *>(&v[r][0]) = *reinterpret_cast<const float4 *>(row);
                *reinterpret_cast<float2 *>(&v[r][4]) = *reinterpret_cast<const float2 *>(row + 4);
            }
#pragma unroll
            for (int k = 0; k < NTAP; k++) {
                float wk[CT];
#pragma unroll
                for (int o = 0; o < CT; o += (CT < 4 ? CT : 4)) {
                    if constexpr (CT >= 4)
                        *reinterpret_cast<float4 *>(&wk[o]) = *reinterpret_cast<const float4 *>(&ws[c][k][og * CT + o]);
                    else if constexpr (CT >= 2)
                        *reinterpret_cast<float2 *>(&wk[o]) = *reinterpret_cast<const float2 *>(&ws[c][k][og * CT + o]);
                    else
                        wk[o] = ws[c][k][og];
                }
#pragma unroll
                for (int o = 0; o < CT; o++)
#pragma unroll
                    for (int p = 0; p < 4; p++) acc[o][p] = fmaf(wk[o], v[k / 3][k % 3 + p], acc[o][p]);
            }
        }
        __syncthreads();
    }
    const int x0 = tx0 + 4 * gx, y = ty0 + gy;
    if (x0 >= W || y >= H) return;
    // rows of whole float4s, from 16-byte aligned arrays
    const bool vec = (W & 3) == 0 && ((((uintptr_t)out) | ((uintptr_t)skip)) & 15) == 0;
#pragma unroll
    for (int o = 0; o < CT; o++) {
        const int co = co0 + og * CT + o;
        if (co >= Cout) break;
        const size_t idx = (((size_t)b * Cout + co) * H + y) * W + x0;
        const float bv = bias ? bias[co] : 0.f;
        float v[4], s[4] = {0.f, 0.f, 0.f, 0.f}, prev[4] = {0.f, 0.f, 0.f, 0.f};
        if (vec) {
            if (skip) *reinterpret_cast<float4 *>(s) = *reinterpret_cast<const float4 *>(skip + idx);
            if (accumulate) *reinterpret_cast<float4 *>(prev) = *reinterpret_cast<const float4 *>(out + idx);
        } else {
#pragma unroll
            for (int p = 0; p < 4; p++)
                if (x0 + p < W) {
                    if (skip) s[p] = skip[idx + p];
                    if (accumulate) prev[p] = out[idx + p];
                }
        }
#pragma unroll
        for (int p = 0; p < 4; p++) {
            v[p] = acc[o][p] + bv;
            if (skip) v[p] += s[p];
            if (relu) v[p] = fmaxf(v[p], 0.f);
            if (accumulate) v[p] = prev[p] + v[p];
        }
        if (vec) {
            *reinterpret_cast<float4 *>(out + idx) = *reinterpret_cast<const float4 *>(v);
        } else {
#pragma unroll
            for (int p = 0; p < 4; p++)
                if (x0 + p < W) out[idx + p] = v[p];
        }
    }
}

// Weight and bias gradient partials: block (NG groups of CO output channels, input
// channel, slice) sums over the images [slice*bps, (slice+1)*bps) and all pixels;
// part[slice][co][ci][tap], bpart[slice][co] (bias, from the blocks of the first
// input channel). Thread t of a group sums the pixels p = t mod 256 in order, image by
// image; the threads' sums go through a shuffle tree and then over the warps
// in order. The input passes through shared memory with its zero border, a chunk of
// whole images or of 256 nstep pixels of one image at a time, the next chunk's copies
// in flight: a pixel is then 9 shared loads and CO loads of g, also ahead, for 9 CO
// FMAs. Masked pixels (g = 0) add nothing and taps outside the image are left out,
// also beside infinities: the products are formed regardless, and a block whose sums
// come out non-finite forms them again pixel by pixel (wg_careful). (With
// the inputs loaded per pixel and every mask applied, 90 instructions went to 9
// FMAs: 16 images of 64^2, 16 -> 16 channels 68 us, now 51; 8^2, 128 -> 128
// 41, now 35.)
#define WG_THREADS 256
#define WG_BUF 5120  // floats of a chunk
struct WgPlan {
    int threads, nimg, nstep;  // threads per group; images per chunk, or steps of 256 pixels of one image
    int ld, xo;                // floats per row of a chunk, offset of a row's first pixel
    int vec, wshift;           // 16-byte copies, of which a row takes 1 << wshift
};
// false: a chunk of one step does not fit
static bool wg_plan(const float *in, int B, int H, int W, WgPlan *p)
{
    const int HW = H * W;
    p->vec = W >= 4 && (W & (W - 1)) == 0 && ((uintptr_t)in & 15) == 0;
    p->wshift = 0;
    while (p->vec && 4 << p->wshift < W) p->wshift++;
    p->xo = p->vec ? 4 : 1;
    p->ld = W + 2 * p->xo;
    p->threads = HW >= WG_THREADS ? WG_THREADS : (HW + 31) / 32 * 32;
    p->nstep = (HW + WG_THREADS - 1) / WG_THREADS;
    p->nimg = (long long)(H + 2) * p->ld <= WG_BUF ? WG_BUF / ((H + 2) * p->ld) : 0;
    if (p->nimg) {
        if (p->nimg > B) p->nimg = B;
        return true;
    }
    p->nimg = 1;
    // the rows that 256 nstep consecutive pixels touch, one above and one below
    int n = (int)((long long)(WG_BUF / p->ld - 3) * W / WG_THREADS);
    if (n > p->nstep) n = p->nstep;
    p->nstep = n;
    return n >= 1;
}

// the sums of one thread pixel by pixel: acc [co][tap], then the bias sums
template <int CO>
__device__ __noinline__ void wg_careful(const float *__restrict__ in, const float *__restrict__ g, int b0, int b1, int ci,
                                        int co0, int Cin, int Cout, int H, int W, int t, float *acc)
{
    const int HW = H * W;
    for (int i = 0; i < CO * NTAP + CO; i++) acc[i] = 0.f;
    for (int b = b0; b < b1; b++)
        for (int p = t; p < HW; p += WG_THREADS) {
            const int y = p / W, x = p - y * W;
            const float *ip = in + ((size_t)b * Cin + ci) * HW + p;
            for (int o = 0; o < CO && co0 + o < Cout; o++) {
                const float gv = g[((size_t)b * Cout + co0 + o) * HW + p];
                if (gv == 0.f) continue;
                acc[CO * NTAP + o] += gv;
                for (int k = 0; k < NTAP; k++) {
                    const int dy = k / 3 - 1, dx = k % 3 - 1;
                    if (y + dy < 0 || y + dy >= H || x + dx < 0 || x + dx >= W) continue;
                    acc[o * NTAP + k] = fmaf(gv, ip[dy * W + dx], acc[o * NTAP + k]);
                }
            }
        }
}

// Sums of N values (at most 32) over the lanes of a warp, into out[0..N-1]: at every level of
// the tree half of the lanes go on with half of the values. The pairs are those of a shuffle tree per value, so
// the sums are the same; 4 instructions a pair instead of 10 a value.
template <int N>
__device__ __forceinline__ void wg_warp_sums(const float *acc, int lane, float *out)
{
    constexpr int M = N > 16 ? 32 : N > 8 ? 16 : N > 4 ? 8 : N > 2 ? 4 : N;  // a power of two
    float v[M];
#pragma unroll
    for (int i = 0; i < M; i++) v[i] = i < N ? acc[i] : 0.f;
    int idx = 0, off = 16;
#pragma unroll
    for (int m = M; off > 0; off >>= 1) {
        if (m > 1) {
            m >>= 1;
            const bool hi = lane & off;
#pragma unroll
            for (int i = 0; i < M / 2; i++)
                if (i < m) {
                    const float keep = hi ? v[i + m] : v[i], send = hi ? v[i] : v[i + m];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            if (hi) idx += m;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
        }
    }
    if (idx < N && (lane & (32 / M - 1)) == 0) out[idx] = v[0];
}

// How a thread steps through a chunk: from row to row (any width), by a fixed stride (the width divides
// 256), or from image to image (an image is one step). WG_WIDE: images of which no chunk of 256
// pixels fits (W > 1,278), pixel by pixel.
enum { WG_ROWS, WG_FIXED, WG_IMAGES, WG_WIDE };
template <int CO, int NG, int U, int MODE>
__global__ void __launch_bounds__(WG_THREADS *NG) k_conv3_wgrad(const float *__restrict__ in,
                                                                const float *__restrict__ g,
                                                                float *__restrict__ part, float *__restrict__ bpart,
                                                                int B, int Cin, int Cout, int H, int W, int bps,
                                                                const WgPlan P)
{
    constexpr int NV = CO * NTAP + CO;
    constexpr bool STAGED = MODE != WG_WIDE;
    __shared__ __align__(16) float xs[STAGED ? 2 : 1][STAGED ? WG_BUF : 4];
    __shared__ float red[NG][WG_THREADS / 32][NV];
    const int t = threadIdx.x % P.threads, grp = threadIdx.x / P.threads;
    const int co0 = (blockIdx.x * NG + grp) * CO, ci = blockIdx.y, slice = blockIdx.z;
    const int b0 = slice * bps, b1 = min(B, b0 + bps);
    const int HW = H * W, LD = P.ld;
    const int lane = threadIdx.x & 31;
    float acc[NV];  // [co][tap], then the bias sums
#pragma unroll
    for (int i = 0; i < NV; i++) acc[i] = 0.f;
    if (STAGED) {
        const int total_steps = (HW + WG_THREADS - 1) / WG_THREADS;
        const bool whole = P.nstep == total_steps;
        const int spi = whole ? 1 : (total_steps + P.nstep - 1) / P.nstep;  // chunks per image
        const int nchunk = whole ? (b1 - b0 + P.nimg - 1) / P.nimg : (b1 - b0) * spi;
        // the borders stay zero
        const int used = whole ? P.nimg * (H + 2) * LD : WG_BUF, nbuf = nchunk > 1 ? 2 : 1;
        for (int b = 0; b < nbuf; b++)
            for (int i = threadIdx.x; i < (used + 3) / 4; i += blockDim.x)
                reinterpret_cast<float4 *>(xs[b])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        // chunk c: images [ib, ib + ni), steps [s0, s1) of each, rows from ylo
        auto range = [&](int c, int &ib, int &ni, int &s0, int &s1, int &ylo, int &rows) {
            if (whole) {
                ib = b0 + c * P.nimg;
                ni = min(P.nimg, b1 - ib);
                s0 = 0;
                s1 = total_steps;
                ylo = -1;
                rows = H + 2;
            } else {
                ib = b0 + c / spi;
                ni = 1;
                s0 = (c % spi) * P.nstep;
                s1 = min(total_steps, s0 + P.nstep);
                ylo = WG_THREADS * s0 / W - 1;
                rows = (min(HW, WG_THREADS * s1) - 1) / W + 1 - ylo + 1;
            }
        };
        // the rows of chunk c (zeros for those outside the image), 16 bytes or one pixel a copy
        auto stage = [&](int c) {
            int ib, ni, s0, s1, ylo, rows;
            range(c, ib, ni, s0, s1, ylo, rows);
            const uint32_t buf = (uint32_t)__cvta_generic_to_shared(&xs[c & 1][P.xo]);
            const float *src = in + ((size_t)ib * Cin + ci) * HW;
            const int lo = whole ? 1 : 0, nr = whole ? H : rows;  // of whole images the border rows stay zero
            for (int im = 0; im < ni; im++, src += (size_t)Cin * HW) {
                const uint32_t dst = buf + 4u * (uint32_t)(im * rows * LD);
                if (P.vec) {
                    for (int e = threadIdx.x; e < nr << P.wshift; e += blockDim.x) {
                        const int r = lo + (e >> P.wshift), x = 4 * (e & ((1 << P.wshift) - 1)), y = ylo + r;
                        const bool ok = y >= 0 && y < H;
                        const int bytes = ok ? 16 : 0;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 4u * (uint32_t)(r * LD + x)),
                                     "l"(ok ? src + (size_t)y * W + x : src), "r"(bytes)
                                     : "memory");
                    }
                } else {
                    for (int e = threadIdx.x; e < nr * W; e += blockDim.x) {
                        const int q = e / W, r = lo + q, x = e - q * W, y = ylo + r;
                        const bool ok = y >= 0 && y < H;
                        const int bytes = ok ? 4 : 0;
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4u * (uint32_t)(r * LD + x)),
                                     "l"(ok ? src + (size_t)y * W + x : src), "r"(bytes)
                                     : "memory");
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        const int dy = WG_THREADS / W, dx = WG_THREADS - dy * W;
        stage(0);
        for (int c = 0; c < nchunk; c++) {
            if (c + 1 < nchunk) {
                stage(c + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            int ib, ni, s0, s1, ylo, rows;
            range(c, ib, ni, s0, s1, ylo, rows);
            // this thread's pixels of the chunk: `per` of each image from pixel t + 256 s0
            const int p0 = t + WG_THREADS * s0;
            const int per = p0 < HW ? min(s1 - s0, (HW - p0 + WG_THREADS - 1) / WG_THREADS) : 0;
            const int y0 = p0 / W, x0 = p0 - y0 * W;
            const int n = MODE == WG_IMAGES ? per * ni : per, outer = MODE == WG_IMAGES ? 1 : ni;
            const int gs = MODE == WG_IMAGES ? Cout * HW : WG_THREADS;
            const int os = MODE == WG_IMAGES ? rows * LD : dy * LD + dx;
            for (int im = 0; im < outer; im++) {
                const float *gp = g + (size_t)(ib + im) * Cout * HW + p0;
                const float *bp = &xs[c & 1][im * rows * LD + (y0 - ylo) * LD + x0 + P.xo];
                const float *gc[CO];  // (channels past the last repeat it; their sums are not stored)
#pragma unroll
                for (int o = 0; o < CO; o++) gc[o] = gp + (size_t)min(co0 + o, Cout - 1) * HW;
                int x = x0;
                float gn[U][CO];
                // g of the next k pixels
                auto fetch = [&](int k) {
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (u < k) {
#pragma unroll
                            for (int o = 0; o < CO; o++) gn[u][o] = __ldg(gc[o] + u * gs);
                        }
#pragma unroll
                    for (int o = 0; o < CO; o++) gc[o] += U * gs;
                };
                // the sums of k pixels, g of the kn after them in flight
                auto run = [&](int k, int kn) {
                    float gv[U][CO], v[U][NTAP];
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (u < k) {
#pragma unroll
                            for (int o = 0; o < CO; o++) gv[u][o] = gn[u][o];
                            const float *q = MODE == WG_ROWS ? bp : bp + u * os;
#pragma unroll
                            for (int t9 = 0; t9 < NTAP; t9++) v[u][t9] = q[(t9 / 3 - 1) * LD + t9 % 3 - 1];
                            if (MODE == WG_ROWS) {
                                bp += os;
                                x += dx;
                                if (x >= W) {
                                    x -= W;
                                    bp += LD - W;
                                }
                            }
                        }
                    if (MODE != WG_ROWS) bp += U * os;
                    fetch(kn);
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (u < k) {
#pragma unroll
                            for (int o = 0; o < CO; o++) {
                                acc[CO * NTAP + o] += gv[u][o];
#pragma unroll
                                for (int t9 = 0; t9 < NTAP; t9++)
                                    acc[o * NTAP + t9] = fmaf(gv[u][o], v[u][t9], acc[o * NTAP + t9]);
                            }
                        }
                };
                int left = n;
                fetch(min(left, U));
                for (; left >= 2 * U; left -= U) run(U, U);
                for (; left > 0; left -= U) run(min(left, U), min(max(left - U, 0), U));
            }
            __syncthreads();  // the chunk after the next takes this buffer
        }
    }
    bool redo = !STAGED;
#pragma unroll
    for (int i = 0; i < NV; i++) redo |= !(fabsf(acc[i]) <= 3.402823466e38f);
    if (__syncthreads_or(redo)) {
        float again[NV];
        wg_careful<CO>(in, g, b0, b1, ci, co0, Cin, Cout, H, W, t, again);
#pragma unroll
        for (int i = 0; i < NV; i++) acc[i] = again[i];
    }
    // fixed-order block reduction: warp shuffles, then one pass over the group's warps
    const int gw = P.threads >> 5;
#pragma unroll
    for (int i = 0; i < NV; i += 32) {
        if constexpr (NV <= 32) wg_warp_sums<NV>(&acc[i], lane, &red[grp][t >> 5][i]);
        else if (i + 32 <= NV) wg_warp_sums<32>(&acc[i], lane, &red[grp][t >> 5][i]);
        else wg_warp_sums<NV % 32 ? NV % 32 : 32>(&acc[i], lane, &red[grp][t >> 5][i]);
    }
    __syncthreads();
    for (int i = t; i < NV; i += P.threads) {
        float v = 0.f;
        for (int w = 0; w < gw; w++) v += red[grp][w][i];
        if (i < CO * NTAP) {
            const int co = co0 + i / NTAP, k = i % NTAP;
            if (co < Cout) part[(((size_t)slice * Cout + co) * Cin + ci) * NTAP + k] = v;
        } else if (blockIdx.y == 0) {
            const int co = co0 + i - CO * NTAP;
            if (co < Cout) bpart[(size_t)slice * Cout + co] = v;
        }
    }
}

// out[i] = sum over slices of part[s][i] (fixed order)
__global__ void k_reduce_slices(const float *__restrict__ part, int n, int slices, float *__restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.f;
    for (int k = 0; k < slices; k++) s += part[(size_t)k * n + i];
    out[i] = s;
}

// The same for a weight gradient (nw values) and its bias gradient (nb) in one launch
__global__ void k_reduce_wgrad(const float *__restrict__ part, int nw, const float *__restrict__ bpart, int nb,
                               int slices, float *__restrict__ dw, float *__restrict__ db)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nw + nb) return;
    const float *p = i < nw ? part + i : bpart + (i - nw);
    const size_t ld = i < nw ? nw : nb;
    float s = 0.f;
    for (int k = 0; k < slices; k++) s += __ldg(p + (size_t)k * ld);
    if (i < nw) dw[i] = s;
    else db[i - nw] = s;
}

__global__ void k_relu_mask(const float *__restrict__ y, float *__restrict__ g, long long n)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(y[i] > 0.f)) g[i] = 0.f;
}

// 2x2 average pool: in [BC][H][W] -> out [BC][H/2][W/2]
__global__ void k_pool2(const float *__restrict__ in, float *__restrict__ out, long long BC, int H, int W)
{
    const int Ho = H / 2, Wo = W / 2;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= BC * Ho * Wo) return;
    const long long bc = i / (Ho * Wo);
    const int r = (int)(i % (Ho * Wo)), y = r / Wo, x = r % Wo;
    const float *p = in + (size_t)bc * H * W + (size_t)(2 * y) * W + 2 * x;
    out[i] = 0.25f * ((p[0] + p[1]) + (p[W] + p[W + 1]));
}

__global__ void k_pool2_bwd(const float *__restrict__ gout, float *__restrict__ gin, long long BC, int H, int W,
                            int accumulate)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= BC * H * W) return;
    const long long bc = i / (H * W);
    const int r = (int)(i % (H * W)), y = r / W, x = r % W;
    const float v = 0.25f * gout[(size_t)bc * (H / 2) * (W / 2) + (y / 2) * (W / 2) + x / 2];
    gin[i] = accumulate ? gin[i] + v : v;
}

// nearest 2x upsample: in [BC][H][W] -> out [BC][2H][2W]
__global__ void k_up2(const float *__restrict__ in, float *__restrict__ out, long long BC, int H, int W)
{
    const int Ho = 2 * H, Wo = 2 * W;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= BC * Ho * Wo) return;
    const long long bc = i / (Ho * Wo);
    const int r = (int)(i % (Ho * Wo)), y = r / Wo, x = r % Wo;
    out[i] = in[(size_t)bc * H * W + (y / 2) * W + x / 2];
}

__global__ void k_up2_bwd(const float *__restrict__ gout, float *__restrict__ gin, long long BC, int H, int W)
{
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= BC * H * W) return;
    const long long bc = i / (H * W);
    const int r = (int)(i % (H * W)), y = r / W, x = r % W;
    const float *p = gout + (size_t)bc * 4 * H * W + (size_t)(2 * y) * (2 * W) + 2 * x;
    gin[i] = (p[0] + p[1]) + (p[2 * W] + p[2 * W + 1]);
}

__device__ __forceinline__ float softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
__device__ __forceinline__ float sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

// The per-image kernels below run on a cluster of HD_CTAS blocks per image, each
// with a contiguous share of its pixels; an image's FP64 sums go over the
// blocks' shared memory in rank order. (One block per image left all but B of
// the SMs idle: head, its backward and the loss took 100, 169 and 18 us for 16
// images of 64^2, the head 366 us for one of 128^2.)
#define HD_CTAS 8

// Sum of NV values over the cluster, the same in every thread. sm: NV * 33 doubles, not in use by any other call
template <int NV>
__device__ void cluster_sum_d(double (&v)[NV], double *sm)
{
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; i++) {
        for (int off = 16; off > 0; off >>= 1) v[i] += __shfl_down_sync(0xffffffffu, v[i], off);
        if (lane == 0) sm[i * 33 + warp] = v[i];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NV; i += blockDim.x) {
        double t = 0.0;
        for (int w = 0; w < nw; w++) t += sm[i * 33 + w];
        sm[i * 33 + 32] = t;
    }
    cl.sync();  // every block's sums are in its shared memory
#pragma unroll
    for (int i = 0; i < NV; i++) {
        double t = 0.0;
        for (int r = 0; r < HD_CTAS; r++) t += *cl.map_shared_rank(&sm[i * 33 + 32], r);
        v[i] = t;
    }
    cl.sync();  // read by every block before it is reused or the block ends
}

// this block's share [p0, p1) of an image's HW pixels
__device__ __forceinline__ void head_share(int HW, int &b, int &p0, int &p1)
{
    b = blockIdx.x / HD_CTAS;
    const int r = blockIdx.x % HD_CTAS, per = (HW + HD_CTAS - 1) / HD_CTAS;
    p0 = min(HW, r * per);
    p1 = min(HW, p0 + per);
}

// Head: z = w . d + bias, a = softplus(z), out = a / sum(a)
__global__ void __cluster_dims__(HD_CTAS, 1, 1) __launch_bounds__(256)
    k_head(const float *__restrict__ d, const float *__restrict__ w, const float *__restrict__ bias_p,
           float *__restrict__ z, float *__restrict__ out, float *__restrict__ asum, int C, int HW)
{
    __shared__ double sm[33];
    int b, p0, p1;
    head_share(HW, b, p0, p1);
    const float bias = *bias_p;
    const float *db = d + (size_t)b * C * HW;
    double s[1] = {0.0};
    for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
        float v = bias;
#pragma unroll 8
        for (int c = 0; c < C; c++) v = fmaf(w[c], __ldg(&db[(size_t)c * HW + p]), v);
        z[(size_t)b * HW + p] = v;
        s[0] += (double)softplus(v);
    }
    cluster_sum_d(s, sm);
    const float inv = (float)(1.0 / s[0]);
    for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x)
        out[(size_t)b * HW + p] = softplus(z[(size_t)b * HW + p]) * inv;
    if (blockIdx.x % HD_CTAS == 0 && threadIdx.x == 0) asum[b] = (float)s[0];
}

// Head backward: gz = ((gout - <gout, out>) / S) sigmoid(z), gd[b][c][p] = w[c] gz, and
// per-image partials of dw[c] (c < C) and dbias (c = C), HB_C channels a pass
#define HB_C 16
__global__ void __cluster_dims__(HD_CTAS, 1, 1) __launch_bounds__(256)
    k_head_bwd(const float *__restrict__ d, const float *__restrict__ w, const float *__restrict__ z,
               const float *__restrict__ out, const float *__restrict__ asum, const float *__restrict__ gout,
               float *__restrict__ gd, float *__restrict__ part, int C, int HW)
{
    __shared__ double sm[(HB_C + 1) * 33];
    int b, p0, p1;
    head_share(HW, b, p0, p1);
    const size_t o = (size_t)b * HW;
    double dot[1] = {0.0};
    for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) dot[0] += (double)gout[o + p] * out[o + p];
    cluster_sum_d(dot, sm);
    const float invS = 1.f / asum[b], fd = (float)dot[0];
    const float *db = d + (size_t)b * C * HW;
    float *gdb = gd + (size_t)b * C * HW;
    for (int c0 = 0; c0 < C; c0 += HB_C) {
        double s[HB_C + 1];
#pragma unroll
        for (int c = 0; c <= HB_C; c++) s[c] = 0.0;
        for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
            const float gz = (gout[o + p] - fd) * invS * sigmoid(z[o + p]);
#pragma unroll
            for (int c = 0; c < HB_C; c++)
                if (c0 + c < C) {
                    s[c] += (double)gz * __ldg(&db[(size_t)(c0 + c) * HW + p]);
                    gdb[(size_t)(c0 + c) * HW + p] = w[c0 + c] * gz;
                }
            s[HB_C] += gz;
        }
        cluster_sum_d(s, sm);
        if (blockIdx.x % HD_CTAS == 0 && threadIdx.x == 0) {
#pragma unroll
            for (int c = 0; c < HB_C; c++)
                if (c0 + c < C) part[(size_t)b * (C + 1) + c0 + c] = (float)s[c];
            if (c0 == 0) part[(size_t)b * (C + 1) + C] = (float)s[HB_C];
        }
    }
}

// Per-image loss and its gradient (x gscale), FP64 sums:
//   mode 0: npix * sum_p (out - t)^2                 g = 2 npix (out - t)
//   mode 1: sum_p (out - t)^2 / sum_p t^2 (relative)  g = 2 (out - t) / sum_p t^2
__global__ void __cluster_dims__(HD_CTAS, 1, 1) __launch_bounds__(256)
    k_mse(const float *__restrict__ out, const float *__restrict__ t, float *__restrict__ g,
          double *__restrict__ loss, int HW, float gscale, int mode)
{
    __shared__ double sm[2 * 33];
    int b, p0, p1;
    head_share(HW, b, p0, p1);
    const size_t o = (size_t)b * HW;
    double s[2] = {0.0, 0.0};  // sum (out - t)^2, sum t^2
    for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) {
        const float e = out[o + p] - t[o + p];
        s[0] += (double)e * e;
        s[1] += (double)t[o + p] * t[o + p];
    }
    cluster_sum_d(s, sm);
    const double tt = mode == 1 && s[1] > 0.0 ? s[1] : 1.0;
    const float f = mode == 1 ? (float)(2.0 / tt) : 2.f * (float)HW;
    if (g)
        for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) g[o + p] = gscale * f * (out[o + p] - t[o + p]);
    if (blockIdx.x % HD_CTAS == 0 && threadIdx.x == 0) loss[b] = mode == 1 ? s[0] / tt : s[0] * HW;
}

__global__ void k_adam(float *__restrict__ p, __nv_bfloat16 *__restrict__ pbf, const float *__restrict__ g,
                       float *__restrict__ m, float *__restrict__ v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    if (pbf) pbf[i] = __float2bfloat16_rn(pi);
}

__global__ void k_to_bf16(const float *__restrict__ src, __nv_bfloat16 *__restrict__ dst, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

// ------------------------------------------------------------ C ABI

static inline int cdiv_ll(long long a, long long b) { return (int)((a + b - 1) / b); }
static inline int cnn_status(void) { return cudaGetLastError() == cudaSuccess ? GPAIR_OK : GPAIR_ERR_CUDA; }
#define CNN_STREAM(s) ((cudaStream_t)(s))

template <int TW4, int TH, int CB, int CT>
static long long conv3_blocks(int B, int Cout, int H, int W)
{
    return (long long)B * cdiv_ll(W, 4 * TW4) * cdiv_ll(H, TH) * cdiv_ll(Cout, CB);
}

template <int TW4, int TH, int CB, int CT, typename... A>
static void conv3_go(int B, int Cout, int H, int W, cudaStream_t st, A... a)
{
    const dim3 g(cdiv_ll(W, 4 * TW4) * cdiv_ll(H, TH), cdiv_ll(Cout, CB), B);
    k_conv3<TW4, TH, CB, CT><<<g, TW4 * TH * (CB / CT), 0, st>>>(a...);
}

// The widest tile whose blocks still give every SM two: a wider tile reads less
// halo and more outputs share a thread's loads, but one image of a small level
// has few tiles, and its chain of Cin x 9 FMAs per output then runs on few SMs. The
// smallest tile gives a thread one channel, for a second warp beside the chain (the six such
// layers of one 128^2 image: 187 us with two channels, 138 with one). On the wider tiles
// fewer channels per thread were slower (4 -> 2: 298 -> 334 us, 2 -> 1: 268 -> 347 of a training step), and
// so was the smallest tile up to twice its blocks (304 -> 343).
static void conv3_launch(const float *in, const __nv_bfloat16 *w, const float *bias, const float *skip, float *out,
                         int B, int Cin, int Cout, int H, int W, int relu, int flip, int accumulate, cudaStream_t st)
{
    const long long want = 2 * 148;
    if (conv3_blocks<8, 8, 16, 8>(B, Cout, H, W) >= want)
        conv3_go<8, 8, 16, 8>(B, Cout, H, W, st, in, w, bias, skip, out, Cin, Cout, H, W, relu, flip, accumulate);
    else if (W > 8 && conv3_blocks<4, 8, 16, 4>(B, Cout, H, W) >= want / 2)
        conv3_go<4, 8, 16, 4>(B, Cout, H, W, st, in, w, bias, skip, out, Cin, Cout, H, W, relu, flip, accumulate);
    else if (conv3_blocks<2, 8, 16, 2>(B, Cout, H, W) >= want / 4)
        conv3_go<2, 8, 16, 2>(B, Cout, H, W, st, in, w, bias, skip, out, Cin, Cout, H, W, relu, flip, accumulate);
    else
        conv3_go<2, 4, 8, 1>(B, Cout, H, W, st, in, w, bias, skip, out, Cin, Cout, H, W, relu, flip, accumulate);
}

extern "C" int gpair_cnn_conv3x3(const float *in, const void *w_bf16, const float *bias, const float *skip, float *out,
                                 int B, int Cin, int Cout, int H, int W, int relu, void *stream)
{
    if (B <= 0 || B > 65535 || Cin <= 0 || Cout <= 0 || H <= 0 || W <= 0) return GPAIR_ERR_INVALID;
    conv3_launch(in, (const __nv_bfloat16 *)w_bf16, bias, skip, out, B, Cin, Cout, H, W, relu, 0, 0, CNN_STREAM(stream));
    return cnn_status();
}

extern "C" int gpair_cnn_conv3x3_bwd_data(const float *gout, const void *w_bf16, float *gin, int B, int Cin, int Cout,
                                          int H, int W, int accumulate, void *stream)
{
    if (B <= 0 || B > 65535 || Cin <= 0 || Cout <= 0 || H <= 0 || W <= 0) return GPAIR_ERR_INVALID;
    conv3_launch(gout, (const __nv_bfloat16 *)w_bf16, nullptr, nullptr, gin, B, Cout, Cin, H, W, 0, 1, accumulate,
                 CNN_STREAM(stream));
    return cnn_status();
}

extern "C" int gpair_cnn_conv3x3_bwd_weight(const float *in, const float *gpre, float *dw, float *db, float *scratch,
                                            long long scratch_floats, int B, int Cin, int Cout, int H, int W,
                                            void *stream)
{
    if (B <= 0 || Cin <= 0 || Cout <= 0 || H <= 0 || W <= 0) return GPAIR_ERR_INVALID;
    // about 64K pixels per slice
    int bps = (int)(65536 / ((long long)H * W));
    if (bps < 1) bps = 1;
    if (bps > B) bps = B;
    const int slices = cdiv_ll(B, bps);
    const long long nw = (long long)Cout * Cin * NTAP;
    if ((long long)slices * (nw + Cout) > scratch_floats) return GPAIR_ERR_INVALID;
    float *part = scratch, *bpart = scratch + (size_t)slices * nw;
    const cudaStream_t st = CNN_STREAM(stream);
    const long long blocks = (long long)Cout * Cin * slices;
    WgPlan p;
    const bool staged = wg_plan(in, B, H, W, &p);
    auto go = [&](auto kernel, int co, int ng) {
        // at most 65,535 input channels a launch (the grid's second dimension); each writes the same bias sums. (Both
        // channels on the first dimension: 100 -> 122 registers and a training step 1 % slower.)
        for (int c = 0; c < Cin; c += 65535)
            kernel<<<dim3(cdiv_ll(Cout, co * ng), Cin - c < 65535 ? Cin - c : 65535, slices), p.threads * ng, 0, st>>>(
                in + (size_t)c * H * W, gpre, part + (size_t)c * NTAP, bpart, B, Cin, Cout, H, W, bps, p);
    };
    // four output channels a block (9 input loads for 36 FMAs) where that still makes two blocks per SM; one
    // each in two groups that share a chunk where blocks are few
#define WG_GO(CO, NG, U)                                                                      \
    do {                                                                                      \
        if (H * W <= WG_THREADS) go(k_conv3_wgrad<CO, NG, U, WG_IMAGES>, CO, NG);             \
        else if (WG_THREADS % W == 0) go(k_conv3_wgrad<CO, NG, U, WG_FIXED>, CO, NG);         \
        else go(k_conv3_wgrad<CO, NG, U, WG_ROWS>, CO, NG);                                   \
    } while (0)
    if (!staged) go(k_conv3_wgrad<1, 1, 1, WG_WIDE>, 1, 1);
    else if (blocks >= 4 * 2 * 148) WG_GO(4, 1, 2);
    else if (blocks >= 2 * 2 * 148) WG_GO(2, 1, 4);
    else if (blocks >= 148) WG_GO(1, 2, 4);
    else WG_GO(1, 1, 4);
#undef WG_GO
    k_reduce_wgrad<<<cdiv_ll(nw + Cout, 256), 256, 0, st>>>(part, (int)nw, bpart, Cout, slices, dw, db);
    return cnn_status();
}

extern "C" int gpair_cnn_relu_mask(const float *y, float *g, long long n, void *stream)
{
    if (n <= 0) return GPAIR_ERR_INVALID;
    k_relu_mask<<<cdiv_ll(n, 256), 256, 0, CNN_STREAM(stream)>>>(y, g, n);
    return cnn_status();
}

extern "C" int gpair_cnn_pool2(const float *in, float *out, long long BC, int H, int W, void *stream)
{
    if (BC <= 0 || H < 2 || W < 2 || (H & 1) || (W & 1)) return GPAIR_ERR_INVALID;
    k_pool2<<<cdiv_ll(BC * (H / 2) * (W / 2), 256), 256, 0, CNN_STREAM(stream)>>>(in, out, BC, H, W);
    return cnn_status();
}

extern "C" int gpair_cnn_pool2_bwd(const float *gout, float *gin, long long BC, int H, int W, int accumulate,
                                   void *stream)
{
    if (BC <= 0 || H < 2 || W < 2 || (H & 1) || (W & 1)) return GPAIR_ERR_INVALID;
    k_pool2_bwd<<<cdiv_ll(BC * H * W, 256), 256, 0, CNN_STREAM(stream)>>>(gout, gin, BC, H, W, accumulate);
    return cnn_status();
}

extern "C" int gpair_cnn_up2(const float *in, float *out, long long BC, int H, int W, void *stream)
{
    if (BC <= 0 || H <= 0 || W <= 0) return GPAIR_ERR_INVALID;
    k_up2<<<cdiv_ll(BC * 4 * H * W, 256), 256, 0, CNN_STREAM(stream)>>>(in, out, BC, H, W);
    return cnn_status();
}

extern "C" int gpair_cnn_up2_bwd(const float *gout, float *gin, long long BC, int H, int W, void *stream)
{
    if (BC <= 0 || H <= 0 || W <= 0) return GPAIR_ERR_INVALID;
    k_up2_bwd<<<cdiv_ll(BC * H * W, 256), 256, 0, CNN_STREAM(stream)>>>(gout, gin, BC, H, W);
    return cnn_status();
}

extern "C" int gpair_cnn_head(const float *d, const float *w, const float *bias, float *z, float *out, float *asum,
                              int B, int C, int HW, void *stream)
{
    if (B <= 0 || C <= 0 || HW <= 0) return GPAIR_ERR_INVALID;
    k_head<<<B * HD_CTAS, 256, 0, CNN_STREAM(stream)>>>(d, w, bias, z, out, asum, C, HW);
    return cnn_status();
}

extern "C" int gpair_cnn_head_bwd(const float *d, const float *w, const float *z, const float *out, const float *asum,
                                  const float *gout, float *gd, float *dw, float *scratch, int B, int C, int HW,
                                  void *stream)
{
    if (B <= 0 || C <= 0 || HW <= 0) return GPAIR_ERR_INVALID;
    k_head_bwd<<<B * HD_CTAS, 256, 0, CNN_STREAM(stream)>>>(d, w, z, out, asum, gout, gd, scratch, C, HW);
    // dw[c] (c < C) and dbias (c = C): fixed-order sums over the images
    k_reduce_slices<<<cdiv_ll(C + 1, 256), 256, 0, CNN_STREAM(stream)>>>(scratch, C + 1, B, dw);
    return cnn_status();
}

extern "C" int gpair_cnn_mse(const float *out, const float *target, float *gout, double *loss, int B, int HW,
                             float gscale, int mode, void *stream)
{
    if (B <= 0 || HW <= 0 || mode < 0 || mode > 1) return GPAIR_ERR_INVALID;
    k_mse<<<B * HD_CTAS, 256, 0, CNN_STREAM(stream)>>>(out, target, gout, loss, HW, gscale, mode);
    return cnn_status();
}

extern "C" int gpair_cnn_adam(float *p, void *p_bf16, const float *g, float *m, float *v, int n, float lr, float b1,
                              float b2, float eps, int step, void *stream)
{
    if (n <= 0 || step <= 0) return GPAIR_ERR_INVALID;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<cdiv_ll(n, 256), 256, 0, CNN_STREAM(stream)>>>(p, (__nv_bfloat16 *)p_bf16, g, m, v, n, lr, b1, b2, eps,
                                                            c1, c2);
    return cnn_status();
}

extern "C" int gpair_cnn_to_bf16(const float *src, void *dst, int n, void *stream)
{
    if (n <= 0) return GPAIR_ERR_INVALID;
    k_to_bf16<<<cdiv_ll(n, 256), 256, 0, CNN_STREAM(stream)>>>(src, (__nv_bfloat16 *)dst, n);
    return cnn_status();
}
