// loss.cu -- L = (1 - lambda) * L1 + lambda * (1 - SSIM) and dL/dpixel.
//
// Follows src/cpu/backward.rs:646-807: per channel, SSIM with an 11-tap
// Gaussian window (sigma 1.5, normalised, backward.rs:759-772) applied as a
// separable blur with zero padding (backward.rs:776-807), C1 = 0.01^2,
// C2 = 0.03^2, and the gradient through five further blurs of the maps P, Q,
// R, Q*mu_y, R*mu_x (backward.rs:718-755). dL1 uses Rust's signum (+1 for
// +0.0), written as copysignf.
//
// B200 mapping: one CTA per 32x32 output tile of any view of the batch. The
// CTA stages the rendered and target channels over a 52x52 region (two
// 5-pixel halos) in shared memory and runs all blurs there, so HBM sees
// each input pixel about once and dL/dpixel is written once. The blurs are
// register-blocked (a thread produces a run of outputs from one sliding
// window, so each shared-memory value and each product is formed once per run).
// k_loss<false>, the default, accumulates with fused multiply-adds and forms the
// SSIM quotients from one reciprocal; k_loss<true> keeps the reference's separate
// multiply and add per tap and its divisions (dL/dpixel bit-identical,
// rgs_options.exact_loss). The scalar loss is reduced per CTA and then per view
// in a fixed order (deterministic).
#include <algorithm>
#include <mutex>

#include "rgs_internal.cuh"
#include "rgs_math.cuh"

namespace rgs {

constexpr int LT = 32;            // output tile edge
constexpr int LR = 5;             // window radius
constexpr int RG = LT + 4 * LR;   // 52: staged input region
constexpr int MG = LT + 2 * LR;   // 42: statistics / map region

// From the blurred statistics of one pixel (means mx, my; second moments
// exx, eyy, exy): its SSIM value (returned) and the maps the gradient blurs
// (backward.rs:718-755): P, Q, R, Q*mu_y, R*mu_x. FAST: one reciprocal for the
// three quotients; otherwise the reference's divisions.
template <bool FAST>
__device__ __forceinline__ float ssim_maps(float mx, float my, float exx, float eyy, float exy, float& P, float& Q, float& R,
                                           float& QM, float& RM) {
    const float C1 = 0.01f * 0.01f;
    const float C2 = 0.03f * 0.03f;
    float sx2 = exx - mx * mx;
    float sy2 = eyy - my * my;
    float sxy = exy - mx * my;
    float a1 = 2.0f * mx * my + C1;
    float a2 = 2.0f * sxy + C2;
    float b1 = mx * mx + my * my + C1;
    float b2 = sx2 + sy2 + C2;
    float num = a1 * a2;
    float den = b1 * b2;
    float inv_den = 1.0f / den;
    const float s_map = FAST ? num * inv_den : num / den;
    const float s_den2 = FAST ? s_map * inv_den : num / (den * den);
    P = inv_den * (2.0f * my * a2) - s_den2 * (2.0f * mx * b2);
    Q = inv_den * (2.0f * a1);
    R = -s_den2 * b1;
    QM = Q * my;
    RM = R * mx;
    return s_map;
}

// Two independent accumulators per packed f32x2 instruction (per lane the
// rounding of the scalar one): the statistics as (x, y), (x^2, y^2), xy; the maps
// as (P, Q), (R, Q mu_y), R mu_x. Pass outputs live in shared memory as float2
// planes of those pairs (plus one float plane).
//
// What bounds it: the shared-memory pipe (60 % of cycles, a quarter of its
// wavefronts bank conflicts) and the latency around the four barriers per channel,
// with 18 warps an SM; the FMA pipe (339 fused multiply-adds per pixel and channel
// with the halos) is 47 % busy. Ten warps
// share a 32x32 tile: with runs of 7, 6, 8 and 4 outputs the four passes have
// 312, 294, 168 and 256 work items for 320 threads (256 threads leave the first
// pass a second round that is three quarters empty). The maps reuse the input's
// shared memory and pass 3's output that of pass 1; the tile arrives a row per
// warp by 4-byte asynchronous copies, the next channel's while this one's last
// pass runs; rows are padded against bank conflicts. 0.84 -> 0.77 ms (1M
// Gaussians x 8 views, 8.5M pixels), 162 -> 151 us (1600x1064), 20.0 -> 17.5 us
// (256x256). 256 and 384 threads 0.85 and 0.83 ms. The exact form, twice the
// operations of each tap, ran on scalars with 256 threads before: 370 -> 315 us
// (three views, 2.75M pixels).
//
// Fewer blurs would do: P', (Q mu_y)' and (R mu_x)' enter the gradient as one
// sum, and E[x^2] + E[y^2] as one; seven blurs ran 0.60 ms, eight 0.71. Not
// kept: the variances and the gradient's terms cancel to 1e-3 of their size, so
// either form carries a rounding error of 2 to 4e-5 of the gradient's norm, and
// two forms differ by as much from one another.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

constexpr int FL_THREADS = 320;
constexpr int FL_WARPS = FL_THREADS / 32;
constexpr int FH1 = 7, FV1 = 6, FH2 = 8, FV2 = 4;  // run lengths of the four passes
constexpr int FRS = RG + 1;   // row strides (float2 / float)
constexpr int FTS = MG + 1;
constexpr int FGS = LT + 1;
static_assert(MG % FH1 == 0 && MG % FV1 == 0 && LT % FH2 == 0 && LT % FV2 == 0, "run lengths must tile the regions");
constexpr size_t FL_IN = sizeof(float2) * RG * FRS;                                   // x, y
constexpr size_t FL_MAPS = (2 * sizeof(float2) + sizeof(float)) * MG * FTS;            // (P, Q), (R, Q mu_y), R mu_x
constexpr size_t FL_AREA0 = ((FL_IN > FL_MAPS ? FL_IN : FL_MAPS) + 15) & ~(size_t)15;
constexpr size_t FL_AREA1 = (2 * sizeof(float2) + sizeof(float)) * RG * FTS;          // pass 1 out; then pass 3 out
constexpr size_t FL_SMEM = FL_AREA0 + FL_AREA1 + sizeof(float) * (16 + 2 * FL_WARPS);
static_assert(FL_AREA0 % 16 == 0 && FL_AREA1 % 16 == 0, "each area starts on a float2 boundary");
static_assert((2 * sizeof(float2) + sizeof(float)) * MG * FGS <= FL_AREA1, "pass-3 output must fit in the pass-1 buffer");

// Four bytes global -> shared, asynchronously; zero when !in (nothing is read).
__device__ __forceinline__ void copy4(float* dst, const float* src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(in ? 4 : 0)
                 : "memory");
}

__device__ __forceinline__ float fl_block_sum(float v, float* s_red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.0f;
    for (int k = 0; k < FL_WARPS; ++k) t += s_red[k];
    return t;
}

// acc + w * x: rounded once, or (EXACT) twice, as the reference's multiply and
// add. `one` is 1 at run time: the compiler joins a packed multiply and add into
// one instruction, but not a multiply and this fma.
template <bool EXACT>
__device__ __forceinline__ float2 tap_add2(float2 w, float2 x, float2 acc, float2 one) {
    return EXACT ? __ffma2_rn(__fmul2_rn(w, x), one, acc) : __ffma2_rn(w, x, acc);
}
template <bool EXACT>
__device__ __forceinline__ float tap_add(float w, float x, float acc) {
    return EXACT ? __fadd_rn(acc, __fmul_rn(w, x)) : __fmaf_rn(w, x, acc);
}

template <bool EXACT>
__global__ void __launch_bounds__(FL_THREADS, 2) k_loss(const DevCam* __restrict__ cams, int nviews, const uint32_t* total_dev,
                                                        int total_host, const float* __restrict__ rgb, float lambda, float one,
                                                        float* __restrict__ dl, float* __restrict__ partials) {
    extern __shared__ __align__(16) unsigned char fl_smem[];
    float2* in = reinterpret_cast<float2*>(fl_smem);               // [RG][FRS]
    float2* m01 = reinterpret_cast<float2*>(fl_smem);              // [MG][FTS], over the input
    float2* m23 = m01 + MG * FTS;
    float* m4 = reinterpret_cast<float*>(m23 + MG * FTS);
    float2* t01 = reinterpret_cast<float2*>(fl_smem + FL_AREA0);   // [RG][FTS]: mu_x, mu_y
    float2* t23 = t01 + RG * FTS;                                  // E[x^2], E[y^2]
    float* t4 = reinterpret_cast<float*>(t23 + RG * FTS);          // E[xy]
    float2* g01 = reinterpret_cast<float2*>(fl_smem + FL_AREA0);   // [MG][FGS], over pass 1's output
    float2* g23 = g01 + MG * FGS;
    float* g4 = reinterpret_cast<float*>(g23 + MG * FGS);
    float* kw = reinterpret_cast<float*>(fl_smem + FL_AREA0 + FL_AREA1);
    float* s_red = kw + 16;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        // gaussian_kernel_1d(5, 1.5), backward.rs:759-772
        float sum = 0.0f;
        float v[11];
        for (int i = 0; i < 11; ++i) {
            float d = (float)i - 5.0f;
            v[i] = exp_cr(-0.5f * d * d / (1.5f * 1.5f));
            sum += v[i];
        }
        for (int i = 0; i < 11; ++i) kw[i] = v[i] / sum;
    }
    __syncthreads();
    float2 ww[6];  // the taps (symmetric), duplicated for the packed lanes
#pragma unroll
    for (int k = 0; k < 6; ++k) ww[k] = f2(kw[k], kw[k]);
    auto tap = [&](int k) { return ww[k < 6 ? k : 10 - k]; };
    const float2 one2 = f2(one, one);
    const int total = total_dev ? (int)*total_dev : total_host;
    for (int blk = blockIdx.x; blk < total; blk += gridDim.x) {
        int v = 0;
        while (v + 1 < nviews && cams[v + 1].loss_base <= blk) ++v;
        const DevCam& c = cams[v];
        const int w = c.width, h = c.height;
        const int lb = blk - c.loss_base;
        const int ox = (lb % c.loss_bx) * LT, oy = (lb / c.loss_bx) * LT;
        const float m_total = (float)((size_t)w * h * 3);
        const float g_l1 = (1.0f - lambda) / m_total;  // times +-1: the reference's quotient exactly
        const float* tgt = c.target;
        const float* img = rgb + (size_t)c.pix_base * 3;
        float* grad_out = dl + (size_t)c.pix_base * 3;
        float l1_local = 0.0f, ssim_local = 0.0f;
        // one row of the region per warp and step, two columns per lane
        const int gx0 = ox - 2 * LR + lane, gx1 = gx0 + 32;
        const bool in0 = gx0 >= 0 && gx0 < w, in1 = lane < RG - 32 && gx1 >= 0 && gx1 < w;
        const ptrdiff_t first = (ptrdiff_t)(oy - 2 * LR + warp) * w + gx0, step = (ptrdiff_t)w * FL_WARPS;
        auto load = [&](int ch) {
            const float* pi = img + first * 3 + ch;
            const float* pt = tgt + first * 4 + ch;
            float2* dst = in + warp * FRS + lane;
#pragma unroll 2
            for (int gy = oy - 2 * LR + warp; gy < oy - 2 * LR + RG; gy += FL_WARPS, pi += step * 3, pt += step * 4, dst += FL_WARPS * FRS) {
                const bool row = gy >= 0 && gy < h;
                copy4(&dst[0].x, row && in0 ? pi : img, row && in0);
                copy4(&dst[0].y, row && in0 ? pt : tgt, row && in0);
                if (lane < RG - 32) {
                    copy4(&dst[32].x, row && in1 ? pi + 32 * 3 : img, row && in1);
                    copy4(&dst[32].y, row && in1 ? pt + 32 * 4 : tgt, row && in1);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        load(0);
#pragma unroll 1
        for (int ch = 0; ch < 3; ++ch) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            // pass 1: horizontal blur of (x, y), (x^2, y^2), xy over rows [0, RG)
            for (int it = tid; it < RG * (MG / FH1); it += FL_THREADS) {
                const int r = it % RG, c0 = (it / RG) * FH1;
                const float2* row = in + r * FRS + c0;
                float2 a01[FH1], a23[FH1];
                float a4[FH1];
#pragma unroll
                for (int o = 0; o < FH1; ++o) {
                    a01[o] = a23[o] = f2(0.0f, 0.0f);
                    a4[o] = 0.0f;
                }
#pragma unroll
                for (int j = 0; j < FH1 + 10; ++j) {
                    const float2 xy = row[j];
                    const float2 sp = __fmul2_rn(xy, xy);
                    const float cr = xy.x * xy.y;
#pragma unroll
                    for (int o = 0; o < FH1; ++o) {
                        const int k = j - o;
                        if (k < 0 || k > 10) continue;
                        a01[o] = tap_add2<EXACT>(tap(k), xy, a01[o], one2);
                        a23[o] = tap_add2<EXACT>(tap(k), sp, a23[o], one2);
                        a4[o] = tap_add<EXACT>(tap(k).x, cr, a4[o]);
                    }
                }
#pragma unroll
                for (int o = 0; o < FH1; ++o) {
                    t01[r * FTS + c0 + o] = a01[o];
                    t23[r * FTS + c0 + o] = a23[o];
                    t4[r * FTS + c0 + o] = a4[o];
                }
            }
            __syncthreads();
            // pass 2: vertical blur -> statistics, then the per-pixel maps
            // (zero outside the image)
            for (int it = tid; it < MG * (MG / FV1); it += FL_THREADS) {
                const int cm = it % MG, r0 = (it / MG) * FV1;
                float2 mu[FV1], sq[FV1];
                float cr[FV1];
#pragma unroll
                for (int o = 0; o < FV1; ++o) {
                    mu[o] = sq[o] = f2(0.0f, 0.0f);
                    cr[o] = 0.0f;
                }
#pragma unroll
                for (int j = 0; j < FV1 + 10; ++j) {
                    const float2 u = t01[(r0 + j) * FTS + cm], q = t23[(r0 + j) * FTS + cm];
                    const float e = t4[(r0 + j) * FTS + cm];
#pragma unroll
                    for (int o = 0; o < FV1; ++o) {
                        const int k = j - o;
                        if (k < 0 || k > 10) continue;
                        mu[o] = tap_add2<EXACT>(tap(k), u, mu[o], one2);
                        sq[o] = tap_add2<EXACT>(tap(k), q, sq[o], one2);
                        cr[o] = tap_add<EXACT>(tap(k).x, e, cr[o]);
                    }
                }
                const int gx = ox - LR + cm;
#pragma unroll
                for (int o = 0; o < FV1; ++o) {
                    const int rm = r0 + o, gy = oy - LR + rm;
                    float P = 0.0f, Q = 0.0f, R = 0.0f, QM = 0.0f, RM = 0.0f;
                    if (gx >= 0 && gx < w && gy >= 0 && gy < h) {
                        const float ssim = ssim_maps<!EXACT>(mu[o].x, mu[o].y, sq[o].x, sq[o].y, cr[o], P, Q, R, QM, RM);
                        if (rm >= LR && rm < LR + LT && cm >= LR && cm < LR + LT) ssim_local += ssim;
                    }
                    m01[rm * FTS + cm] = f2(P, Q);
                    m23[rm * FTS + cm] = f2(R, QM);
                    m4[rm * FTS + cm] = RM;
                }
            }
            __syncthreads();
            // pass 3: horizontal blur of the maps: rows [0, MG), output columns [0, LT)
            for (int it = tid; it < MG * (LT / FH2); it += FL_THREADS) {
                const int rm = it % MG, c0 = (it / MG) * FH2;
                float2 a[FH2], d[FH2];
                float e[FH2];
#pragma unroll
                for (int o = 0; o < FH2; ++o) {
                    a[o] = d[o] = f2(0.0f, 0.0f);
                    e[o] = 0.0f;
                }
#pragma unroll
                for (int j = 0; j < FH2 + 10; ++j) {
                    const int p = rm * FTS + c0 + j;
                    const float2 t = m01[p], u = m23[p];
                    const float q = m4[p];
#pragma unroll
                    for (int o = 0; o < FH2; ++o) {
                        const int k = j - o;
                        if (k < 0 || k > 10) continue;
                        a[o] = tap_add2<EXACT>(tap(k), t, a[o], one2);
                        d[o] = tap_add2<EXACT>(tap(k), u, d[o], one2);
                        e[o] = tap_add<EXACT>(tap(k).x, q, e[o]);
                    }
                }
#pragma unroll
                for (int o = 0; o < FH2; ++o) {
                    g01[rm * FGS + c0 + o] = a[o];
                    g23[rm * FGS + c0 + o] = d[o];
                    g4[rm * FGS + c0 + o] = e[o];
                }
            }
            __syncthreads();
            // the maps are read: the next channel's region may take their place
            if (ch < 2) load(ch + 1);
            // pass 4: vertical blur -> gradient, combined with the L1 term
            for (int it = tid; it < LT * (LT / FV2); it += FL_THREADS) {
                const int co = it % LT, r0 = (it / LT) * FV2;
                const int gx = ox + co, gy0 = oy + r0;
                const ptrdiff_t p0 = (ptrdiff_t)gy0 * w + gx;
                float x[FV2], y[FV2];
#pragma unroll
                for (int o = 0; o < FV2; ++o) {
                    const bool ok = gx < w && gy0 + o < h;
                    x[o] = ok ? img[(p0 + (ptrdiff_t)o * w) * 3 + ch] : 0.0f;
                    y[o] = ok ? tgt[(p0 + (ptrdiff_t)o * w) * 4 + ch] : 0.0f;
                }
                float2 a[FV2], g[FV2];
                float e[FV2];
#pragma unroll
                for (int o = 0; o < FV2; ++o) {
                    a[o] = g[o] = f2(0.0f, 0.0f);
                    e[o] = 0.0f;
                }
#pragma unroll
                for (int j = 0; j < FV2 + 10; ++j) {
                    const int p = (r0 + j) * FGS + co;
                    const float2 t = g01[p], u = g23[p];
                    const float q = g4[p];
#pragma unroll
                    for (int o = 0; o < FV2; ++o) {
                        const int k = j - o;
                        if (k < 0 || k > 10) continue;
                        a[o] = tap_add2<EXACT>(tap(k), t, a[o], one2);
                        g[o] = tap_add2<EXACT>(tap(k), u, g[o], one2);
                        e[o] = tap_add<EXACT>(tap(k).x, q, e[o]);
                    }
                }
#pragma unroll
                for (int o = 0; o < FV2; ++o) {
                    if (gx >= w || gy0 + o >= h) continue;
                    const float grad = a[o].x + y[o] * a[o].y - g[o].y + 2.0f * x[o] * g[o].x - 2.0f * e[o];
                    const float d = x[o] - y[o];
                    l1_local += fabsf(d);
                    const float sg = (d != d) ? d : copysignf(1.0f, d);
                    grad_out[(p0 + (ptrdiff_t)o * w) * 3 + ch] = g_l1 * sg + -lambda * grad / m_total;
                }
            }
        }
        float l1s = fl_block_sum(l1_local, s_red);
        float sss = fl_block_sum(ssim_local, s_red + FL_WARPS);
        if (tid == 0) {
            partials[(size_t)blk * 2 + 0] = l1s;
            partials[(size_t)blk * 2 + 1] = sss;
        }
    }
}

// One CTA per view: each thread sums a strided subset of the view's per-block
// partials in double, then a fixed-shape tree combines the threads, so the
// result does not depend on scheduling.
constexpr int FIN_THREADS = 256;
__global__ void __launch_bounds__(FIN_THREADS) k_loss_finalize(const DevCam* __restrict__ cams, int nviews,
                                                               const float* __restrict__ partials, float lambda,
                                                               float* __restrict__ losses) {
    __shared__ double s_l1[FIN_THREADS], s_ss[FIN_THREADS];
    const int v = blockIdx.x, tid = threadIdx.x;
    if (v >= nviews) return;
    const DevCam& c = cams[v];
    const int nb = c.loss_bx * ((c.height + LT - 1) / LT);
    double l1 = 0.0, ss = 0.0;
    for (int b = tid; b < nb; b += FIN_THREADS) {
        l1 += (double)partials[(size_t)(c.loss_base + b) * 2 + 0];
        ss += (double)partials[(size_t)(c.loss_base + b) * 2 + 1];
    }
    s_l1[tid] = l1;
    s_ss[tid] = ss;
    __syncthreads();
    for (int o = FIN_THREADS / 2; o > 0; o >>= 1) {
        if (tid < o) {
            s_l1[tid] += s_l1[tid + o];
            s_ss[tid] += s_ss[tid + o];
        }
        __syncthreads();
    }
    if (tid == 0) {
        float m = (float)((size_t)c.width * c.height * 3);
        float l1m = (float)(s_l1[0] / (double)m);
        float ssm = (float)(s_ss[0] / (double)m);
        losses[v] = (1.0f - lambda) * l1m + lambda * (1.0f - ssm);
    }
}

cudaError_t prepare_loss_kernel() {
    static std::mutex mu;
    static bool ready[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (ready[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(k_loss<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FL_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_loss<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FL_SMEM);
    if (e == cudaSuccess) ready[dev] = true;
    return e;
}

cudaError_t launch_loss(const DevCam* cams, int nviews, int total_blocks, const float* rgb, float lambda, float* dl,
                        float* partials, float* losses, const uint32_t* total_dev, bool exact, cudaStream_t st) {
    cudaError_t e = prepare_loss_kernel();
    if (e != cudaSuccess) return e;
    const int sms = device_sm_count();
    const int most = sms * 2;
    const int grid = std::max(1, total_dev ? most : std::min(total_blocks, most));
    (exact ? k_loss<true> : k_loss<false>)<<<grid, FL_THREADS, FL_SMEM, st>>>(cams, nviews, total_dev, total_blocks, rgb, lambda,
                                                                             1.0f, dl, partials);
    if (nviews > 0) k_loss_finalize<<<nviews, FIN_THREADS, 0, st>>>(cams, nviews, partials, lambda, losses);
    return cudaGetLastError();
}

}  // namespace rgs
