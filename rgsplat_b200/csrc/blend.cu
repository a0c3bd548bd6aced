// blend.cu -- per-tile alpha blending (forward) and its analytic reverse pass.
//
// Forward follows src/cpu/backward.rs:296-385 (`forward_pass`): per pixel, walk
// the tile's depth-ordered list; power = -1/2 d^T conic d; skip power > 0;
// alpha = min(opacity * e^power, 0.99); skip alpha < 1/255; composite
// front-to-back; stop after the update that drops T below 1e-4; output
// C + T * bg, the final T and the index of the last contributor.
// Backward follows backward.rs:391-512 (`backward_pass`): from the last
// contributor down to 0, rebuild T by T /= (1 - alpha) -- no per-Gaussian
// blend state is stored -- and accumulate d color, d opacity, d conic and
// d mean per splat.
//
// B200 mapping: one CTA per CTA tile (TW x TH pixels, one pixel per thread),
// persistent CTAs pulling tiles of every view of the batch from one atomic
// counter. Splat records are staged BATCH at a time in shared memory and read
// by all threads as broadcasts. The kernels are issue-bound, so work that the
// reference's own tests would discard is removed without changing any result:
//   * per splat, alpha < 1/255 is guaranteed once power < thr with
//     thr = ln(1 / (255 opacity)) - 0.01, so such pixels skip exp;
//   * per (tile, splat), if the conic's quadratic form is bounded below over
//     the box of the tile's pixel centres so that power < thr everywhere, the
//     splat is dropped from the staged batch (the batch is compacted, keeping
//     each splat's index in the full tile list for last_contrib);
//   * backward: per (warp, staged splat), the same test on the box of the
//     warp's own strip of pixel rows; a warp whose strip the splat cannot
//     reach skips it (warp-uniform). (The same skip in the forward measured
//     slower, as a per-splat branch and as a per-warp list of the needed
//     splats alike: a pair that does not contribute costs the packed forward
//     about five instructions per pixel, less than the strip tests add to
//     every staging round.)
//   * backward warps skip splats past the warp's largest last_contrib.
// Backward gathers each warp's partial gradients of eight splats in shared
// memory, reads them back transposed (four lanes per splat) and issues one
// 3 x 16-byte vector reduction (red.global.add.v4.f32) per splat per warp.
//
// CTA tiles other than 16x16 keep the reference's per-pixel semantics: each
// record carries its reference-tile rectangle in pixels and a pixel only
// evaluates splats whose rectangle contains it (RECT = true).
#include <algorithm>
#include <mutex>

#include "rgs_internal.cuh"
#include "rgs_math.cuh"
#include "tiles.cuh"

namespace rgs {

__device__ __forceinline__ int find_view(const DevCam* cams, int nviews, int tile) {
    int v = 0;
    while (v + 1 < nviews && cams[v + 1].tile_base <= tile) ++v;
    return v;
}

__device__ __forceinline__ bool in_rect(float rx, float ry, int px, int py) {
    uint32_t x = __float_as_uint(rx), y = __float_as_uint(ry);
    return px >= (int)(x & 0xffffu) && px < (int)(x >> 16) && py >= (int)(y & 0xffffu) && py < (int)(y >> 16);
}

// Stages the tile-list entries [first, end) (at most BATCH) into shared memory,
// dropping splats the tile test rejects; returns the kept count (block-uniform).
// li0 is the tile-list index of `first`. Must be called by the whole block.
// When s_rall is given, every staged entry's pixel rectangle (kept or not) is
// recorded at its batch position.
template <int NT, int BATCH>
__device__ __forceinline__ int stage_batch(const BlendArgs& a, size_t S, uint32_t first, uint32_t end, int li0, float x0c,
                                           float x1c, float y0c, float y1c, float4* s_a, float4* s_c, float4* s_k, int* s_li,
                                           int* s_wsum, uint2* s_rall) {
    constexpr int NW = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int kept = 0;
#pragma unroll
    for (int c0 = 0; c0 < BATCH; c0 += NT) {
        const int j = c0 + tid;
        const uint32_t idx = first + (uint32_t)j;
        bool keep = false;
        float4 A, Q, K;
        if (j < BATCH && idx < end) {
            const uint32_t slot = a.pair_vals[idx];
            A = a.rec[slot];
            Q = a.rec[S + slot];
            K = a.rec[2 * S + slot];
            A.w = power_floor(A.z);
            const TileTest t = tile_test_setup(A.x, A.y, Q.x, Q.y, Q.z, A.w);
            keep = !tile_rejects(t, x0c, x1c, y0c, y1c);
            if (s_rall) s_rall[j] = make_uint2(__float_as_uint(Q.w), __float_as_uint(K.w));
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s_wsum[w] = __popc(m);
        __syncthreads();
        int off = kept, total = 0;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            const int t = s_wsum[k];
            off += k < w ? t : 0;
            total += t;
        }
        if (keep) {
            const int p = off + __popc(m & ((1u << lane) - 1u));
            s_a[p] = A;
            s_c[p] = Q;
            s_k[p] = K;
            s_li[p] = li0 + j;
        }
        kept += total;
        __syncthreads();
    }
    return kept;
}

// Forward. PPT vertically adjacent pixels per thread share dx and the
// dx-only products of power, which are evaluated once per (splat, thread) in
// the reference's rounding order.
// The TW threads that share a pixel row would each form dy and Q.z*dy*dy for
// every splat; where the shared memory allows (ROWTERMS), the CTA forms them
// once per (staged splat, tile row) after staging, with the same operations.
template <int BATCH, int TH, int PPT>
struct RowTerms {
    static constexpr bool on = BATCH * TH <= 2048 && PPT % 2 == 0;
};

template <int TW, int TH, int BATCH, bool RECT, int PPT, bool STORE = false>
__global__ void __launch_bounds__(TW * TH / PPT) k_blend_fwd(BlendArgs a) {
    constexpr int NT = TW * TH / PPT;
    constexpr bool ROWTERMS = RowTerms<BATCH, TH, PPT>::on;
    // two pixels per thread in packed f32x2 lanes (the store-all study keeps
    // the scalar loop)
    constexpr bool PACK = PPT == 2 && !STORE;
    const float2 one2 = make_float2(a.one, a.one);
    __shared__ float4 s_a[BATCH];
    __shared__ float4 s_c[BATCH];
    __shared__ float4 s_k[BATCH];
    __shared__ int s_li[BATCH];
    __shared__ int s_wsum[NT / 32];
    __shared__ uint2 s_rall[RECT ? BATCH : 1];
    __shared__ __align__(16) float2 s_row[ROWTERMS ? BATCH : 1][ROWTERMS ? TH : 1];  // (dy, Q.z*dy*dy)
    __shared__ int s_tile;
    const int tid = threadIdx.x;
    const int total_tiles = a.total_tiles ? (int)*a.total_tiles : a.total_tiles_host;
    const size_t S = (size_t)a.n_per_view * a.nviews;
    for (;;) {
        if (tid == 0) s_tile = (int)atomicAdd(a.work, 1u);
        __syncthreads();
        const int tile = s_tile;
        if (tile >= total_tiles) break;
        const int v = find_view(a.cams, a.nviews, tile);
        const DevCam& c = a.cams[v];
        const int lt = tile - c.tile_base;
        const int tx = lt % c.tiles_x, ty = lt / c.tiles_x;
        const int px = tx * TW + (tid % TW), py0 = ty * TH + (tid / TW) * PPT;
        const float pxf = (float)px + 0.5f;
        // box of the tile's pixel centres
        const float x0c = (float)(tx * TW) + 0.5f, x1c = (float)(min(tx * TW + TW, c.width) - 1) + 0.5f;
        const float y0c = (float)(ty * TH) + 0.5f, y1c = (float)(min(ty * TH + TH, c.height) - 1) + 0.5f;
        const uint2 rg = a.ranges[tile];
        float T[PPT], C0[PPT], C1[PPT], C2[PPT], pyc[PPT];
        int last[PPT];
        bool done[PPT], seen[PPT];
        bool all_done = true;
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            pyc[p] = (float)(py0 + p) + 0.5f;
            T[p] = 1.0f;
            C0[p] = a.bg_start ? a.bg[0] : 0.0f;
            C1[p] = a.bg_start ? a.bg[1] : 0.0f;
            C2[p] = a.bg_start ? a.bg[2] : 0.0f;
            last[p] = -1;
            done[p] = !(px < c.width && py0 + p < c.height);
            all_done &= done[p];
            // whether the pixel's reference tile list is non-empty
            seen[p] = !RECT && rg.y > rg.x;
        }
        for (uint32_t b0 = rg.x; b0 < rg.y; b0 += BATCH) {
            if (__syncthreads_count(!all_done) == 0) break;
            const bool need_seen = RECT && a.empty_tile_black;
            const int nb = stage_batch<NT, BATCH>(a, S, b0, rg.y, (int)(b0 - rg.x), x0c, x1c, y0c, y1c, s_a, s_c, s_k, s_li,
                                                  s_wsum, need_seen ? s_rall : nullptr);
            if (need_seen) {
                // a pixel's reference tile list is non-empty iff some entry (kept
                // or rejected) covers the pixel
                const int staged = (int)min((uint32_t)BATCH, rg.y - b0);
#pragma unroll
                for (int p = 0; p < PPT; ++p)
                    for (int j = 0; j < staged && !seen[p]; ++j)
                        if (in_rect(__uint_as_float(s_rall[j].x), __uint_as_float(s_rall[j].y), px, py0 + p)) seen[p] = true;
            }
            if (ROWTERMS) {
                for (int idx = tid; idx < nb * TH; idx += NT) {
                    const int k = idx / TH, r = idx - k * TH;
                    const float dy = ((float)(ty * TH + r) + 0.5f) - s_a[k].y;
                    s_row[k][r] = make_float2(dy, s_c[k].z * dy * dy);
                }
                __syncthreads();
            }
            const int rbase = (tid / TW) * PPT;  // this thread's first row in the tile
            for (int k = 0; k < nb && !all_done; ++k) {
                const float4 A = s_a[k];
                const float4 Q = s_c[k];
                const float dx = pxf - A.x;
                const float tdx = Q.x * dx * dx;
                const float t2b = 2.0f * Q.y * dx;
                float4 rw[(PPT + 1) / 2];  // two rows' (dy, Q.z*dy*dy) per 16-byte load
#pragma unroll
                for (int h = 0; h < (PPT + 1) / 2; ++h)
                    rw[h] = ROWTERMS ? *reinterpret_cast<const float4*>(&s_row[k][rbase + 2 * h]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (PACK && !a.bg_start) {
                    // both pixels in packed f32x2 lanes, each lane rounded exactly as
                    // the scalar loop below rounds that pixel; a pixel that does not
                    // take this splat gets alpha = 0, which leaves its colour
                    // (+0 added to a non-negative sum) and T (times 1) unchanged
                    float2 dy2, qdd2;
                    if (ROWTERMS) {
                        dy2 = make_float2(rw[0].x, rw[0].z);
                        qdd2 = make_float2(rw[0].y, rw[0].w);
                    } else {
                        dy2 = __fadd2_rn(make_float2(pyc[0], pyc[PPT > 1 ? 1 : 0]), bc2(-A.y));
                        qdd2 = __fmul2_rn(__fmul2_rn(bc2(Q.z), dy2), dy2);
                    }
                    // power = -0.5 * ((tdx + t2b * dy) + qdd)
                    const float2 s1 = __ffma2_rn(__fmul2_rn(bc2(t2b), dy2), one2, bc2(tdx));
                    const float2 s2 = ROWTERMS ? __fadd2_rn(s1, qdd2) : __ffma2_rn(qdd2, one2, s1);
                    const float2 pw = __fmul2_rn(s2, bc2(-0.5f));
                    bool act0 = !done[0] && !(pw.x > 0.0f) && !(pw.x < A.w);
                    bool act1 = !done[PPT > 1 ? 1 : 0] && !(pw.y > 0.0f) && !(pw.y < A.w);
                    if (RECT) {
                        act0 = act0 && in_rect(Q.w, s_k[k].w, px, py0);
                        act1 = act1 && in_rect(Q.w, s_k[k].w, px, py0 + 1);
                    }
                    if (act0 || act1) {
                        const float2 ar = __fmul2_rn(bc2(A.z), expf_fast_nonpos2(pw, one2));
                        float al0 = fminf(ar.x, 0.99f), al1 = fminf(ar.y, 0.99f);
                        act0 = act0 && !(al0 < 1.0f / 255.0f);
                        act1 = act1 && !(al1 < 1.0f / 255.0f);
                        if (act0 || act1) {
                            const float4 K = s_k[k];
                            const float2 al = make_float2(act0 ? al0 : 0.0f, act1 ? al1 : 0.0f);
                            float2 T2 = make_float2(T[0], T[PPT > 1 ? 1 : 0]);
                            const float2 w = __fmul2_rn(al, T2);
                            const float2 c0 = __ffma2_rn(__fmul2_rn(bc2(K.x), w), one2, make_float2(C0[0], C0[PPT > 1 ? 1 : 0]));
                            const float2 c1 = __ffma2_rn(__fmul2_rn(bc2(K.y), w), one2, make_float2(C1[0], C1[PPT > 1 ? 1 : 0]));
                            const float2 c2 = __ffma2_rn(__fmul2_rn(bc2(K.z), w), one2, make_float2(C2[0], C2[PPT > 1 ? 1 : 0]));
                            T2 = __fmul2_rn(T2, __ffma2_rn(al, make_float2(-one2.x, -one2.y), one2));
                            C0[0] = c0.x; C1[0] = c1.x; C2[0] = c2.x; T[0] = T2.x;
                            C0[PPT - 1] = c0.y; C1[PPT - 1] = c1.y; C2[PPT - 1] = c2.y; T[PPT - 1] = T2.y;
                            const int li = s_li[k];
                            if (act0) {
                                last[0] = li;
                                if (T2.x < 1e-4f) done[0] = true;
                            }
                            if (act1) {
                                last[PPT - 1] = li;
                                if (T2.y < 1e-4f) done[PPT - 1] = true;
                            }
                        }
                    }
                } else {
#pragma unroll
                for (int p = 0; p < PPT; ++p) {
                    if (done[p]) continue;
                    if (RECT && !in_rect(Q.w, s_k[k].w, px, py0 + p)) continue;
                    float dy, qdd;
                    if (ROWTERMS) {
                        dy = (p & 1) ? rw[p >> 1].z : rw[p >> 1].x;
                        qdd = (p & 1) ? rw[p >> 1].w : rw[p >> 1].y;
                    } else {
                        dy = pyc[p] - A.y;
                        qdd = Q.z * dy * dy;
                    }
                    const float power = -0.5f * (tdx + t2b * dy + qdd);
                    if (power > 0.0f || power < A.w) continue;
                    const float alpha = fminf(A.z * expf_fast_nonpos(power), 0.99f);
                    if (alpha < 1.0f / 255.0f) continue;
                    const float4 K = s_k[k];
                    if (STORE) a.tstore[(size_t)(rg.x + (uint32_t)s_li[k]) * (TW * TH) + (tid / TW) * PPT * TW + p * TW + tid % TW] = T[p];
                    const float weight = alpha * T[p];
                    C0[p] += K.x * weight;
                    C1[p] += K.y * weight;
                    C2[p] += K.z * weight;
                    T[p] *= 1.0f - alpha;
                    last[p] = s_li[k];
                    if (T[p] < 1e-4f) done[p] = true;
                }
                }
                all_done = true;
#pragma unroll
                for (int p = 0; p < PPT; ++p) all_done &= done[p];
            }
            __syncthreads();
        }
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            const int py = py0 + p;
            if (px < c.width && py < c.height) {
                size_t pix = (size_t)c.pix_base + (size_t)py * c.width + px;
                // forward_pass skips tiles whose list is empty, leaving their pixels
                // at 0 rather than bg (src/cpu/backward.rs:313-315, 124)
                const bool black = a.empty_tile_black && !seen[p];
                a.rgb[pix * 3 + 0] = black ? 0.0f : a.bg_start ? C0[p] : C0[p] + T[p] * a.bg[0];
                a.rgb[pix * 3 + 1] = black ? 0.0f : a.bg_start ? C1[p] : C1[p] + T[p] * a.bg[1];
                a.rgb[pix * 3 + 2] = black ? 0.0f : a.bg_start ? C2[p] : C2[p] + T[p] * a.bg[2];
                a.final_t[pix] = T[p];
                a.last[pix] = last[p];
            }
        }
        __syncthreads();
    }
}


__device__ __forceinline__ void red_add_v4(float4* addr, float x, float y, float z, float w) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// One pixel of the backward decided with the forward's own arithmetic: nal is
// minus its alpha (0 when it does not take the splat) and um minus the raw
// alpha that scales dL/dalpha (0 when the raw alpha was clamped,
// backward.rs:459-461). A NaN power passes both tests and fminf turns it into
// alpha = 0.99, as in the forward. Kept out of line: a few pixels in 10^5 come
// here.
__device__ __noinline__ float2 bwd_exact_pixel(float dx, float dy, float4 q, float thr) {
    const float tdx = q.x * dx * dx;
    const float t2b = 2.0f * q.y * dx;
    const float power = -0.5f * (tdx + t2b * dy + q.z * dy * dy);
    if (power > 0.0f || power < thr) return make_float2(0.0f, 0.0f);
    const float ar = q.w * expf_fast_nonpos(power);
    const float al = fminf(ar, 0.99f);
    if (al < 1.0f / 255.0f) return make_float2(0.0f, 0.0f);
    return make_float2(-al, ar > 0.99f ? 0.0f : -ar);
}

// Backward. A thread owns PPT vertical pixels in packed f32x2 lanes; T is
// rebuilt as T * 1/(1 - alpha) with the hardware reciprocal (within 2 ulp; the
// reference divides, backward.rs:452).
//
// What bounds it: instruction issue (70 % of cycles; FMA pipe 42 %, ALU 37 %),
// so the loop is built around the fewest instructions per (warp, splat). It
// replaces a loop that tested both thresholds on each pixel's alpha and reduced
// nine sums over the warp for every splat: 3.29 -> 1.60 ms on 1M Gaussians x 8
// views, 1.57 -> 0.60 ms on 97k x 3 views of 1277x719 with a white background,
// 262 -> 70 us on 10k at 256x256 (where one tile's serial walk is the time).
//
// Alpha comes from one SFU exponential of p = power log2(e) + log2(opacity),
// with the power rounded exactly as the forward rounds it. (A power from two
// packed FMAs over prescaled coefficients saves four packed instructions per
// pixel pair and ran 4 % faster; but an ill-conditioned conic's terms cancel,
// and its alpha then strays from the forward's by up to 1e-4.) The
// contributing set must be the forward's exactly, so a pixel whose p lies
// within BWD_BAND of a decision (alpha >= 1/255; alpha_raw > 0.99; power > 0,
// where p reaches log2(opacity)) is decided by bwd_exact_pixel: the roundings
// of p (|p| <= 8), of log2(opacity) and of the forward's own alpha add up to
// less than 2e-6 in log2 units, half the band. Every test reads a NaN as
// "decide exactly".
//
// The nine gradient sums of a splat are not reduced across the warp per splat
// (14 shuffles and two shared atomics each, serialised): a lane stores its six
// column sums (colour x3, u, u dy, u dy^2 with u = dL/dpower) for up to
// BWD_GRP splats in the warp's own shared memory, then the warp reads them
// transposed, four lanes per splat, each adding eight columns, expands the
// moments in dx, and issues one red.global.add.v4 per accumulator plane. The
// stores and loads are swizzled by the splat's place in the group, so neither
// has bank conflicts. Warps share only the staged batch and the two barriers
// around it.
//
// Every lane of a warp that some lane's pixels need runs the whole update (its
// terms are zero); a branch per thread ran 4 % slower. Ten CTAs per SM (96
// registers) with four pixels per thread: 11 and 12 ran 3 % and 5 % slower.
// 64 staged splats: 128 ran 3 % slower. Also measured slower: coefficients
// stored twice so that a 16-byte load fills both lanes of two operands (+9 %),
// the next splat's coefficients loaded ahead (+9 %), the next batch's records
// prefetched into L1 (+8 %).
constexpr float BWD_BAND = 4e-6f;
constexpr int BWD_GRP = 8;
constexpr int BWD_BATCH = 64;

template <int TW, int TH, bool RECT, int PPT, bool STORE = false>
__global__ void __launch_bounds__(TW * TH / PPT, PPT == 2 ? 5 : 10) k_blend_bwd(BlendArgs a) {
    constexpr int NT = TW * TH / PPT;
    constexpr int NW = NT / 32;
    constexpr int H = PPT / 2;
    constexpr float LOG2E = 1.44269504f;
    constexpr float L255 = 7.99435344f;    // log2(255)
    constexpr float L099 = -0.0144995697f;  // log2(0.99)
    __shared__ float4 s_a[BWD_BATCH];  // sx, sy, log2(opacity), opacity
    __shared__ float4 s_c[BWD_BATCH];  // a, b, c, largest p decided without the exact arithmetic
    __shared__ float4 s_k[BWD_BATCH];  // colour, power floor
    __shared__ uint2 s_r[RECT ? BWD_BATCH : 1];
    __shared__ uint32_t s_slot[BWD_BATCH];
    __shared__ uint8_t s_wm[BWD_BATCH];
    __shared__ float4 s_b4[NW][BWD_GRP][32];
    __shared__ float2 s_b2[NW][BWD_GRP][32];
    __shared__ int s_tile;
    __shared__ int s_maxlc;
    constexpr int RW = (32 / TW) * PPT;  // pixel rows per warp
    const float2 one2 = make_float2(a.one, a.one);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int total_tiles = a.total_tiles ? (int)*a.total_tiles : a.total_tiles_host;
    const size_t S = (size_t)a.n_per_view * a.nviews;
    for (;;) {
        if (tid == 0) {
            s_tile = (int)atomicAdd(a.work, 1u);
            s_maxlc = -1;
        }
        __syncthreads();
        const int tile = s_tile;
        if (tile >= total_tiles) break;
        const int v = find_view(a.cams, a.nviews, tile);
        const DevCam& c = a.cams[v];
        const int lt = tile - c.tile_base;
        const int tx = lt % c.tiles_x, ty = lt / c.tiles_x;
        const int px = tx * TW + (tid % TW), py0 = ty * TH + (tid / TW) * PPT;
        const float pxf = (float)px + 0.5f;
        const float x0c = (float)(tx * TW) + 0.5f, x1c = (float)(min(tx * TW + TW, c.width) - 1) + 0.5f;
        const uint2 rg = a.ranges[tile];
        int lc[PPT];
        float2 T[H], d0[H], d1[H], d2[H], nsb[H], pyc[H];
        int my_maxlc = -1;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            float t[2], e0[2], e1[2], e2[2], sb[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int py = py0 + 2 * h + j;
                int l = -1;
                t[j] = e0[j] = e1[j] = e2[j] = 0.0f;
                if (px < c.width && py < c.height) {
                    const size_t pix = (size_t)c.pix_base + (size_t)py * c.width + px;
                    l = a.last[pix];
                    t[j] = a.final_t[pix];
                    e0[j] = a.dl[pix * 3 + 0];
                    e1[j] = a.dl[pix * 3 + 1];
                    e2[j] = a.dl[pix * 3 + 2];
                }
                // dL/dpixel . (colour behind the current splat), behind = T_final * bg
                sb[j] = __fmaf_rn(e2[j], t[j] * a.bg[2], __fmaf_rn(e1[j], t[j] * a.bg[1], e0[j] * (t[j] * a.bg[0])));
                lc[2 * h + j] = l;
                my_maxlc = max(my_maxlc, l);
            }
            T[h] = make_float2(t[0], t[1]);
            d0[h] = make_float2(e0[0], e0[1]);
            d1[h] = make_float2(e1[0], e1[1]);
            d2[h] = make_float2(e2[0], e2[1]);
            nsb[h] = make_float2(-sb[0], -sb[1]);
            pyc[h] = make_float2((float)(py0 + 2 * h) + 0.5f, (float)(py0 + 2 * h) + 1.5f);
        }
        const int warp_maxlc = __reduce_max_sync(0xffffffffu, my_maxlc);
        if (lane == 0 && warp_maxlc >= 0) atomicMax(&s_maxlc, warp_maxlc);
        __syncthreads();
        const int maxlc = s_maxlc;
        for (int hi_li = maxlc; hi_li >= 0; hi_li -= BWD_BATCH) {
            const int lo = max(hi_li - BWD_BATCH + 1, 0);
            // ---- stage list entries [lo, hi_li], each with the mask of the warps
            // whose strip of pixel rows it can reach
            for (int j = tid; j < BWD_BATCH; j += NT) {
                uint32_t wm = 0;
                if (lo + j <= hi_li) {
                    const uint32_t slot = a.pair_vals[rg.x + (uint32_t)(lo + j)];
                    const float4 A = a.rec[slot];
                    const float4 Q = a.rec[S + slot];
                    const float4 K = a.rec[2 * S + slot];
                    const float thr = power_floor(A.z);
                    const TileTest t = tile_test_setup(A.x, A.y, Q.x, Q.y, Q.z, thr);
#pragma unroll
                    for (int ww = 0; ww < NW; ++ww) {
                        const int r0 = ty * TH + ww * RW;
                        if (r0 >= c.height) continue;
                        const float sy0 = (float)r0 + 0.5f, sy1 = (float)(min(r0 + RW, c.height) - 1) + 0.5f;
                        if (!tile_rejects(t, x0c, x1c, sy0, sy1)) wm |= 1u << ww;
                    }
                    if (wm) {
                        const float lop = log2f(A.z);
                        s_a[j] = make_float4(A.x, A.y, lop, A.z);
                        // a conic or colour outside any sane range (NaN and inf among
                        // them) sends every pixel to the exact arithmetic
                        const float mag = fabsf(Q.x) + fabsf(Q.y) + fabsf(Q.z) + fabsf(K.x) + fabsf(K.y) + fabsf(K.z);
                        s_c[j] = make_float4(Q.x, Q.y, Q.z, mag <= 1e25f ? fminf(L099, lop) - BWD_BAND : __int_as_float(0x7fc00000));
                        s_k[j] = make_float4(K.x, K.y, K.z, thr);
                        s_slot[j] = slot;
                        if (RECT) s_r[j] = make_uint2(__float_as_uint(Q.w), __float_as_uint(K.w));
                    }
                }
                s_wm[j] = (uint8_t)wm;
            }
            __syncthreads();
            // ---- this warp's entries, back to front
            int cnt = 0, my_k = 0;
            auto flush = [&]() {
                __syncwarp();
                const int g = lane & (BWD_GRP - 1), q = lane / BWD_GRP;
                const float4 ctr = s_a[my_k], cq = s_c[my_k];
                const uint32_t slot = s_slot[my_k];
                float dx = ((float)(tx * TW + (q * 8) % TW) + 0.5f) - ctr.x;
                float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, u0 = 0.0f, u1 = 0.0f, u2 = 0.0f, w0 = 0.0f, w1 = 0.0f, w2 = 0.0f;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int l = (q * 8 + e) ^ g;
                    const float4 f = s_b4[warp][g][l];
                    const float2 f2 = s_b2[warp][g][l];
                    c0 += f.x;
                    c1 += f.y;
                    c2 += f.z;
                    const float du = dx * f.w;
                    u0 += f.w;
                    u1 += du;
                    u2 = __fmaf_rn(du, dx, u2);
                    w0 += f2.x;
                    w1 = __fmaf_rn(dx, f2.x, w1);
                    w2 += f2.y;
                    dx += 1.0f;
                }
#pragma unroll
                for (int o = BWD_GRP; o < 32; o <<= 1) {
                    c0 += __shfl_xor_sync(0xffffffffu, c0, o);
                    c1 += __shfl_xor_sync(0xffffffffu, c1, o);
                    c2 += __shfl_xor_sync(0xffffffffu, c2, o);
                    u0 += __shfl_xor_sync(0xffffffffu, u0, o);
                    u1 += __shfl_xor_sync(0xffffffffu, u1, o);
                    u2 += __shfl_xor_sync(0xffffffffu, u2, o);
                    w0 += __shfl_xor_sync(0xffffffffu, w0, o);
                    w1 += __shfl_xor_sync(0xffffffffu, w1, o);
                    w2 += __shfl_xor_sync(0xffffffffu, w2, o);
                }
                // the sums are of negated terms
                if (g < cnt) {
                    if (q == 0) red_add_v4(a.acc + slot, -c0, -c1, -c2, -u0 / ctr.w);
                    if (q == 1) red_add_v4(a.acc + S + slot, 0.5f * u2, w1, 0.5f * w2, -__fmaf_rn(cq.y, w0, cq.x * u1));
                    if (q == 2) red_add_v4(a.acc + 2 * S + slot, -__fmaf_rn(cq.z, w0, cq.y * u1), 0.0f, 0.0f, 0.0f);
                }
                __syncwarp();
                cnt = 0;
            };
#pragma unroll 1
            for (int half = BWD_BATCH / 32 - 1; half >= 0; --half) {
                const int kk = half * 32 + lane;
                unsigned todo = __ballot_sync(0xffffffffu, ((s_wm[kk] >> warp) & 1u) && lo + kk <= warp_maxlc);
                while (todo) {
                    const int b = 31 - __clz(todo);
                    todo ^= 1u << b;
                    const int k = half * 32 + b;
                    const int li = lo + k;
                    const float4 A = s_a[k];
                    const float4 Q = s_c[k];
                    const float dx = pxf - A.x;
                    const float tdx = Q.x * dx * dx;
                    const float t2b = 2.0f * Q.y * dx;
                    float2 dy[H], nal[H], um[H];
                    bool any = false, sure = true;
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        dy[h] = __fadd2_rn(pyc[h], bc2(-A.y));
                        // -2 power = (tdx + t2b dy) + (c dy) dy
                        const float2 s1 = __ffma2_rn(__fmul2_rn(bc2(t2b), dy[h]), one2, bc2(tdx));
                        const float2 s2 = __ffma2_rn(__fmul2_rn(__fmul2_rn(bc2(Q.z), dy[h]), dy[h]), one2, s1);
                        const float2 p = __ffma2_rn(s2, bc2(-0.5f * LOG2E), bc2(A.z));
                        const float2 d = __fadd2_rn(p, bc2(L255));
                        bool a0 = li <= lc[2 * h], a1 = li <= lc[2 * h + 1];
                        if (RECT) {
                            const uint2 r = s_r[k];
                            a0 = a0 && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h);
                            a1 = a1 && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h + 1);
                        }
                        sure = sure && fminf(fabsf(d.x), fabsf(d.y)) >= BWD_BAND && fmaxf(p.x, p.y) <= Q.w;
                        a0 = a0 && d.x > 0.0f;
                        a1 = a1 && d.y > 0.0f;
                        any = any || a0 || a1;
                        const float e0 = ex2_sfu(p.x), e1 = ex2_sfu(p.y);
                        nal[h] = make_float2(a0 ? -e0 : 0.0f, a1 ? -e1 : 0.0f);
                        um[h] = nal[h];
                    }
                    float4 K = s_k[k];
                    if (!sure) {
                        const float4 q = make_float4(Q.x, Q.y, Q.z, A.w);
#pragma unroll
                        for (int h = 0; h < H; ++h) {
                            const float2 zero = make_float2(0.0f, 0.0f);
                            bool a0 = li <= lc[2 * h], a1 = li <= lc[2 * h + 1];
                            if (RECT) {
                                const uint2 r = s_r[k];
                                a0 = a0 && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h);
                                a1 = a1 && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h + 1);
                            }
                            const float2 x0 = a0 ? bwd_exact_pixel(dx, dy[h].x, q, K.w) : zero;
                            const float2 x1 = a1 ? bwd_exact_pixel(dx, dy[h].y, q, K.w) : zero;
                            nal[h] = make_float2(x0.x, x1.x);
                            um[h] = make_float2(x0.y, x1.y);
                            any = any || x0.x != 0.0f || x1.x != 0.0f;
                        }
                        // a colour that is not finite reaches no pixel that does not take it
                        if (!any) K = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                    if (!__any_sync(0xffffffffu, any)) continue;
                    float2 G0, G1, G2, SU, SUD, SUDD;
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        // a pixel that does not take the splat has alpha = 0: 1 - alpha = 1
                        // and rcp(1) = 1 leave its T and behind-colour sum as they are, and
                        // its terms are zero
                        const float2 om = __fadd2_rn(one2, nal[h]);
                        float2 inv;
                        if (STORE) {
                            // store-all variant: T before this splat as the forward saw it
                            const float* ts = a.tstore + (size_t)(rg.x + (uint32_t)li) * (TW * TH) + ((tid / TW) * PPT + 2 * h) * TW + tid % TW;
                            if (nal[h].x != 0.0f) T[h].x = ts[0];
                            if (nal[h].y != 0.0f) T[h].y = ts[TW];
                            inv = make_float2(1.0f / om.x, 1.0f / om.y);
                        } else {
                            inv = make_float2(rcp_sfu(om.x), rcp_sfu(om.y));
                            T[h] = __fmul2_rn(T[h], inv);
                        }
                        const float2 nw = __fmul2_rn(nal[h], T[h]);
                        const float2 dk = __ffma2_rn(d2[h], bc2(K.z), __ffma2_rn(d1[h], bc2(K.y), __fmul2_rn(d0[h], bc2(K.x))));
                        const float2 dda = __ffma2_rn(T[h], dk, __fmul2_rn(nsb[h], inv));
                        nsb[h] = __ffma2_rn(nw, dk, nsb[h]);
                        const float2 nu = __fmul2_rn(dda, um[h]);
                        const float2 nud = __fmul2_rn(nu, dy[h]);
                        if (h == 0) {
                            G0 = __fmul2_rn(d0[h], nw);
                            G1 = __fmul2_rn(d1[h], nw);
                            G2 = __fmul2_rn(d2[h], nw);
                            SU = nu;
                            SUD = nud;
                            SUDD = __fmul2_rn(nud, dy[h]);
                        } else {
                            G0 = __ffma2_rn(d0[h], nw, G0);
                            G1 = __ffma2_rn(d1[h], nw, G1);
                            G2 = __ffma2_rn(d2[h], nw, G2);
                            SU = __fadd2_rn(SU, nu);
                            SUD = __fadd2_rn(SUD, nud);
                            SUDD = __ffma2_rn(nud, dy[h], SUDD);
                        }
                    }
                    s_b4[warp][cnt][lane ^ cnt] = make_float4(G0.x + G0.y, G1.x + G1.y, G2.x + G2.y, SU.x + SU.y);
                    s_b2[warp][cnt][lane ^ cnt] = make_float2(SUD.x + SUD.y, SUDD.x + SUDD.y);
                    if ((lane & (BWD_GRP - 1)) == cnt) my_k = k;
                    if (++cnt == BWD_GRP) flush();
                }
            }
            if (cnt) flush();
            __syncthreads();
        }
        __syncthreads();  // every thread has read s_tile / s_maxlc before thread 0 rewrites them
    }
}

// ---- launch plumbing -----------------------------------------------------
typedef void (*BlendKernel)(BlendArgs);

// The forward runs `pixels_per_thread` (1 or 2) pixels per thread, the
// backward twice that: its per-splat warp reduction is then shared by twice
// the pixels (measured 3 % faster at 4 than at 2 on the 1M-Gaussian step,
// while the forward is slower at 4).
template <int TW, int TH, int BATCH, bool RECT>
static BlendKernel pick(bool fwd, int ppt) {
    if (fwd) return ppt == 1 ? (BlendKernel)k_blend_fwd<TW, TH, BATCH, RECT, 1> : (BlendKernel)k_blend_fwd<TW, TH, BATCH, RECT, 2>;
    return ppt == 2 ? (BlendKernel)k_blend_bwd<TW, TH, RECT, 2> : (BlendKernel)k_blend_bwd<TW, TH, RECT, 4>;
}

template <int TW, int TH, bool RECT>
static BlendKernel pick_batch(int batch, bool fwd, int ppt) {
    switch (batch) {
        case 128: return pick<TW, TH, 128, RECT>(fwd, ppt);
        case 512: return pick<TW, TH, 512, RECT>(fwd, ppt);
        default: return pick<TW, TH, 256, RECT>(fwd, ppt);
    }
}

static BlendKernel select_kernel(int tw, int th, int batch, bool rect, bool fwd, int ppt) {
    if (tw == 8 && th == 32) return pick_batch<8, 32, true>(batch, fwd, ppt);
    if (tw == 32 && th == 8) return pick_batch<32, 8, true>(batch, fwd, ppt);
    return rect ? pick_batch<16, 16, true>(batch, fwd, ppt) : pick_batch<16, 16, false>(batch, fwd, ppt);
}

// Persistent grid of a blend kernel on the current device: SMs x resident CTAs,
// cached per (kernel, device ordinal).
static int grid_for(BlendKernel k, int threads) {
    struct Entry { BlendKernel k; int dev; int grid; };
    static std::mutex mu;
    static Entry cache[256];
    static int ncache = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    const int sms = device_sm_count();
    std::lock_guard<std::mutex> g(mu);
    for (int i = 0; i < ncache; ++i)
        if (cache[i].k == k && cache[i].dev == dev) return cache[i].grid;
    int per = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, (const void*)k, threads, 0) != cudaSuccess) {
        cudaGetLastError();
        per = 1;
    }
    int grid = sms * std::max(per, 1);
    if (ncache < 256) cache[ncache++] = {k, dev, grid};
    return grid;
}

static void launch(const BlendArgs& a, int tw, int th, int batch, bool fwd, cudaStream_t st) {
    bool rect = a.rect_filter != 0 || !(tw == REF_TILE && th == REF_TILE);
    int ppt = (a.pixels_per_thread == 1 ? 1 : 2) * (fwd ? 1 : 2);
    BlendKernel k = select_kernel(tw, th, batch, rect, fwd, ppt);
    int threads = tw * th / ppt;
    cudaMemsetAsync(a.work, 0, sizeof(uint32_t), st);
    int grid = grid_for(k, threads);
    if (!a.total_tiles) grid = std::min(grid, std::max(a.total_tiles_host, 1));
    k<<<grid, threads, 0, st>>>(a);
}

// (pixel, splat) pairs the blend evaluates, per pixel of view blockIdx.y: the
// forward walks the pixel's tile list until T < 1e-4 ends it at its last
// contributor (final T below 1e-4) or the list runs out; the backward walks
// from the last contributor down to the front. out[0] += forward pairs,
// out[1] += backward pairs.
__global__ void __launch_bounds__(256) k_evaluated_pairs(const DevCam* __restrict__ cams, const uint2* __restrict__ ranges,
                                                         const float* __restrict__ final_t, const int* __restrict__ last,
                                                         int tile_w, int tile_h, unsigned long long* out) {
    const DevCam& c = cams[blockIdx.y];
    const uint32_t px = (uint32_t)c.width * (uint32_t)c.height;
    unsigned long long f = 0, b = 0;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < px; p += gridDim.x * blockDim.x) {
        const uint32_t x = p % (uint32_t)c.width, y = p / (uint32_t)c.width;
        const uint2 r = ranges[c.tile_base + (y / tile_h) * c.tiles_x + x / tile_w];
        const int l = last[(size_t)c.pix_base + p];
        const float t = final_t[(size_t)c.pix_base + p];
        f += t < 1e-4f ? (unsigned long long)(l + 1) : (unsigned long long)(r.y - r.x);
        b += l >= 0 ? (unsigned long long)(l + 1) : 0ull;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        f += __shfl_down_sync(0xffffffffu, f, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if ((threadIdx.x & 31) == 0 && (f | b)) {
        atomicAdd(out, f);
        atomicAdd(out + 1, b);
    }
}

// Largest |exp_sfu_nonpos(x) / expf_fast_nonpos(x) - 1| over n points spaced
// evenly on [lo, hi] (hi <= 0), as float bits in *out (non-negative floats
// order like their bits).
__global__ void k_exp_sfu_error(float lo, float hi, uint32_t n, unsigned int* out) {
    float m = 0.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float x = lo + (hi - lo) * ((float)i / (float)(n > 1 ? n - 1 : 1));
        const float e = expf_fast_nonpos(x);
        m = fmaxf(m, fabsf(exp_sfu_nonpos(x) / e - 1.0f));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(m));
}

void launch_exp_sfu_error(float lo, float hi, uint32_t n, unsigned int* out, cudaStream_t st) {
    k_exp_sfu_error<<<device_sm_count() * 4, 256, 0, st>>>(lo, hi, n, out);
}

void launch_evaluated_pairs(const DevCam* cams, int nviews, const uint2* ranges, const float* final_t, const int* last,
                            int tile_w, int tile_h, unsigned long long* out, cudaStream_t st) {
    if (nviews <= 0) return;
    k_evaluated_pairs<<<dim3((unsigned)device_sm_count() * 2, (unsigned)nviews), 256, 0, st>>>(cams, ranges, final_t, last,
                                                                                            tile_w, tile_h, out);
}

void launch_blend_forward(const BlendArgs& a, int tw, int th, int batch, cudaStream_t st) { launch(a, tw, th, batch, true, st); }
void launch_blend_backward(const BlendArgs& a, int tw, int th, int batch, cudaStream_t st) { launch(a, tw, th, batch, false, st); }

// Store-all variant (16x16 tiles, 256-splat batches, 2 pixels per thread): the
// forward writes T before every contributing splat of every pixel to
// a.tstore[(list position) * 256 + pixel in tile], the backward reads it back
// instead of rebuilding T from the final T.
void launch_blend_store_all(const BlendArgs& a, bool fwd, cudaStream_t st) {
    BlendKernel k = fwd ? (BlendKernel)k_blend_fwd<16, 16, 256, false, 2, true> : (BlendKernel)k_blend_bwd<16, 16, false, 2, true>;
    cudaMemsetAsync(a.work, 0, sizeof(uint32_t), st);
    int grid = grid_for(k, 128);
    if (!a.total_tiles) grid = std::min(grid, std::max(a.total_tiles_host, 1));
    k<<<grid, 128, 0, st>>>(a);
}

}  // namespace rgs
