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
// B200 mapping: one CTA per CTA tile (TW x TH pixels, two or four pixels per
// thread in packed f32x2 lanes), persistent CTAs pulling tiles of every view of
// the batch from one atomic counter. Splat records are staged one per thread at
// a time in shared memory, fetched asynchronously a batch ahead, and read by
// all threads as broadcasts. Work that the reference's own tests would discard
// is removed without changing any result:
//   * per splat, alpha < 1/255 is guaranteed once power < thr with
//     thr = ln(1 / (255 opacity)) - 0.01, so such pixels skip exp;
//   * per (warp, staged splat), if the conic's quadratic form is bounded below
//     over the box of the pixel centres of the warp's own strip of rows so that
//     power < thr everywhere, the warp never visits the splat: it walks a bit
//     mask of the ones it can reach;
//   * backward warps skip splats past the warp's largest last_contrib.
// Backward gathers each warp's partial gradients of eight splats in shared
// memory, reads them back transposed (four lanes per splat) and adds 48 bytes per
// splat and warp to global memory: colour and opacity as one red.v4.f32, the
// conic's three sums in 64 bits, the mean as a red.v2.f32.
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

// ---- staging ---------------------------------------------------------------
// A tile's list is staged in batches of one entry per thread. The records of a
// batch arrive by 16-byte asynchronous copies into one of two shared-memory
// buffers while the previous batch is blended (and the list entries of the
// batch after that are read), so the gather's latency, from DRAM where the
// records outgrow L2, is off the blend's path; then each thread tests its own
// entry in place.
constexpr uint32_t NO_SLOT = 0xffffffffu;

__device__ __forceinline__ void copy16(float4* dst, const float4* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// Starts the copies of this thread's entry (none for NO_SLOT) as one group.
__device__ __forceinline__ void fetch_entry(const BlendArgs& a, size_t S, uint32_t slot, float4* A, float4* Q, float4* K) {
    if (slot != NO_SLOT) {
        copy16(A, a.rec + slot);
        copy16(Q, a.rec + S + slot);
        copy16(K, a.rec + 2 * S + slot);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// Waits for this thread's copies, all but the newest LATER groups.
template <int LATER>
__device__ __forceinline__ void fetch_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(LATER) : "memory");
}

// The warps whose strip of pixel rows (RW rows of the tile each) a splat can
// reach: the tile test on the strip's pixel centres (strips past the image hold
// no pixel).
template <int NW, int RW>
__device__ __forceinline__ uint32_t reached_warps(const float4& A, const float4& Q, float thr, float x0c, float x1c, int ytile,
                                                  int height) {
    const TileTest t = tile_test_setup(A.x, A.y, Q.x, Q.y, Q.z, thr);
    uint32_t wm = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        const int r0 = ytile + w * RW;
        if (r0 >= height) continue;
        const float y0 = (float)r0 + 0.5f, y1 = (float)(min(r0 + RW, height) - 1) + 0.5f;
        if (!tile_rejects(t, x0c, x1c, y0, y1)) wm |= 1u << w;
    }
    return wm;
}

// A conic or colour outside any sane range (NaN and inf among them).
__device__ __forceinline__ bool not_sane(const float4& Q, const float4& K) {
    return !(fabsf(Q.x) + fabsf(Q.y) + fabsf(Q.z) + fabsf(K.x) + fabsf(K.y) + fabsf(K.z) <= 1e25f);
}

// Forward. A thread owns PPT vertical pixels in packed f32x2 lanes, each lane
// rounded exactly as the reference rounds that pixel. A pixel that does not
// take a splat gets alpha = 0: +0 is added to its non-negative colour sums and
// its T is multiplied by 1, bit-identical to skipping it. (A splat whose conic
// or colour is not finite goes through a scalar loop, so 0 * NaN reaches no
// pixel that does not take it.)
//
// What bounds it: the FMA pipe (73 % of cycles; two thirds of its work is the
// reference's exact exponential, 18 packed instructions per pixel pair), so what
// matters is not to evaluate pairs that cannot contribute. Each warp walks the
// bit mask of the staged splats that can reach its own strip of rows (about half
// of the (strip, splat) pairs of a tile's list cannot), formed by one ballot per
// 32 splats from the strip tests of the thread that staged each. A warp whose
// pixels all pass by a splat asks whether any is still alive, else it is done; the
// tile ends before the first batch that finds no pixel of it alive. (That vote on
// the warps' own flags ended no tile with a strip below the image: an opaque scene at
// 1600x1064, two thirds of a tile row, took 260 us, now 106. A warp that starts out
// done where its strip is below the image cost all others 1 to 3 %.)
//
// Measured (1M Gaussians x 8 views): 1.80 ms for the loop that compacted each
// batch by the tile test and visited every kept splat; 1.42 ms now. 97k x 3
// views of 1277x719, white background: 645 -> 525 us; 3M anisotropic x 8 views
// of 1920x1080, where the records come from DRAM: 4.14 -> 3.98 ms (4.55 without
// the asynchronous fetch). Twelve CTAs per SM; 10, 14 and 16 were 2 %, 0.5 % and
// 3 % slower. Also slower: strips of 16x4 with a branch per pixel pair (+13 %:
// the two pairs' independent chains are what hides latency), per-row terms of
// the power precomputed in shared memory (+4 %), a branch per thread (+1 %), the
// alive test after every fourth idle splat instead of each (0 to +1 %).
template <int TW, int TH, bool RECT, int PPT, bool STORE = false>
__global__ void __launch_bounds__(TW * TH / PPT, PPT == 2 ? 6 : 12) k_blend_fwd(BlendArgs a) {
    constexpr int NT = TW * TH / PPT;
    constexpr int NW = NT / 32;
    constexpr int H = PPT / 2;
    constexpr int RW = (32 / TW) * PPT;  // pixel rows per warp
    const float2 one2 = make_float2(a.one, a.one);
    __shared__ float4 s_a2[2][NT];  // sx, sy, opacity, -2 x power floor
    __shared__ float4 s_c2[2][NT];  // a, b, c, 0 or NaN (take the scalar loop)
    __shared__ float4 s_k2[2][NT];  // colour
    __shared__ uint2 s_r[RECT ? NT : 1];
    __shared__ uint8_t s_wm[NT];
    __shared__ int s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
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
        const float x0c = (float)(tx * TW) + 0.5f, x1c = (float)(min(tx * TW + TW, c.width) - 1) + 0.5f;
        const uint2 rg = a.ranges[tile];
        // a pixel is done once its T is below 1e-4; those outside the image start there
        float2 T[H], C0[H], C1[H], C2[H], pyc[H];
        int last[PPT];
        bool seen[PPT];
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const int py = py0 + 2 * h;
            pyc[h] = make_float2((float)py + 0.5f, (float)py + 1.5f);
            T[h] = make_float2(px < c.width && py < c.height ? 1.0f : 0.0f, px < c.width && py + 1 < c.height ? 1.0f : 0.0f);
            C0[h] = bc2(a.bg_start ? a.bg[0] : 0.0f);
            C1[h] = bc2(a.bg_start ? a.bg[1] : 0.0f);
            C2[h] = bc2(a.bg_start ? a.bg[2] : 0.0f);
            last[2 * h] = last[2 * h + 1] = -1;
            // whether the pixel's reference tile list is non-empty
            seen[2 * h] = seen[2 * h + 1] = !RECT && rg.y > rg.x;
        }
        bool done = false;  // warp-uniform: every pixel of the warp is done
        const bool need_seen = RECT && a.empty_tile_black;
        auto entry = [&](uint32_t i) { return i < rg.y ? a.pair_vals[i] : NO_SLOT; };
        uint32_t here = entry(rg.x + tid), next = entry(rg.x + NT + tid);
        fetch_entry(a, S, here, &s_a2[0][tid], &s_c2[0][tid], &s_k2[0][tid]);
        int buf = 0;
        for (uint32_t b0 = rg.x; b0 < rg.y; b0 += NT, buf ^= 1) {
            bool alive = false;
#pragma unroll
            for (int h = 0; h < H; ++h) alive = alive || !(T[h].x < 1e-4f) || !(T[h].y < 1e-4f);
            if (__syncthreads_and(!alive)) break;
            fetch_entry(a, S, next, &s_a2[buf ^ 1][tid], &s_c2[buf ^ 1][tid], &s_k2[buf ^ 1][tid]);
            float4* s_a = s_a2[buf];
            float4* s_c = s_c2[buf];
            float4* s_k = s_k2[buf];
            fetch_wait<1>();
            uint32_t wm = 0;
            if (here != NO_SLOT) {
                const float4 A = s_a[tid], Q = s_c[tid], K = s_k[tid];
                const float thr = power_floor(A.z);
                wm = reached_warps<NW, RW>(A, Q, thr, x0c, x1c, ty * TH, c.height);
                if (RECT) s_r[tid] = make_uint2(__float_as_uint(Q.w), __float_as_uint(K.w));
                s_a[tid].w = -2.0f * thr;
                s_c[tid].w = not_sane(Q, K) ? __int_as_float(0x7fc00000) : 0.0f;
            }
            s_wm[tid] = (uint8_t)wm;
            here = next;
            next = entry(b0 + 2 * NT + tid);
            __syncthreads();
            if (need_seen) {
                // a pixel's reference tile list is non-empty iff some entry (kept
                // or rejected) covers the pixel
                const int staged = (int)min((uint32_t)NT, rg.y - b0);
#pragma unroll
                for (int p = 0; p < PPT; ++p)
                    for (int j = 0; j < staged && !seen[p]; ++j)
                        if (in_rect(__uint_as_float(s_r[j].x), __uint_as_float(s_r[j].y), px, py0 + p)) seen[p] = true;
            }
            if (done) continue;
#pragma unroll 1
            for (int part = 0; part < NT / 32 && !done; ++part) {
                unsigned todo = __ballot_sync(0xffffffffu, (s_wm[part * 32 + lane] >> warp) & 1u);
                while (todo) {
                    const int k = part * 32 + __ffs(todo) - 1;
                    todo &= todo - 1;
                    const float4 A = s_a[k];
                    const float4 Q = s_c[k];
                    const float dx = pxf - A.x;
                    const float tdx = Q.x * dx * dx;
                    const float t2b = 2.0f * Q.y * dx;
                    float2 y[H];  // -2 power
                    bool act[PPT];
                    bool any = false;
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float2 dy = __fadd2_rn(pyc[h], bc2(-A.y));
                        // power = -0.5 * ((tdx + t2b * dy) + qdd)
                        const float2 s1 = __ffma2_rn(__fmul2_rn(bc2(t2b), dy), one2, bc2(tdx));
                        y[h] = __ffma2_rn(__fmul2_rn(__fmul2_rn(bc2(Q.z), dy), dy), one2, s1);
                        act[2 * h] = !(T[h].x < 1e-4f) && !(y[h].x < 0.0f) && !(y[h].x > A.w);
                        act[2 * h + 1] = !(T[h].y < 1e-4f) && !(y[h].y < 0.0f) && !(y[h].y > A.w);
                        if (RECT) {
                            const uint2 r = s_r[k];
                            act[2 * h] = act[2 * h] && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h);
                            act[2 * h + 1] = act[2 * h + 1] && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h + 1);
                        }
                        any = any || act[2 * h] || act[2 * h + 1];
                    }
                    if (!__any_sync(0xffffffffu, any)) {
                        bool alive = false;
#pragma unroll
                        for (int h = 0; h < H; ++h) alive = alive || !(T[h].x < 1e-4f) || !(T[h].y < 1e-4f);
                        if (!__any_sync(0xffffffffu, alive)) {
                            done = true;
                            break;
                        }
                        continue;
                    }
                    const float4 K = s_k[k];
                    const int li = (int)(b0 - rg.x) + k;
                    if (Q.w != Q.w) {
                        // not finite: pixel by pixel
#pragma unroll
                        for (int p = 0; p < PPT; ++p) {
                            if (!act[p]) continue;
                            float& t = (p & 1) ? T[p / 2].y : T[p / 2].x;
                            const float alpha = fminf(A.z * expf_fast_nonpos(-0.5f * ((p & 1) ? y[p / 2].y : y[p / 2].x)), 0.99f);
                            if (alpha < 1.0f / 255.0f) continue;
                            if (STORE) a.tstore[(size_t)(rg.x + (uint32_t)li) * (TW * TH) + ((tid / TW) * PPT + p) * TW + tid % TW] = t;
                            const float w = alpha * t;
                            float& c0 = (p & 1) ? C0[p / 2].y : C0[p / 2].x;
                            float& c1 = (p & 1) ? C1[p / 2].y : C1[p / 2].x;
                            float& c2 = (p & 1) ? C2[p / 2].y : C2[p / 2].x;
                            c0 += K.x * w;
                            c1 += K.y * w;
                            c2 += K.z * w;
                            t *= 1.0f - alpha;
                            last[p] = li;
                        }
                        continue;
                    }
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float2 ar = __fmul2_rn(bc2(A.z), expf_fast_neghalf2(y[h], one2));
                        float2 al = make_float2(fminf(ar.x, 0.99f), fminf(ar.y, 0.99f));
                        const bool t0 = act[2 * h] && !(al.x < 1.0f / 255.0f), t1 = act[2 * h + 1] && !(al.y < 1.0f / 255.0f);
                        if (STORE) {
                            float* ts = a.tstore + (size_t)(rg.x + (uint32_t)li) * (TW * TH) + ((tid / TW) * PPT + 2 * h) * TW + tid % TW;
                            if (t0) ts[0] = T[h].x;
                            if (t1) ts[TW] = T[h].y;
                        }
                        al = make_float2(t0 ? al.x : 0.0f, t1 ? al.y : 0.0f);
                        const float2 w = __fmul2_rn(al, T[h]);
                        C0[h] = __ffma2_rn(__fmul2_rn(bc2(K.x), w), one2, C0[h]);
                        C1[h] = __ffma2_rn(__fmul2_rn(bc2(K.y), w), one2, C1[h]);
                        C2[h] = __ffma2_rn(__fmul2_rn(bc2(K.z), w), one2, C2[h]);
                        T[h] = __fmul2_rn(T[h], __ffma2_rn(al, make_float2(-one2.x, -one2.y), one2));
                        last[2 * h] = t0 ? li : last[2 * h];
                        last[2 * h + 1] = t1 ? li : last[2 * h + 1];
                    }
                }
            }
        }
        fetch_wait<0>();  // a batch fetched ahead lands before its buffer is used again
#pragma unroll
        for (int p = 0; p < PPT; ++p) {
            const int py = py0 + p;
            if (px < c.width && py < c.height) {
                const size_t pix = (size_t)c.pix_base + (size_t)py * c.width + px;
                const float t = (p & 1) ? T[p / 2].y : T[p / 2].x;
                const float c0 = (p & 1) ? C0[p / 2].y : C0[p / 2].x;
                const float c1 = (p & 1) ? C1[p / 2].y : C1[p / 2].x;
                const float c2 = (p & 1) ? C2[p / 2].y : C2[p / 2].x;
                // forward_pass skips tiles whose list is empty, leaving their pixels
                // at 0 rather than bg (src/cpu/backward.rs:313-315, 124)
                const bool black = a.empty_tile_black && !seen[p];
                // no splat taken: the sums are still bg (a -0.0 bg included)
                const bool bare = a.bg_start && last[p] < 0;
                a.rgb[pix * 3 + 0] = black ? 0.0f : bare ? a.bg[0] : a.bg_start ? c0 : c0 + t * a.bg[0];
                a.rgb[pix * 3 + 1] = black ? 0.0f : bare ? a.bg[1] : a.bg_start ? c1 : c1 + t * a.bg[1];
                a.rgb[pix * 3 + 2] = black ? 0.0f : bare ? a.bg[2] : a.bg_start ? c2 : c2 + t * a.bg[2];
                a.final_t[pix] = t;
                a.last[pix] = last[p];
            }
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void red_add_v4(float4* addr, float x, float y, float z, float w) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

__device__ __forceinline__ void red_add_v2(float2* addr, float x, float y) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(x), "f"(y) : "memory");
}

__device__ __forceinline__ void red_add_f64(double* addr, double x) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(addr), "d"(x) : "memory");
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
// What bounds it: instruction issue (78 % of cycles; FMA pipe 59 %, ALU 39 %),
// so the loop is built around the fewest instructions per (warp, splat). It
// replaces a loop that tested both thresholds on each pixel's alpha and reduced
// nine sums over the warp for every splat: 3.29 -> 1.52 ms on 1M Gaussians x 8
// views, 1.57 -> 0.57 ms on 97k x 3 views of 1277x719 with a white background,
// 262 -> 52 us on 10k at 256x256 (where one tile's serial walk is the time).
//
// Alpha is the opacity times one SFU exponential of t = power log2(e), with the
// power rounded exactly as the forward rounds it. (A power from two
// packed FMAs over prescaled coefficients saves four packed instructions per
// pixel pair and ran 4 % faster; but an ill-conditioned conic's terms cancel,
// and its alpha then strays from the forward's by up to 1e-4. The opacity as
// log2(opacity) in the exponent saves one; but its rounding, up to 3e-7 of
// alpha, is then every pixel's.) The
// contributing set must be the forward's exactly, so a pixel whose t lies
// within BWD_BAND of a decision (alpha >= 1/255; alpha_raw > 0.99; power > 0)
// is decided by bwd_exact_pixel: the roundings of t (|t| <= 8), of the limits
// and of the forward's own alpha add up to less than 2e-6 in log2 units, half
// the band. A NaN conic, colour or opacity makes the limit NaN, and every pixel
// of that splat is decided exactly.
//
// The nine gradient sums of a splat are not reduced across the warp per splat
// (14 shuffles and two shared atomics each, serialised): a lane stores its six
// column sums (colour x3, u, u dy, u dy^2 with u = dL/dpower) for up to
// BWD_GRP splats in the warp's own shared memory, then the warp reads them
// transposed, four lanes per splat, each adding eight columns, expands the
// moments in dx, and adds them to the slot's sums with three reductions. Those of
// the conic are 64-bit: across tiles they add up in any order, and the geometry's
// gradient is a difference of them that cancels by the covariance's condition
// number; in 32 bits, two passes over a scene of needles differed by the whole of
// their rotations' gradient, and over 3M anisotropic Gaussians by 1 to 5 % of all
// gradients (now 5e-7; the same time, 6.18 ms a step of 1M x 8 views and 31.7 of
// 3M). The stores and loads are swizzled by the splat's place in the group, so neither
// has bank conflicts. Warps share only the staged batch and the two barriers
// around it.
//
// Every lane of a warp that some lane's pixels need runs the whole update (its
// terms are zero); a branch per thread ran 4 % slower. Nine CTAs per SM with
// four pixels per thread: 8, 10 and 11 ran 9 %, 5 % and 7 % slower.
// Also measured slower: coefficients stored twice so that a 16-byte load fills
// both lanes of two operands (+9 %), the next splat's coefficients loaded ahead
// (+9 %), the next batch's records prefetched into L1 instead of copied (+8 %),
// one strip per packed pair with a branch each (+18 %).
constexpr float BWD_BAND = 4e-6f;
constexpr int BWD_GRP = 8;

// A splat's limits on t: it contributes where t + reach > 0; up to `limit` its raw
// alpha is at most 0.99 and its power at most 0.
struct BwdLimits {
    float reach, limit;
};
__device__ __forceinline__ BwdLimits bwd_limits(float opacity) {
    const float lop = log2f(opacity);
    return {7.99435344f + lop, fminf(-0.0144995697f - lop, lop != lop ? lop : 0.0f) - BWD_BAND};  // log2(255), log2(0.99)
}
constexpr float BWD_T = -0.5f * 1.44269504f;  // t of -2 power

template <int TW, int TH, bool RECT, int PPT, bool STORE = false>
__global__ void __launch_bounds__(TW * TH / PPT, PPT == 2 ? 5 : 9) k_blend_bwd(BlendArgs a) {
    constexpr int NT = TW * TH / PPT;
    constexpr int NW = NT / 32;
    constexpr int H = PPT / 2;
    __shared__ float4 s_a2[2][NT];  // sx, sy, -opacity, reach
    __shared__ float4 s_c2[2][NT];  // a, b, c, limit
    __shared__ float4 s_k2[2][NT];  // colour, power floor
    __shared__ uint2 s_r[RECT ? NT : 1];
    __shared__ uint32_t s_slot[NT];
    __shared__ uint8_t s_wm[NT];
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
        // entry `tid` of the batch that ends at list index hi
        auto entry = [&](int hi) {
            const int i = max(hi - NT + 1, 0) + tid;
            return i <= hi ? a.pair_vals[rg.x + (uint32_t)i] : NO_SLOT;
        };
        uint32_t here = entry(maxlc), next = entry(maxlc - NT);
        fetch_entry(a, S, here, &s_a2[0][tid], &s_c2[0][tid], &s_k2[0][tid]);
        int buf = 0;
        for (int hi_li = maxlc; hi_li >= 0; hi_li -= NT, buf ^= 1) {
            const int lo = max(hi_li - NT + 1, 0);
            fetch_entry(a, S, next, &s_a2[buf ^ 1][tid], &s_c2[buf ^ 1][tid], &s_k2[buf ^ 1][tid]);
            float4* s_a = s_a2[buf];
            float4* s_c = s_c2[buf];
            float4* s_k = s_k2[buf];
            fetch_wait<1>();
            // ---- each entry of list indices [lo, hi_li] gets the mask of the warps
            // whose strip of pixel rows it can reach
            uint32_t wm = 0;
            if (here != NO_SLOT) {
                const float4 A = s_a[tid], Q = s_c[tid], K = s_k[tid];
                const float thr = power_floor(A.z);
                wm = reached_warps<NW, RW>(A, Q, thr, x0c, x1c, ty * TH, c.height);
                const BwdLimits lim = bwd_limits(A.z);
                s_a[tid].z = -A.z;
                s_a[tid].w = lim.reach;
                s_c[tid].w = not_sane(Q, K) ? __int_as_float(0x7fc00000) : lim.limit;
                s_k[tid].w = thr;
                s_slot[tid] = here;
                if (RECT) s_r[tid] = make_uint2(__float_as_uint(Q.w), __float_as_uint(K.w));
            }
            s_wm[tid] = (uint8_t)wm;
            here = next;
            next = entry(hi_li - 2 * NT);
            __syncthreads();
            // ---- this warp's entries, back to front
            int cnt = 0, my_k = 0;
            auto flush = [&]() {
                __syncwarp();
                const int g = lane & (BWD_GRP - 1), q = lane / BWD_GRP;
                const float4 ctr = s_a[my_k], cq = s_c[my_k];
                const uint32_t slot = s_slot[my_k];
                const float col0 = (float)(tx * TW + (q * 8) % TW) + 0.5f;
                float c0 = 0.0f, c1 = 0.0f, c2 = 0.0f, u0 = 0.0f, u1 = 0.0f, u2 = 0.0f, w0 = 0.0f, w1 = 0.0f, w2 = 0.0f;
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int l = (q * 8 + e) ^ g;
                    const float4 f = s_b4[warp][g][l];
                    const float2 f2 = s_b2[warp][g][l];
                    c0 += f.x;
                    c1 += f.y;
                    c2 += f.z;
                    const float dx = (col0 + (float)e) - ctr.x;  // as the pixels formed it
                    const float du = dx * f.w;
                    u0 += f.w;
                    u1 += du;
                    u2 = __fmaf_rn(du, dx, u2);
                    w0 += f2.x;
                    w1 = __fmaf_rn(dx, f2.x, w1);
                    w2 += f2.y;
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
                    // a slot's second and third record: conic a, b | conic c, (sx, sy)
                    double* conic = reinterpret_cast<double*>(a.acc + (q == 3 ? 2 * S : S) + slot) + (q == 2 ? 1 : 0);
                    const float part = q == 1 ? 0.5f * u2 : q == 2 ? w1 : 0.5f * w2;
                    if (q == 0) red_add_v4(a.acc + slot, -c0, -c1, -c2, u0 / ctr.z);
                    else red_add_f64(conic, (double)part);
                    if (q == 3)
                        red_add_v2(reinterpret_cast<float2*>(a.acc + 2 * S + slot) + 1, -__fmaf_rn(cq.y, w0, cq.x * u1),
                                   -__fmaf_rn(cq.z, w0, cq.y * u1));
                }
                __syncwarp();
                cnt = 0;
            };
#pragma unroll 1
            for (int half = NT / 32 - 1; half >= 0; --half) {
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
                        const float2 t = __fmul2_rn(s2, bc2(BWD_T));
                        const float2 d = __fadd2_rn(t, bc2(A.w));
                        bool a0 = li <= lc[2 * h], a1 = li <= lc[2 * h + 1];
                        if (RECT) {
                            const uint2 r = s_r[k];
                            a0 = a0 && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h);
                            a1 = a1 && in_rect(__uint_as_float(r.x), __uint_as_float(r.y), px, py0 + 2 * h + 1);
                        }
                        sure = sure && fminf(fabsf(d.x), fabsf(d.y)) >= BWD_BAND && fmaxf(t.x, t.y) <= Q.w;
                        a0 = a0 && d.x > 0.0f;
                        a1 = a1 && d.y > 0.0f;
                        any = any || a0 || a1;
                        const float2 e = __fmul2_rn(bc2(A.z), make_float2(ex2_sfu(t.x), ex2_sfu(t.y)));
                        nal[h] = make_float2(a0 ? e.x : 0.0f, a1 ? e.y : 0.0f);
                        um[h] = nal[h];
                    }
                    float4 K = s_k[k];
                    if (!sure) {
                        const float4 q = make_float4(Q.x, Q.y, Q.z, -A.z);
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
                        // a colour that is not finite reaches no thread whose pixels all pass
                        // the splat by (the other pixels of a thread that takes it lie in the
                        // loss window of a pixel that is NaN, and so is their dL/dpixel)
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
        fetch_wait<0>();
        __syncthreads();  // every thread has read s_tile / s_maxlc before thread 0 rewrites them
    }
}

// ---- launch plumbing -----------------------------------------------------
typedef void (*BlendKernel)(BlendArgs);

template <int TW, int TH, bool RECT>
static BlendKernel pick(bool fwd, int ppt) {
    if (fwd) return ppt == 2 ? (BlendKernel)k_blend_fwd<TW, TH, RECT, 2> : (BlendKernel)k_blend_fwd<TW, TH, RECT, 4>;
    return ppt == 2 ? (BlendKernel)k_blend_bwd<TW, TH, RECT, 2> : (BlendKernel)k_blend_bwd<TW, TH, RECT, 4>;
}

static BlendKernel select_kernel(int tw, int th, bool rect, bool fwd, int ppt) {
    if (tw == 8 && th == 32) return pick<8, 32, true>(fwd, ppt);
    if (tw == 32 && th == 8) return pick<32, 8, true>(fwd, ppt);
    return rect ? pick<16, 16, true>(fwd, ppt) : pick<16, 16, false>(fwd, ppt);
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

// Pixels per thread. Four share a splat's loads and per-column terms among the
// most pixels, but a tile is then walked by two warps only, and the launch ends
// with its longest tile's serial walk; with few tiles per resident CTA two
// pixels per thread (four warps a tile) finish sooner. Measured (one view, us,
// two / four pixels): forward 47 / 64 at 256 tiles, 91 / 130 at 1024, 114 / 132
// at 2500, 139 / 144 at 3600, 180 / 175 at 4761; backward 52 / 64 at 256, 107 /
// 128 at 1600, 126 / 127 at 2025, 143 / 123 at 2500. So two up to four forward
// waves (3552 tiles on 148 SMs) and two and a half backward waves (1850).
static int pixels_for(const BlendArgs& a, int tw, int th, bool rect, bool fwd) {
    if (a.pixels_per_thread == 1) return 2;
    const long long wave = grid_for(select_kernel(tw, th, rect, fwd, 2), tw * th / 2);
    return 2ll * a.total_tiles_host <= (fwd ? 8 : 5) * wave ? 2 : 4;
}

static void launch(const BlendArgs& a, int tw, int th, bool fwd, cudaStream_t st) {
    const bool rect = a.rect_filter != 0 || !(tw == REF_TILE && th == REF_TILE);
    const int ppt = pixels_for(a, tw, th, rect, fwd);
    BlendKernel k = select_kernel(tw, th, rect, fwd, ppt);
    const int threads = tw * th / ppt;
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

// The backward's alpha and its 1/255 decision against 64 bits, as float bits: out[0]
// the largest relative error of alpha over n x n powers (evenly on [power_lo, 0])
// and opacities (by ratio on [op_lo, op_hi]), out[1] the largest error of t + reach
// over powers within 3e-5 of the decision.
__global__ void k_bwd_alpha_error(float power_lo, float op_lo, float op_hi, uint32_t n, unsigned int* out) {
    float m = 0.0f, d = 0.0f;
    const float step = 1.0f / (float)(n > 1 ? n - 1 : 1);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n * n; i += gridDim.x * blockDim.x) {
        const float op = op_lo * powf(op_hi / op_lo, (float)(i / n) * step);
        const float power = power_lo * ((float)(i % n) * step);
        const float al = op * ex2_sfu(-2.0f * power * BWD_T);
        m = fmaxf(m, (float)fabs((double)al / ((double)op * exp((double)power)) - 1.0));
        const float cut = -logf(255.0f * op) + ((float)(i % 61u) - 30.0f) * 1e-6f;
        if (!(cut <= 0.0f)) continue;
        const float reach = -2.0f * cut * BWD_T + bwd_limits(op).reach;
        d = fmaxf(d, (float)fabs((double)reach - log2(255.0 * (double)op * exp((double)cut))));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        d = fmaxf(d, __shfl_xor_sync(0xffffffffu, d, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(out, __float_as_uint(m));
        atomicMax(out + 1, __float_as_uint(d));
    }
}

void launch_bwd_alpha_error(float power_lo, float op_lo, float op_hi, uint32_t n, unsigned int* out, cudaStream_t st) {
    k_bwd_alpha_error<<<device_sm_count() * 4, 256, 0, st>>>(power_lo, op_lo, op_hi, n, out);
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

void launch_blend_forward(const BlendArgs& a, int tw, int th, cudaStream_t st) { launch(a, tw, th, true, st); }
void launch_blend_backward(const BlendArgs& a, int tw, int th, cudaStream_t st) { launch(a, tw, th, false, st); }

// Store-all variant (16x16 tiles, 256-splat batches, 2 pixels per thread): the
// forward writes T before every contributing splat of every pixel to
// a.tstore[(list position) * 256 + pixel in tile], the backward reads it back
// instead of rebuilding T from the final T.
void launch_blend_store_all(const BlendArgs& a, bool fwd, cudaStream_t st) {
    BlendKernel k = fwd ? (BlendKernel)k_blend_fwd<16, 16, false, 2, true> : (BlendKernel)k_blend_bwd<16, 16, false, 2, true>;
    int grid = grid_for(k, 128);
    if (!a.total_tiles) grid = std::min(grid, std::max(a.total_tiles_host, 1));
    k<<<grid, 128, 0, st>>>(a);
}

}  // namespace rgs
