// bin.cu -- binning the depth-sorted slots by supertile.
//
// The reference sorts visible splats by depth and then, serially, pushes each
// splat's index into every tile its 3-sigma rectangle touches
// (src/cpu/backward.rs:190-205). Here:
//   compact:    the slots with at least one tile pair are gathered in slot
//               order with their depth keys (the depth sort, sort.cu, then
//               orders only them);
//   entry scan: exclusive scan of the slots' supertile-entry counts in depth
//               order, in 64 bits (the total stays on the device, a count past
//               32 bits is reported, never wrapped);
//   emit:       every block expands its chunk of depth-sorted slots into
//               (supertile id, slot) entries with the masks of their tiles;
// then a stable radix sort on the supertile id (sort.cu) groups the entries
// by supertile while keeping depth order inside each, and supertile.cu
// expands them into the per-tile lists. The projection leaves one 32-byte bin
// record per slot (rgs_internal.cuh).
#include <algorithm>

#include "rgs_internal.cuh"
#include "tiles.cuh"

namespace rgs {

constexpr int BIN_THREADS = 256;
constexpr int BIN_SUB = BIN_THREADS;  // slots per emit sub-tile
constexpr uint32_t EMIT_STAGE = 2048;  // entries of a sub-tile staged before they are written

// Blocks of the entry scan and the emission for up to S slots: chunks of at
// least one sub-tile, and short ones, since near splats (the front of the
// order) have many times the entries of far ones: 4, 8, 16, 32 and 64 blocks
// per SM took 0.40, 0.24, 0.20, 0.19 and 0.21 ms on 1M Gaussians x 8 views.
int bin_grid_blocks(size_t S) {
    const size_t most = (size_t)bin_grid_max();
    return (int)std::max<size_t>(1, std::min(most, (S + BIN_SUB - 1) / BIN_SUB));
}
int bin_grid_max() { return device_sm_count() * 32; }

__device__ __forceinline__ void bin_chunk(uint32_t n, int G, int b, uint32_t& begin, uint32_t& end) {
    uint32_t chunk = (uint32_t)(((uint64_t)n + G - 1) / G);
    chunk = (chunk + 31u) & ~31u;
    uint64_t bg = (uint64_t)chunk * b;
    begin = (uint32_t)(bg < (uint64_t)n ? bg : (uint64_t)n);
    end = (uint32_t)(bg + chunk < (uint64_t)n ? bg + chunk : (uint64_t)n);
}

// Block b's sum of the entry counts of its chunk of the order.
__global__ void __launch_bounds__(BIN_THREADS) k_entry_sums(EmitArgs a) {
    __shared__ unsigned long long s_w[BIN_THREADS / 32];
    uint32_t begin, end;
    bin_chunk(*a.n_order, gridDim.x, blockIdx.x, begin, end);
    unsigned long long s = 0;
    for (uint32_t r = begin + threadIdx.x; r < end; r += BIN_THREADS) s += a.st_cnt[a.order[r]];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < BIN_THREADS / 32; ++w) t += s_w[w];
        a.block_sums[blockIdx.x] = t;
    }
}

// Exclusive scan of the G block sums (single block) in 64 bits; writes the
// total to *total64 and, saturated at 2^32 - 1, to *total.
constexpr int SUMS_PER = 8;
__global__ void __launch_bounds__(1024) k_scan_block_sums(unsigned long long* __restrict__ block_sums, int G,
                                                          uint32_t* __restrict__ total,
                                                          unsigned long long* __restrict__ total64) {
    __shared__ unsigned long long s_w[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long carry = 0;  // the same in every thread
    for (int base = 0; base < G; base += 1024 * SUMS_PER) {
        const int i0 = base + (int)threadIdx.x * SUMS_PER;
        unsigned long long v[SUMS_PER], sum = 0;
#pragma unroll
        for (int k = 0; k < SUMS_PER; ++k) {
            v[k] = i0 + k < G ? block_sums[i0 + k] : 0ull;
            sum += v[k];
        }
        unsigned long long x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_w[w] = x;
        __syncthreads();
        if (w == 0) {
            unsigned long long t = s_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            s_w[lane] = t;
        }
        __syncthreads();
        unsigned long long run = carry + (w ? s_w[w - 1] : 0ull) + x - sum;
#pragma unroll
        for (int k = 0; k < SUMS_PER; ++k) {
            if (i0 + k < G) block_sums[i0 + k] = run;
            run += v[k];
        }
        carry += s_w[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *total = carry > 0xffffffffull ? 0xffffffffu : (uint32_t)carry;
        *total64 = carry;
    }
}

void launch_entry_scan(const EmitArgs& a, int grid, cudaStream_t st) {
    k_entry_sums<<<grid, BIN_THREADS, 0, st>>>(a);
    k_scan_block_sums<<<1, 1024, 0, st>>>(a.block_sums, grid, a.total, a.total64);
}

// Row blockIdx.y: one view's pairs, summed by the row's blocks into out[view]
// (zeroed before).
__global__ void __launch_bounds__(BIN_THREADS) k_view_pairs(const uint32_t* __restrict__ cnt, uint32_t n,
                                                            unsigned long long* __restrict__ out) {
    __shared__ unsigned long long s_w[BIN_THREADS / 32];
    const uint32_t* c = cnt + (size_t)blockIdx.y * n;
    unsigned long long t = 0;
    for (uint32_t i = blockIdx.x * BIN_THREADS + threadIdx.x; i < n; i += gridDim.x * BIN_THREADS) t += c[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long v = 0;
        for (int w = 0; w < BIN_THREADS / 32; ++w) v += s_w[w];
        if (v) atomicAdd(out + blockIdx.y, v);
    }
}

void launch_view_pairs(const uint32_t* cnt, uint32_t n, int V, unsigned long long* out, cudaStream_t st) {
    if (V <= 0) return;
    cudaMemsetAsync(out, 0, (size_t)V * 8, st);
    k_view_pairs<<<dim3((unsigned)device_sm_count(), (unsigned)V), BIN_THREADS, 0, st>>>(cnt, n, out);
}

// ---- emission ---------------------------------------------------------------
// A block expands its chunk of the depth order, BIN_SUB slots (one per thread) at
// a time, into (supertile id, slot) entries, each with the mask of the
// supertile's tiles the slot keeps. Two kinds of slot:
//   small (at most 15 columns and SPAN_ROWS rows): its thread walks its supertile
//     rows; a row's four packed spans come out of the bin record by one funnel
//     shift, become column bits, and every four columns of those are one
//     supertile's mask. The block's entries are staged so that consecutive lanes
//     write consecutive entries;
//   large: one warp per slot, one lane per tile row: the rows' kept spans are
//     recomputed once per supertile row from the record, by the test the
//     projection counted with on the same floats, and the lanes then take the
//     entries of the 8 supertile rows at hand.
// Masks formed here, where a slot's record is read once, and not after the sort,
// where every entry gathers it again; supertiles of the rectangle that the kept
// spans miss are left out. Entry scan + emission + supertile sort + masks + tile
// lists: 1.32 -> 0.84 ms (1M Gaussians x 8 views), 29.8 -> 13 ms (3M anisotropic
// x 8 views of 1920x1080). A thread per four consecutive entries, found by
// binary search, took 0.33 ms for this kernel where this takes 0.19.
template <bool PRUNE>
__global__ void __launch_bounds__(BIN_THREADS, 5) k_emit(EmitArgs a) {
    __shared__ uint32_t s_off[BIN_SUB];  // large slots: first entry within the sub-tile
    __shared__ uint32_t s_slot[BIN_SUB];
    __shared__ uint2 s_ent[EMIT_STAGE];  // staged entries: key, slot
    // large slots: (sx, sy, conic a, b), (conic c, power floor, first tile, size)
    __shared__ float4 s_la[BIN_SUB], s_lb[BIN_SUB];
    __shared__ uint32_t s_w[BIN_THREADS / 32];
    __shared__ int s_large;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const float inv_n = 1.0f / (float)a.n_per_view;
    uint32_t begin, end;
    bin_chunk(*a.n_order, gridDim.x, blockIdx.x, begin, end);
    if (blockIdx.x == 0 && tid == 0) *a.eff = min(*a.total, a.cap);
    unsigned long long base = a.block_sums[blockIdx.x];
    for (uint32_t r0 = begin; r0 < end; r0 += BIN_SUB) {
        const bool in = r0 + (uint32_t)tid < end;
        uint32_t slot = 0;
        uint4 d = make_uint4(0u, 0u, 0u, 0u), sp = make_uint4(0u, 0u, 0u, 0u);
        if (tid == 0) s_large = 0;
        if (in) {
            slot = a.order[r0 + (uint32_t)tid];
            d = a.spans[2 * (size_t)slot + 1];
            if (PRUNE) sp = a.spans[2 * (size_t)slot];
        }
        const int rw = (int)(d.y & 0xffffu), rh = (int)(d.y >> 16);
        const bool large = in && (rw > 15 || rh > SPAN_ROWS);
        if (!PRUNE && in && !large) {
            // every row keeps the whole rectangle
            const uint32_t b = (uint32_t)rw << 4 | (uint32_t)rw << 12 | (uint32_t)rw << 20 | (uint32_t)rw << 28;
            sp = make_uint4(rh >= 4 ? b : b & ((1u << (8 * rh)) - 1u), rh >= 8 ? b : rh > 4 ? b & ((1u << (8 * (rh - 4))) - 1u) : 0u,
                            rh >= 12 ? b : rh > 8 ? b & ((1u << (8 * (rh - 8))) - 1u) : 0u,
                            rh >= 16 ? b : rh > 12 ? b & ((1u << (8 * (rh - 12))) - 1u) : 0u);
        }
        uint32_t x = d.z;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_w[w] = x;
        __syncthreads();
        uint32_t pre = 0, sub_total = 0;
#pragma unroll
        for (int k = 0; k < BIN_THREADS / 32; ++k) {
            const uint32_t t = s_w[k];
            if (k < w) pre += t;
            sub_total += t;
        }
        uint32_t at = pre + x - d.z;
        s_off[tid] = at;
        s_slot[tid] = large ? slot : 0xffffffffu;
        if (large) {
            float4 A = make_float4(0.0f, 0.0f, 0.0f, 0.0f), Q = A;
            if (PRUNE) {
                A = a.rec[slot];
                Q = a.rec[(size_t)a.S + slot];
            }
            s_la[tid] = make_float4(A.x, A.y, Q.x, Q.y);
            s_lb[tid] = make_float4(Q.z, PRUNE ? power_floor(A.z) : 0.0f, __uint_as_float(d.x), __uint_as_float(d.y));
            s_large = 1;
        }
        if (in && !large) {
            // the slot's view (slots below 2^32: the quotient's estimate is off by
            // at most one)
            uint32_t v = (uint32_t)((float)slot * inv_n);
            if (v * a.n_per_view > slot) --v;
            if (slot - v * a.n_per_view >= a.n_per_view) ++v;
            const DevCam& cm = a.cams[v];
            const uint32_t cx0 = d.x & 0xffffu, ty0 = d.x >> 16;
            uint32_t id = (uint32_t)cm.st_base + ty0 / ST_EDGE * (uint32_t)cm.st_x + cx0 / ST_EDGE;
            const int cx = (int)(cx0 % ST_EDGE), sh = 8 * (int)(ty0 % ST_EDGE);
            const uint32_t words[6] = {0u, sp.x, sp.y, sp.z, sp.w, 0u};
#pragma unroll
            for (int k = 0; k < 5; ++k, id += (uint32_t)cm.st_x) {
                // bytes of the supertile row's tile rows (zero outside the rectangle)
                const uint32_t wk = __funnelshift_l(words[k], words[k + 1], sh);
                uint32_t rb[ST_EDGE];
#pragma unroll
                for (int kk = 0; kk < ST_EDGE; ++kk) {
                    const uint32_t b = (wk >> (8 * kk)) & 0xffu;
                    rb[kk] = ((1u << (b >> 4)) - 1u) << (cx + (int)(b & 0xfu));
                }
                const uint32_t all = rb[0] | rb[1] | rb[2] | rb[3];
                if (!all) continue;
                const int last = (31 - __clz(all)) / ST_EDGE;
                for (int q = (__ffs(all) - 1) / ST_EDGE; q <= last; ++q, ++at) {
                    uint32_t m = 0;
#pragma unroll
                    for (int kk = 0; kk < ST_EDGE; ++kk) m |= ((rb[kk] >> (ST_EDGE * q)) & 0xfu) << (ST_EDGE * kk);
                    const uint32_t key = (id + (uint32_t)q) | (a.packed ? m << 16 : 0u);
                    if (sub_total <= EMIT_STAGE) {
                        s_ent[at] = make_uint2(key, slot);
                    } else if (base + at < a.cap) {
                        a.keys[base + at] = key;
                        a.vals[base + at] = slot;
                    } else {
                        *a.overflow = 1;
                    }
                }
            }
        }
        __syncthreads();
        const bool staged = sub_total <= EMIT_STAGE;
        if (s_large) {
            for (int r = w; r < BIN_SUB; r += BIN_THREADS / 32) {
                const uint32_t ls = s_slot[r];
                if (ls == 0xffffffffu) continue;
                const uint32_t v = ls / a.n_per_view;
                const DevCam& cm = a.cams[v];
                const float4 la = s_la[r], lb = s_lb[r];
                const uint32_t xy = __float_as_uint(lb.z), wh = __float_as_uint(lb.w);
                const int cx0 = (int)(xy & 0xffffu), ty0 = (int)(xy >> 16), lw = (int)(wh & 0xffffu), lh = (int)(wh >> 16);
                SpanSetup u;
                if (PRUNE) u = span_setup(la.x, la.y, la.z, la.w, lb.x, lb.y);
                uint32_t out = s_off[r];
                const int sy0 = ty0 / ST_EDGE, rows = (ty0 + lh - 1) / ST_EDGE - sy0 + 1;
                for (int g0 = 0; g0 < rows; g0 += 32 / ST_EDGE) {
                    const int ty = (sy0 + g0) * ST_EDGE + lane;
                    int c0 = 0, c1 = 0;
                    if (ty >= ty0 && ty < ty0 + lh) {
                        if (PRUNE) kept_cols(u, ty, a.tile_w, a.tile_h, cm.height, cx0, cx0 + lw, c0, c1);
                        else {
                            c0 = cx0;
                            c1 = cx0 + lw;
                        }
                    }
                    int first = c1 > c0 ? c0 : 0x7fffffff, last = c1 > c0 ? c1 - 1 : -1;
#pragma unroll
                    for (int o = 1; o < ST_EDGE; o <<= 1) {
                        first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
                        last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
                    }
                    const int f = last >= 0 ? first / ST_EDGE : 0;
                    const int cnt = last >= 0 ? last / ST_EDGE - f + 1 : 0;
                    int incl = lane % ST_EDGE == 0 ? cnt : 0;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int up = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += up;
                    }
                    const int total = __shfl_sync(0xffffffffu, incl, 31);
                    const int start = incl - cnt;  // the supertile row's first entry (all of its four lanes)
                    const uint32_t cols = (uint32_t)c0 | ((uint32_t)c1 << 16);
                    for (int e0 = 0; e0 < total; e0 += 32) {
                        const int e = e0 + lane;
                        int qd = 0;
#pragma unroll
                        for (int q = 1; q < 32 / ST_EDGE; ++q)
                            if (__shfl_sync(0xffffffffu, start, q * ST_EDGE) <= e) qd = q;
                        const int qs = __shfl_sync(0xffffffffu, start, qd * ST_EDGE), qf = __shfl_sync(0xffffffffu, f, qd * ST_EDGE);
                        const int sc = qf + e - qs;  // supertile column
                        uint32_t m = 0;
#pragma unroll
                        for (int kk = 0; kk < ST_EDGE; ++kk) {
                            const uint32_t cc = __shfl_sync(0xffffffffu, cols, qd * ST_EDGE + kk);
                            m |= row_bits((int)(cc & 0xffffu), (int)(cc >> 16), sc * ST_EDGE, kk);
                        }
                        if (e < total) {
                            const uint32_t key = (uint32_t)(cm.st_base + (sy0 + g0 + qd) * cm.st_x + sc) | (a.packed ? m << 16 : 0u);
                            const unsigned long long pos = base + out + (unsigned)e;
                            if (staged) {
                                s_ent[out + (unsigned)e] = make_uint2(key, ls);
                            } else if (pos < a.cap) {
                                a.keys[pos] = key;
                                a.vals[pos] = ls;
                            } else {
                                *a.overflow = 1;
                            }
                        }
                    }
                    out += (unsigned)total;
                }
            }
            __syncthreads();
        }
        if (staged) {
            for (uint32_t i = tid; i < sub_total; i += BIN_THREADS) {
                const uint2 e = s_ent[i];
                if (base + i < a.cap) {
                    a.keys[base + i] = e.x;
                    a.vals[base + i] = e.y;
                } else {
                    *a.overflow = 1;
                }
            }
        }
        base += sub_total;
        __syncthreads();
    }
}

void launch_emit_supertiles(const EmitArgs& a, int grid, cudaStream_t st) {
    if (a.prune) k_emit<true><<<grid, BIN_THREADS, 0, st>>>(a);
    else k_emit<false><<<grid, BIN_THREADS, 0, st>>>(a);
}

// ---- slots with tile pairs, compacted in slot order ------------------------
// Before the depth sort, the slots that emit at least one pair are gathered,
// in slot order, with their depth keys: the sort then orders only them, and
// because it is stable and the gather keeps slot order, equal depths still
// leave Gaussians of a view in index order. Chunks of CMP_CHUNK consecutive
// slots: count per chunk, one exclusive scan, then a stable in-chunk scatter.
constexpr int CMP_PER = 4;
constexpr int CMP_CHUNK = BIN_THREADS * CMP_PER;

__global__ void __launch_bounds__(BIN_THREADS) k_visible_counts(const uint32_t* __restrict__ cnt, uint32_t S,
                                                                unsigned long long* __restrict__ chunk_counts,
                                                                unsigned long long* __restrict__ pairs64) {
    __shared__ uint32_t s_w[BIN_THREADS / 32];
    __shared__ unsigned long long s_p[BIN_THREADS / 32];
    const uint32_t base = blockIdx.x * (uint32_t)CMP_CHUNK + threadIdx.x * CMP_PER;
    uint32_t c = 0;
    unsigned long long p = 0;
#pragma unroll
    for (int k = 0; k < CMP_PER; ++k) {
        const uint32_t v = base + k < S ? cnt[base + k] : 0u;
        c += v != 0u ? 1u : 0u;
        p += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_xor_sync(0xffffffffu, c, o);
        p += __shfl_xor_sync(0xffffffffu, p, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_w[threadIdx.x >> 5] = c;
        s_p[threadIdx.x >> 5] = p;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        unsigned long long q = 0;
        for (int w = 0; w < BIN_THREADS / 32; ++w) {
            t += s_w[w];
            q += s_p[w];
        }
        chunk_counts[blockIdx.x] = t;
        if (q) atomicAdd(pairs64, q);
    }
}

__global__ void __launch_bounds__(BIN_THREADS) k_compact_visible(const uint32_t* __restrict__ cnt, const uint32_t* __restrict__ key,
                                                                 uint32_t S, const unsigned long long* __restrict__ chunk_offs,
                                                                 uint32_t* __restrict__ ckey, uint32_t* __restrict__ cslot) {
    __shared__ uint32_t s_w[BIN_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t base = blockIdx.x * (uint32_t)CMP_CHUNK + threadIdx.x * CMP_PER;
    // every slot's count and depth key in one round trip (a culled slot's key
    // is whatever an earlier step left: read and dropped)
    bool f[CMP_PER];
    uint32_t kv[CMP_PER];
    uint32_t local = 0;
#pragma unroll
    for (int k = 0; k < CMP_PER; ++k) {
        const bool in = base + k < S;
        f[k] = in && cnt[base + k] != 0u;
        kv[k] = in ? key[base + k] : 0u;
        local += f[k] ? 1u : 0u;
    }
    uint32_t x = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[w] = x;
    __syncthreads();
    uint32_t wpre = 0;
    for (int k = 0; k < w; ++k) wpre += s_w[k];
    uint32_t pos = (uint32_t)chunk_offs[blockIdx.x] + wpre + x - local;
#pragma unroll
    for (int k = 0; k < CMP_PER; ++k) {
        if (f[k]) {
            const uint32_t slot = base + k;
            ckey[pos] = kv[k];
            cslot[pos] = slot;
            ++pos;
        }
    }
}

size_t compact_chunks(size_t S) { return (S + CMP_CHUNK - 1) / CMP_CHUNK; }

void launch_compact_visible(const uint32_t* cnt, const uint32_t* key, uint32_t S, unsigned long long* chunk_counts,
                            uint32_t* ckey, uint32_t* cslot, uint32_t* n_out, unsigned long long* n_out64,
                            unsigned long long* pairs64, cudaStream_t st) {
    const unsigned chunks = (unsigned)compact_chunks(S);
    if (chunks == 0) {
        cudaMemsetAsync(n_out, 0, 4, st);
        cudaMemsetAsync(n_out64, 0, 8, st);
        return;
    }
    k_visible_counts<<<chunks, BIN_THREADS, 0, st>>>(cnt, S, chunk_counts, pairs64);
    k_scan_block_sums<<<1, 1024, 0, st>>>(chunk_counts, (int)chunks, n_out, n_out64);
    k_compact_visible<<<chunks, BIN_THREADS, 0, st>>>(cnt, key, S, chunk_counts, ckey, cslot);
}

}  // namespace rgs
