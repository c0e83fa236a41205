// nd_bvh.cu -- LBVH neighbour search for sm_103a.
//
// Reference: src/Neighbors/BVHTraverse.jl (NaiveDynamics.jl).  The pipeline is
//   Morton codes (mortoncodes!, :237-288)  -> stable radix sort (sortperm, :570)
//   -> gather + leaf boxes (leafcluster_primitives :376-410 / cluster_primitives :341-375)
//   -> Apetrei bottom-up build with CAS (bvh_interior!, :704-846)
//   -> stackless rope traversal (leafneighbor_traverse :1236-1323,
//      neighbor_traverse :1125-1183) with pair emission.
// Everything that decides which pairs exist is computed with the reference's
// exact single-precision operation order (no FMA contraction, IEEE division and
// square root) so that codes, order, tree and pair list are bit-identical.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "nd_internal.cuh"

namespace nd {

// =================================================================== Morton

// mortoncodes! with K = Int32 (BVHTraverse.jl:259-284), one position.
__device__ __forceinline__ int32_t code_reference(const float* __restrict__ xyz, int32_t i,
                                                  float binwidth, int32_t* err) {
    const int32_t magic[3] = {153391689, 306783378, 613566756};
    int32_t code = 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float p = xyz[3 * (int64_t)i + d];
        if (!isfinite(p)) { set_error(err, ND_ERR_NONFINITE, i); return 0; }
        float q = floorf(__fdiv_rn(p, binwidth));
        // trunc(Int32, ::Float32) accepts -2^31 <= q < 2^31 (Julia Base float.jl)
        if (!(q >= -2147483648.0f && q < 2147483648.0f)) { set_error(err, ND_ERR_RANGE, i); return 0; }
        int32_t qi = (int32_t)q;
        int32_t yin = qi & magic[d];
        int32_t yang = qi | ~magic[d];
        code |= (yin & yang);
    }
    return code;
}

// Spatial code: 3-D Hilbert index over the bounding box, 1024 bins per axis.
// bbox: order-preserving images (f2o) of min[3], max[3].
__device__ __forceinline__ int32_t code_spatial(const float* __restrict__ xyz, int32_t i,
                                                const uint32_t* bbox) {
    uint32_t q[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float lo = o2f(bbox[d]), hi = o2f(bbox[3 + d]);
        float ext = __fsub_rn(hi, lo);
        float s = ext > 0.0f ? __fdiv_rn(1024.0f, ext) : 0.0f;
        float t = floorf(__fmul_rn(__fsub_rn(xyz[3 * (int64_t)i + d], lo), s));
        int32_t qi = (t < 0.0f) ? 0 : (t > 1023.0f ? 1023 : (int32_t)t);
        q[d] = (uint32_t)qi;
    }
    return (int32_t)hilbert3_10(q[0], q[1], q[2]);
}

// Min and max images of the finite coordinates of position i.
__device__ __forceinline__ void bbox_add(const float* __restrict__ xyz, int64_t i,
                                         uint32_t (&mn)[3], uint32_t (&mx)[3], int32_t* err) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float p = xyz[3 * i + d];
        if (!isfinite(p)) { set_error(err, ND_ERR_NONFINITE, (int32_t)i); continue; }
        uint32_t o = f2o(p);
        mn[d] = min(mn[d], o);
        mx[d] = max(mx[d], o);
    }
}

// The warps' boxes in s_b[warp][6] (after this, a __syncthreads by the caller).
__device__ __forceinline__ void bbox_warp(uint32_t (&mn)[3], uint32_t (&mx)[3],
                                          uint32_t (*s_b)[6]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        mn[d] = __reduce_min_sync(0xffffffffu, mn[d]);
        mx[d] = __reduce_max_sync(0xffffffffu, mx[d]);
    }
    if (lane == 0)
#pragma unroll
        for (int d = 0; d < 3; ++d) { s_b[warp][d] = mn[d]; s_b[warp][3 + d] = mx[d]; }
}
// Component k (0-2 min, 3-5 max) over the block's warps.
__device__ __forceinline__ uint32_t bbox_block(const uint32_t (*s_b)[6], int k) {
    uint32_t v = s_b[0][k];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = k < 3 ? min(v, s_b[w][k]) : max(v, s_b[w][k]);
    return v;
}

// Bounding box of the positions (order-preserving uint atomics), used by the
// spatial code.  bbox[0..2] = min keys, bbox[3..5] = max keys.
__global__ void k_bbox(const float* __restrict__ xyz, int32_t n, uint32_t* bbox, int32_t* err) {
    uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu};
    uint32_t mx[3] = {0u, 0u, 0u};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        bbox_add(xyz, i, mn, mx, err);
    // block reduction first: one atomic per block and component
    __shared__ uint32_t s_b[32][6];
    bbox_warp(mn, mx, s_b);
    __syncthreads();
    if (threadIdx.x < 6) {
        const int k = threadIdx.x;
        const uint32_t v = bbox_block(s_b, k);
        if (k < 3) atomicMin(&bbox[k], v);
        else atomicMax(&bbox[k], v);
    }
}

__global__ void k_bbox_init(uint32_t* bbox) {
    if (threadIdx.x < 6) bbox[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
}

// A given frame in place of the bounding box.
struct CodeFrame {
    float v[6];
    int32_t given;
};
__global__ void k_bbox_set(uint32_t* bbox, CodeFrame fr) {
    if (threadIdx.x < 6) bbox[threadIdx.x] = f2o(fr.v[threadIdx.x]);
}

constexpr int RS_BINS = 256;
constexpr int RS_TILE = 2048;  // keys per block of the counting and scattering kernels

// Keys per block of the one-kernel pass: few keys go to small blocks (the time
// of a pass is then a block's: 20,000 keys 7.6 us a pass with 2,048 keys a
// block, 11.2 us with 4,096), many to large ones (the time is then in adding up
// the tiles' counts: 262,144 keys 18.0 and 13.7 us).
__host__ __device__ inline int32_t pass_tile(int32_t n) {
    return n <= 32768 ? 1024 : n <= 131072 ? 2048 : 4096;
}

// Codes of all positions, the identity permutation, and (hist given) the
// digit counts of the sort's first pass, per tile of pass_tile(n) positions.
__global__ void k_morton(const float* __restrict__ xyz, int32_t n, int32_t order, float binwidth,
                         const uint32_t* __restrict__ bbox, int32_t* __restrict__ codes,
                         int32_t* __restrict__ iota, uint32_t* __restrict__ hist, int32_t* err) {
    int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t code = order == ND_ORDER_SPATIAL ? code_spatial(xyz, i, bbox)
                                                   : code_reference(xyz, i, binwidth, err);
    codes[i] = code;
    if (iota) iota[i] = i;
    if (hist) atomicAdd(&hist[(i / pass_tile(n)) * RS_BINS + (code & 0xff)], 1u);
}

constexpr float kBinWidth = (float)(1.0 / 1023.0);  // Float32(1/1023), BVHTraverse.jl:184

static nd_status codes_kernels(Ctx* c, const float* xyz, int32_t n, int32_t order, int32_t* codes,
                               int32_t* iota, const float* frame, uint32_t* hist) {
    const int T = 256;
    if (order == ND_ORDER_SPATIAL) {
        nd_status st = ensure(c, c->misc, 64);
        if (st) return st;
        if (frame) {
            CodeFrame fr{};
            for (int k = 0; k < 6; ++k) fr.v[k] = frame[k];
            k_bbox_set<<<1, 32, 0, c->stream>>>((uint32_t*)c->misc.p, fr);
            c->launches++;
        } else {
            k_bbox_init<<<1, 32, 0, c->stream>>>((uint32_t*)c->misc.p);
            c->launches++;
            int blocks = (int)std::min<int64_t>(cdiv(n, T), 152 * 8);
            k_bbox<<<blocks, T, 0, c->stream>>>(xyz, n, (uint32_t*)c->misc.p, c->d_err);
            c->launches++;
        }
    }
    k_morton<<<(int)cdiv(n, T), T, 0, c->stream>>>(xyz, n, order, kBinWidth,
                                                   (const uint32_t*)c->misc.p, codes, iota, hist,
                                                   c->d_err);
    c->launches++;
    return check_launch(c, "morton");
}

nd_status morton_codes(Ctx* c, const float* xyz, int32_t n, int32_t order, int32_t* codes,
                       int32_t* iota, const float* frame) {
    if (n <= 0) return ND_OK;
    return codes_kernels(c, xyz, n, order, codes, iota, frame, nullptr);
}

// ================================================================ radix sort
// Stable LSD radix sort, 8-bit digits, no block waits for another.  Three
// forms, by size:
//  * up to kSmallSort keys: one block does everything (codes included), one
//    launch; 512 positions took 15 launches, 50 us, before;
//  * up to kDirectKeys: one kernel per pass (k_rs_pass), at most 128 blocks.  A
//    block adds up the digit counts of the tiles before its own by itself
//    (coalesced rows, 16 or 32 loads in flight; at 128 tiles 128 KB from L2 a block)
//    and counts, while it scatters, the next pass's digits at their
//    destination tiles, so a pass needs no counting and no scanning kernel;
//  * more: digit counts per tile (k_rs_upsweep), a scan per digit over the
//    tiles (k_rs_scan), the scatter (k_rs_scatter): the rows would be read
//    ntiles^2 times.

constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = RS_TILE / RS_THREADS;
constexpr int32_t kSmallSort = 4096;
constexpr int32_t kDirectKeys = 128 * 4096;
static_assert(RS_THREADS == RS_BINS, "scatter maps one thread per digit");

size_t sort_scratch_bytes(int32_t n) {
    const size_t rows = n <= kDirectKeys ? 4 * (size_t)cdiv(n, pass_tile(n)) : (size_t)cdiv(n, RS_TILE);
    return sizeof(uint32_t) * (RS_BINS * rows + RS_BINS);
}

// Lanes of the warp with this lane's digit (0 .. 255; 256 for no item): one
// ballot per bit (a match instruction takes several times as long on 32
// different values).
__device__ __forceinline__ unsigned digit_peers(uint32_t dg) {
    unsigned peers = __ballot_sync(0xffffffffu, dg < 256u);
    if (dg >= 256u) peers = ~peers;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = (dg >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, one);
        peers &= one ? m : ~m;
    }
    return peers;
}

// Ranks of a warp's ITEMS x 32 digits (held i-major: item i of lane l is the
// (32 i + l)-th) among the equal digits before them in the warp; cnt[digit]
// counts the warp's digits (zeroed by the caller).  Digit 256 is no item.
template <int ITEMS, class C>
__device__ __forceinline__ void warp_ranks(const uint32_t (&dg)[ITEMS], C* cnt,
                                           uint32_t (&rank)[ITEMS]) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const unsigned peers = digit_peers(dg[i]);
        const int lead = __ffs(peers) - 1;
        uint32_t old = 0;
        if (lane == lead && dg[i] < 256u) {
            old = cnt[dg[i]];
            cnt[dg[i]] = (C)(old + __popc(peers));
        }
        old = __shfl_sync(0xffffffffu, old, lead);
        rank[i] = old + __popc(peers & lt);
        __syncwarp();
    }
}

// Exclusive scan of one value per digit over the first 256 threads of the
// block; every thread calls it.
__device__ __forceinline__ uint32_t digits_scan(uint32_t v, uint32_t* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
        if (lane >= s) x += y;
    }
    if (warp < 8 && lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) before += w < warp ? s_warp[w] : 0u;
    return before + x - v;
}

// One block: codes (xyz given) or given keys and values, sorted into
// keys/vals.  Each warp holds ITEMS x 32 consecutive items.
template <int ITEMS>
__global__ void __launch_bounds__(1024)
    k_small_order(const float* __restrict__ xyz, int32_t n, int32_t order, float binwidth,
                  CodeFrame frame, uint32_t* keys, int32_t* vals, int passes, int32_t* err) {
    __shared__ __align__(4) uint16_t s_cnt[32][RS_BINS];
    __shared__ uint32_t s_x[1024 * ITEMS];
    __shared__ uint32_t s_part[4][RS_BINS];
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_b[32][6];
    __shared__ uint32_t s_box[6];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    uint32_t key[ITEMS];
    int32_t val[ITEMS];
    const int32_t at0 = w * 32 * ITEMS + lane;
    if (xyz) {
        if (order == ND_ORDER_SPATIAL) {
            uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu};
            uint32_t mx[3] = {0u, 0u, 0u};
            if (!frame.given)
                for (int32_t i = t; i < n; i += 1024) bbox_add(xyz, i, mn, mx, err);
            bbox_warp(mn, mx, s_b);
            __syncthreads();
            if (t < 6) s_box[t] = frame.given ? f2o(frame.v[t]) : bbox_block(s_b, t);
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int32_t k = at0 + 32 * i;
            val[i] = k;
            key[i] = k >= n ? 0u
                     : order == ND_ORDER_SPATIAL
                         ? (uint32_t)code_spatial(xyz, k, s_box)
                         : (uint32_t)code_reference(xyz, k, binwidth, err);
        }
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const int32_t k = at0 + 32 * i;
            key[i] = k < n ? keys[k] : 0u;
            val[i] = k < n ? vals[k] : 0;
        }
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        for (int k = t; k < 32 * RS_BINS / 2; k += 1024) reinterpret_cast<uint32_t*>(s_cnt)[k] = 0u;
        __syncthreads();
        uint32_t dg[ITEMS], rank[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) dg[i] = at0 + 32 * i < n ? (key[i] >> shift) & 0xffu : 256u;
        warp_ranks<ITEMS>(dg, s_cnt[w], rank);
        __syncthreads();
        // digit-major prefix: four groups of eight warps' counts per digit
        const int d = t & 255, g = t >> 8;
        uint32_t sum = 0, c8[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) { c8[k] = s_cnt[8 * g + k][d]; sum += c8[k]; }
        s_part[g][d] = sum;
        __syncthreads();
        const uint32_t tot = s_part[0][d] + s_part[1][d] + s_part[2][d] + s_part[3][d];
        const uint32_t ex = digits_scan(tot, s_warp);
        if (g == 0) s_x[d] = ex;
        __syncthreads();
        uint32_t run = s_x[d];
        for (int k = 0; k < g; ++k) run += s_part[k][d];
#pragma unroll
        for (int k = 0; k < 8; ++k) { s_cnt[8 * g + k][d] = (uint16_t)run; run += c8[k]; }
        __syncthreads();
        uint32_t pos[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) pos[i] = dg[i] < 256u ? s_cnt[w][dg[i]] + rank[i] : 0u;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (dg[i] < 256u) s_x[pos[i]] = key[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) key[i] = s_x[at0 + 32 * i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if (dg[i] < 256u) s_x[pos[i]] = (uint32_t)val[i];
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) val[i] = (int32_t)s_x[at0 + 32 * i];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int32_t k = at0 + 32 * i;
        if (k < n) { keys[k] = key[i]; vals[k] = val[i]; }
    }
}

static void small_order(Ctx* c, const float* xyz, int32_t n, int32_t order, const float* frame,
                        uint32_t* keys, int32_t* vals, int passes) {
    CodeFrame fr{};
    if (frame) {
        for (int k = 0; k < 6; ++k) fr.v[k] = frame[k];
        fr.given = 1;
    }
#define ND_SMALL(I)                                                                             \
    k_small_order<I><<<1, 1024, 0, c->stream>>>(xyz, n, order, kBinWidth, fr, keys, vals, passes, \
                                                c->d_err)
    if (n <= 1024) ND_SMALL(1);
    else if (n <= 2048) ND_SMALL(2);
    else ND_SMALL(4);
#undef ND_SMALL
    c->launches++;
}

// Digit counts per tile of keys that come from elsewhere.
__global__ void k_rs_count(const uint32_t* __restrict__ keys, int32_t n, uint32_t* __restrict__ hist) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) atomicAdd(&hist[(i / pass_tile(n)) * RS_BINS + (keys[i] & 0xffu)], 1u);
}

// One pass over one tile of 1,024 keys per group of eight warps (GROUPS = 1,
// 2, 4): hist[tile][digit] are this pass's counts, hist_next (null in the last
// pass) receives the next pass's.
template <int GROUPS>
__global__ void __launch_bounds__(256 * GROUPS)
    k_rs_pass(const uint32_t* __restrict__ kin, const int32_t* __restrict__ vin,
              uint32_t* __restrict__ kout, int32_t* __restrict__ vout, int32_t n, int shift,
              const uint32_t* __restrict__ hist, uint32_t* __restrict__ hist_next, int32_t ntiles) {
    constexpr int ITEMS = 4, THREADS = 256 * GROUPS, W = 8 * GROUPS, TILE = THREADS * ITEMS;
    __shared__ __align__(4) uint16_t s_cnt[W][RS_BINS];
    __shared__ uint32_t s_pre[GROUPS][RS_BINS], s_tot[GROUPS][RS_BINS], s_part[GROUPS][RS_BINS];
    __shared__ uint32_t s_base[RS_BINS], s_warp[8];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, d = t & 255, g = t >> 8;
    const int32_t tile = blockIdx.x;
    const int64_t at0 = (int64_t)tile * TILE + w * 32 * ITEMS + lane;
    uint32_t key[ITEMS], dg[ITEMS], rank[ITEMS];
    int32_t val[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int64_t k = at0 + 32 * i;
        key[i] = k < n ? kin[k] : 0u;
        val[i] = k < n ? vin[k] : 0;
    }
    for (int k = t; k < W * RS_BINS / 2; k += THREADS) reinterpret_cast<uint32_t*>(s_cnt)[k] = 0u;
    uint32_t pre = 0, tot = 0;
    constexpr int ROWS = GROUPS == 1 ? 32 : 16;  // in flight a thread
    for (int32_t r0 = g; r0 < ntiles; r0 += ROWS * GROUPS) {
        uint32_t v[ROWS];
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
            const int32_t r = r0 + GROUPS * k;
            v[k] = r < ntiles ? __ldg(&hist[r * RS_BINS + d]) : 0u;
        }
#pragma unroll
        for (int k = 0; k < ROWS; ++k) {
            tot += v[k];
            pre += r0 + GROUPS * k < tile ? v[k] : 0u;
        }
    }
    s_pre[g][d] = pre;
    s_tot[g][d] = tot;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) dg[i] = at0 + 32 * i < n ? (key[i] >> shift) & 0xffu : 256u;
    __syncthreads();
    warp_ranks<ITEMS>(dg, s_cnt[w], rank);
    uint32_t all = 0, before = 0;
#pragma unroll
    for (int k = 0; k < GROUPS; ++k) { all += s_tot[k][d]; before += s_pre[k][d]; }
    const uint32_t ex = digits_scan(all, s_warp);  // (a barrier inside)
    if (g == 0) s_base[d] = ex + before;
    uint32_t sum = 0, c8[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) { c8[k] = s_cnt[8 * g + k][d]; sum += c8[k]; }
    s_part[g][d] = sum;
    __syncthreads();
    // positions of the warps' first items relative to the digit's first here
    // (they fit 16 bits)
    uint32_t run = 0;
    for (int k = 0; k < g; ++k) run += s_part[k][d];
#pragma unroll
    for (int k = 0; k < 8; ++k) { s_cnt[8 * g + k][d] = (uint16_t)run; run += c8[k]; }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if (dg[i] < 256u) {
            const uint32_t pos = s_base[dg[i]] + s_cnt[w][dg[i]] + rank[i];
            kout[pos] = key[i];
            vout[pos] = val[i];
            if (hist_next)
                atomicAdd(&hist_next[(pos / TILE) * RS_BINS + ((key[i] >> (shift + 8)) & 0xffu)], 1u);
        }
}

__global__ void __launch_bounds__(RS_THREADS)
    k_rs_upsweep(const uint32_t* __restrict__ keys, int32_t n, int shift,
                 uint32_t* __restrict__ hist, int32_t ntiles) {
    __shared__ uint32_t sh[RS_BINS];
    sh[threadIdx.x] = 0;
    __syncthreads();
    int64_t base = (int64_t)blockIdx.x * RS_TILE;
    const unsigned lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 0; k < RS_ITEMS; ++k) {
        int64_t idx = base + k * RS_THREADS + threadIdx.x;
        bool valid = idx < n;
        uint32_t dg = valid ? ((keys[idx] >> shift) & 0xffu) : 0x100u;
        unsigned peers = digit_peers(dg);
        if (valid && lane == (unsigned)(__ffs(peers) - 1)) atomicAdd(&sh[dg], (uint32_t)__popc(peers));
    }
    __syncthreads();
    hist[(int64_t)threadIdx.x * ntiles + blockIdx.x] = sh[threadIdx.x];
}

__device__ __forceinline__ uint32_t block_excl_scan_256(uint32_t v, uint32_t* s_warp,
                                                        uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, s);
        if (lane >= s) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (int)(blockDim.x >> 5) ? s_warp[lane] : 0u;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, s);
            if (lane >= s) w += y;
        }
        if (lane < (int)(blockDim.x >> 5)) s_warp[lane] = w;  // inclusive warp prefix
    }
    __syncthreads();
    uint32_t wp = warp ? s_warp[warp - 1] : 0u;
    if (total) *total = s_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return wp + x - v;
}

// One CTA per digit: exclusive scan of that digit's per-tile counts.
__global__ void __launch_bounds__(RS_THREADS)
    k_rs_scan(uint32_t* __restrict__ hist, int32_t ntiles, uint32_t* __restrict__ totals) {
    __shared__ uint32_t s_warp[32];
    uint32_t* h = hist + (int64_t)blockIdx.x * ntiles;
    uint32_t carry = 0;
    for (int32_t b = 0; b < ntiles; b += RS_THREADS) {
        int32_t i = b + threadIdx.x;
        uint32_t v = i < ntiles ? h[i] : 0u;
        uint32_t tot;
        uint32_t ex = block_excl_scan_256(v, s_warp, &tot);
        if (i < ntiles) h[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

__global__ void __launch_bounds__(RS_THREADS)
    k_rs_scatter(const uint32_t* __restrict__ kin, const int32_t* __restrict__ vin,
                 uint32_t* __restrict__ kout, int32_t* __restrict__ vout, int32_t n, int shift,
                 const uint32_t* __restrict__ hist, const uint32_t* __restrict__ totals,
                 int32_t ntiles) {
    constexpr int W = RS_THREADS / 32;
    __shared__ uint32_t s_base[RS_BINS];
    __shared__ uint32_t s_run[RS_BINS];
    __shared__ uint32_t s_wh[W][RS_BINS];
    __shared__ uint32_t s_warp[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t ex = block_excl_scan_256(totals[t], s_warp, nullptr);
    s_base[t] = ex + hist[(int64_t)t * ntiles + blockIdx.x];
    s_run[t] = 0;
    const unsigned lt = (1u << lane) - 1u;
    int64_t base = (int64_t)blockIdx.x * RS_TILE;
    for (int k = 0; k < RS_ITEMS; ++k) {
#pragma unroll
        for (int w = 0; w < W; ++w) s_wh[w][t] = 0;
        __syncthreads();
        int64_t idx = base + k * RS_THREADS + t;
        bool valid = idx < n;
        uint32_t key = valid ? kin[idx] : 0u;
        int32_t val = valid ? vin[idx] : 0;
        uint32_t dg = valid ? ((key >> shift) & 0xffu) : 0x100u;
        unsigned peers = digit_peers(dg);
        int rank = __popc(peers & lt);
        if (valid && lane == __ffs(peers) - 1) s_wh[warp][dg] = (uint32_t)__popc(peers);
        __syncthreads();
        {
            uint32_t run = s_run[t];
#pragma unroll
            for (int w = 0; w < W; ++w) {
                uint32_t cnt = s_wh[w][t];
                s_wh[w][t] = run;
                run += cnt;
            }
            s_run[t] = run;
        }
        __syncthreads();
        if (valid) {
            uint32_t pos = s_base[dg] + s_wh[warp][dg] + (uint32_t)rank;
            kout[pos] = key;
            vout[pos] = val;
        }
        __syncthreads();
    }
}

// The passes of the direct form; hist[0] already counted.  Results end in
// keys/vals.
static nd_status direct_passes(Ctx* c, uint32_t* keys, int32_t* vals, int32_t n, int passes) {
    const int32_t tile = pass_tile(n), ntiles = (int32_t)cdiv(n, tile);
    uint32_t* hist = (uint32_t*)c->hist.p;
    uint32_t *ka = keys, *kb = (uint32_t*)c->codes_alt.p;
    int32_t *va = vals, *vb = (int32_t*)c->perm_alt.p;
    const size_t row = (size_t)RS_BINS * ntiles;
    for (int p = 0; p < passes; ++p) {
#define ND_PASS(G)                                                                               \
    k_rs_pass<G><<<ntiles, 256 * G, 0, c->stream>>>(                                             \
        ka, va, kb, vb, n, 8 * p, hist + p * row, p + 1 < passes ? hist + (p + 1) * row : nullptr, \
        ntiles)
        if (tile == 1024) ND_PASS(1);
        else if (tile == 2048) ND_PASS(2);
        else ND_PASS(4);
#undef ND_PASS
        c->launches++;
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != keys) {
        cudaMemcpyAsync(keys, ka, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToDevice, c->stream);
        cudaMemcpyAsync(vals, va, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, c->stream);
    }
    return check_launch(c, "radix sort");
}

static nd_status sort_buffers(Ctx* c, int32_t n) {
    nd_status st;
    if ((st = ensure(c, c->codes_alt, sizeof(uint32_t) * (size_t)n))) return st;
    if ((st = ensure(c, c->perm_alt, sizeof(int32_t) * (size_t)n))) return st;
    return ensure(c, c->hist, sort_scratch_bytes(n));
}

static nd_status reset_counts(Ctx* c, int32_t n, int passes) {
    cudaError_t e = cudaMemsetAsync(
        c->hist.p, 0, sizeof(uint32_t) * RS_BINS * (size_t)cdiv(n, pass_tile(n)) * passes, c->stream);
    return e == cudaSuccess ? ND_OK : cuda_fail(c, e, "digit counts reset");
}

nd_status radix_sort_pairs(Ctx* c, uint32_t* keys, int32_t* vals, int32_t n, int bits) {
    if (n <= 1) return ND_OK;
    const int passes = (bits + 7) / 8;
    if (n <= kSmallSort) {
        small_order(c, nullptr, n, 0, nullptr, keys, vals, passes);
        return check_launch(c, "radix sort");
    }
    nd_status st = sort_buffers(c, n);
    if (st) return st;
    if (n <= kDirectKeys) {
        if ((st = reset_counts(c, n, passes))) return st;
        k_rs_count<<<(unsigned)cdiv(n, 256), 256, 0, c->stream>>>(keys, n, (uint32_t*)c->hist.p);
        c->launches++;
        return direct_passes(c, keys, vals, n, passes);
    }
    const int32_t ntiles = (int32_t)cdiv(n, RS_TILE);
    uint32_t* hist = (uint32_t*)c->hist.p;
    uint32_t* totals = hist + (size_t)RS_BINS * ntiles;
    uint32_t* ka = keys;
    int32_t* va = vals;
    uint32_t* kb = (uint32_t*)c->codes_alt.p;
    int32_t* vb = (int32_t*)c->perm_alt.p;
    for (int p = 0; p < passes; ++p) {
        int shift = 8 * p;
        k_rs_upsweep<<<ntiles, RS_THREADS, 0, c->stream>>>(ka, n, shift, hist, ntiles);
        k_rs_scan<<<RS_BINS, RS_THREADS, 0, c->stream>>>(hist, ntiles, totals);
        k_rs_scatter<<<ntiles, RS_THREADS, 0, c->stream>>>(ka, va, kb, vb, n, shift, hist, totals,
                                                          ntiles);
        c->launches += 3;
        std::swap(ka, kb);
        std::swap(va, vb);
    }
    if (ka != keys) {
        cudaMemcpyAsync(keys, ka, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToDevice, c->stream);
        cudaMemcpyAsync(vals, va, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToDevice, c->stream);
    }
    return check_launch(c, "radix sort");
}

nd_status order_positions(Ctx* c, const float* xyz, int32_t n, int32_t order, int32_t* codes,
                          int32_t* perm, const float* frame) {
    if (n <= 0) return ND_OK;
    if (n <= kSmallSort) {
        small_order(c, xyz, n, order, frame, (uint32_t*)codes, perm, 4);
        return check_launch(c, "order");
    }
    nd_status st;
    if (n > kDirectKeys) {
        if ((st = codes_kernels(c, xyz, n, order, codes, perm, frame, nullptr))) return st;
        return radix_sort_pairs(c, (uint32_t*)codes, perm, n, 30);
    }
    if ((st = sort_buffers(c, n)) || (st = reset_counts(c, n, 4))) return st;
    if ((st = codes_kernels(c, xyz, n, order, codes, perm, frame, (uint32_t*)c->hist.p))) return st;
    return direct_passes(c, (uint32_t*)codes, perm, n, 4);
}

// ============================================================== leaf boxes

// Gather sorted positions and build leaf boxes: leafcluster_primitives
// (BVHTraverse.jl:376-410, h = r/2) or cluster_primitives (:341-375, h = r).
// pos4.w carries the 1-based original index (bit pattern).
__global__ void k_leaf_boxes(const float* __restrict__ xyz, const int32_t* __restrict__ perm,
                             int32_t nL, int32_t apl, float h, float4* __restrict__ pos4,
                             int32_t* __restrict__ idx, float4* __restrict__ keys) {
    int32_t leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= nL) return;
    int64_t bird = (int64_t)leaf * apl;
    float mn[3], mx[3];
    for (int32_t a = 0; a < apl; ++a) {
        int32_t o = perm[bird + a];
        float p[3] = {xyz[3 * (int64_t)o], xyz[3 * (int64_t)o + 1], xyz[3 * (int64_t)o + 2]};
        pos4[bird + a] = make_float4(p[0], p[1], p[2], __int_as_float(o + 1));
        idx[bird + a] = o + 1;
        if (a == 0) {
#pragma unroll
            for (int d = 0; d < 3; ++d) { mn[d] = __fsub_rn(p[d], h); mx[d] = __fadd_rn(p[d], h); }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            mn[d] = jl_min(mn[d], __fsub_rn(p[d], h));
            mx[d] = jl_max(mx[d], __fadd_rn(p[d], h));
        }
    }
    keys[2 * (int64_t)leaf] = make_float4(mn[0], mn[1], mn[2], mx[0]);
    keys[2 * (int64_t)leaf + 1] = make_float4(mx[1], mx[2], __int_as_float(0), __int_as_float(0));
}

// ==================================================================== build

// exptdelta (BVHTraverse.jl:677-696), 1-based leaf index, Int32 wrap-around.
__device__ __forceinline__ int32_t delta_ref(int32_t i, const int32_t* __restrict__ code,
                                             int32_t nL, int32_t apl) {
    if (i >= nL || i < 1) return INT32_MAX;
    int32_t a = __ldg(&code[(int64_t)(i - 1) * apl]);
    int32_t b = __ldg(&code[(int64_t)i * apl]);
    uint32_t x = (uint32_t)(a ^ b);
    uint32_t add = (x == 0u) ? (0x80000000u + (uint32_t)(i ^ (i + 1))) : 0u;
    return (int32_t)(x + add - 1u);
}

__device__ __forceinline__ void load_box_cg(const float4* keys, int32_t node /*1-based*/,
                                            float mn[3], float mx[3]) {
    float4 a = __ldcg(&keys[2 * (int64_t)(node - 1)]);
    float4 b = __ldcg(&keys[2 * (int64_t)(node - 1) + 1]);
    mn[0] = a.x; mn[1] = a.y; mn[2] = a.z;
    mx[0] = a.w; mx[1] = b.x; mx[2] = b.y;
}

// bvh_interior! (BVHTraverse.jl:704-846), one thread per leaf.  The second
// thread to reach an internal node (the CAS on store[split] returns non-zero)
// merges the sibling box and continues upward.  __threadfence() before the CAS
// publishes this thread's node writes; the fence after a successful read of a
// non-zero slot orders the sibling-box loads, which bypass L1 (ld.cg).  No
// thread ever waits on another, so the kernel cannot hang; a climb longer than
// nL levels flags ND_ERR_INTERNAL.  gate (may be null): nothing is done while
// *gate is 0.
__global__ void k_bvh_build(float4* keys, int32_t* store, const int32_t* __restrict__ code,
                            int32_t nL, int32_t apl, int32_t* err,
                            const unsigned* __restrict__ gate) {
    int32_t i = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (i > nL || (gate && *gate == 0u)) return;
    int32_t rangel = i, ranger = i;
    int32_t dell = delta_ref(rangel - 1, code, nL, apl);
    int32_t delr = delta_ref(ranger, code, nL, apl);
    float bmin[3], bmax[3];
    load_box_cg(keys, i, bmin, bmax);
    int32_t lskip;
    if (i == nL) {
        lskip = 0;
    } else {
        int32_t ir = i + 1;
        lskip = (delr < delta_ref(ir, code, nL, apl)) ? ir : nL + ir;
    }
    reinterpret_cast<int32_t*>(&keys[2 * (int64_t)(i - 1) + 1])[3] = lskip;

    for (int32_t guard = 0; guard <= nL + 1; ++guard) {
        int32_t leftChild;
        int32_t sib;
        if (delr < dell) {
            leftChild = i;
            int32_t split = ranger;
            __threadfence();
            ranger = atomicCAS(&store[split - 1], 0, rangel);
            if (ranger == 0) return;
            __threadfence();
            delr = delta_ref(ranger, code, nL, apl);
            sib = split + 1;
            if (sib != ranger) sib = nL + sib;
        } else {
            int32_t split = rangel - 1;
            __threadfence();
            rangel = atomicCAS(&store[split - 1], 0, ranger);
            if (rangel == 0) return;
            __threadfence();
            dell = delta_ref(rangel - 1, code, nL, apl);
            leftChild = split;
            if (leftChild != rangel) leftChild = nL + leftChild;
            sib = leftChild;
        }
        float smin[3], smax[3];
        load_box_cg(keys, sib, smin, smax);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            bmax[d] = jl_max(smax[d], bmax[d]);
            bmin[d] = jl_min(smin[d], bmin[d]);
        }
        int32_t q = (delr < dell) ? ranger : rangel;
        int32_t parent = nL + q;
        int32_t skip;
        if (ranger == nL) {
            skip = 0;
        } else {
            int32_t r = ranger + 1;
            skip = (delr < delta_ref(r, code, nL, apl)) ? r : nL + r;
        }
        __stcg(&keys[2 * (int64_t)(parent - 1)], make_float4(bmin[0], bmin[1], bmin[2], bmax[0]));
        __stcg(&keys[2 * (int64_t)(parent - 1) + 1],
               make_float4(bmax[1], bmax[2], __int_as_float(leftChild), __int_as_float(skip)));
        i = parent;
        if (i == nL + 1) return;
    }
    set_error(err, ND_ERR_INTERNAL, i);
}

__global__ void k_root_overwrite(float4* keys, int32_t nL) {
    // bounding_volume_hierarchy! (BVHTraverse.jl:856-858) forces the root box to [0,1]^3.
    float4 b = keys[2 * (int64_t)nL + 1];
    keys[2 * (int64_t)nL] = make_float4(0.f, 0.f, 0.f, 1.f);
    keys[2 * (int64_t)nL + 1] = make_float4(1.f, 1.f, b.z, b.w);
}

nd_status build_internal_nodes(Ctx* c, float4* keys, int32_t* store, const int32_t* codes,
                               int32_t nL, int32_t apl, const unsigned* gate) {
    cudaError_t e = cudaMemsetAsync(store, 0, sizeof(int32_t) * (size_t)(nL - 1), c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "store reset");
    k_bvh_build<<<(int)cdiv(nL, 256), 256, 0, c->stream>>>(keys, store, codes, nL, apl, c->d_err, gate);
    c->launches++;
    return check_launch(c, "bvh build");
}

nd_status build_tree(Ctx* c, const float* xyz_dev, int32_t n, float r, int32_t apl,
                     int32_t order, int32_t boxes, int64_t nkeys, bool overwrite_root,
                     TreeBuffers* out, bool leaves_only) {
    int32_t nL = n / apl;
    nd_status st;
    if ((st = ensure(c, c->codes, sizeof(int32_t) * (size_t)n))) return st;
    if ((st = ensure(c, c->perm, sizeof(int32_t) * (size_t)n))) return st;
    if ((st = ensure(c, c->pos4, sizeof(float4) * (size_t)n))) return st;
    if ((st = ensure(c, c->idx, sizeof(int32_t) * (size_t)n))) return st;
    if ((st = ensure(c, c->keys, 32 * (size_t)nkeys))) return st;
    if ((st = ensure(c, c->store, sizeof(int32_t) * (size_t)std::max(nL - 1, 1)))) return st;
    int32_t* codes = (int32_t*)c->codes.p;
    int32_t* perm = (int32_t*)c->perm.p;
    if ((st = order_positions(c, xyz_dev, n, order, codes, perm))) return st;
    float4* keys = (float4*)c->keys.p;
    if (!leaves_only) {
        cudaError_t e = cudaMemsetAsync(keys, 0, 32 * (size_t)nkeys, c->stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "keys reset");
    }
    float h = (boxes == ND_BOX_LEAF) ? r / 2.0f : r;
    k_leaf_boxes<<<(int)cdiv(nL, 128), 128, 0, c->stream>>>(xyz_dev, perm, nL, apl, h,
                                                           (float4*)c->pos4.p,
                                                           (int32_t*)c->idx.p, keys);
    c->launches++;
    if ((st = check_launch(c, "leaf boxes"))) return st;
    if (!leaves_only &&
        (st = build_internal_nodes(c, keys, (int32_t*)c->store.p, codes, nL, apl)))
        return st;
    if (overwrite_root) {
        k_root_overwrite<<<1, 1, 0, c->stream>>>(keys, nL);
        c->launches++;
    }
    out->n = n;
    out->nL = nL;
    out->apl = apl;
    out->codes = codes;
    out->perm = perm;
    out->pos4 = (const float4*)c->pos4.p;
    out->idx = (const int32_t*)c->idx.p;
    out->keys = keys;
    out->nkeys = nkeys;
    out->internal = !leaves_only;
    return check_launch(c, "tree");
}

// Sorted -> original permutation (0-based) from the 1-based original indices
// of a kept order.
__global__ void k_kept_perm(const int32_t* __restrict__ idx1, int32_t n, int32_t* __restrict__ perm) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) perm[i] = idx1[i] - 1;
}

// Tree of new positions in a kept order: the sorted codes and the order of an
// earlier build are reused, so the Apetrei build (which depends on the sorted
// codes only) reproduces that build's topology, and the leaf and internal
// boxes are those of the new positions -- the refit that TreeData!
// (src/Neighbors/BVHTraverse.jl:601-655) intends between rebuilds.  idx1 and
// codes are device arrays (1-based original index and code, sorted order).
nd_status build_tree_kept(Ctx* c, const float* xyz_dev, int32_t n, float r, int32_t apl,
                          const int32_t* idx1, const int32_t* codes_sorted, int64_t nkeys,
                          TreeBuffers* out) {
    int32_t nL = n / apl;
    nd_status st;
    if ((st = ensure(c, c->perm, sizeof(int32_t) * (size_t)n))) return st;
    if ((st = ensure(c, c->pos4, sizeof(float4) * (size_t)n))) return st;
    if ((st = ensure(c, c->idx, sizeof(int32_t) * (size_t)n))) return st;
    if ((st = ensure(c, c->keys, 32 * (size_t)nkeys))) return st;
    if ((st = ensure(c, c->store, sizeof(int32_t) * (size_t)std::max(nL - 1, 1)))) return st;
    int32_t* perm = (int32_t*)c->perm.p;
    k_kept_perm<<<(unsigned)cdiv(n, 256), 256, 0, c->stream>>>(idx1, n, perm);
    c->launches++;
    float4* keys = (float4*)c->keys.p;
    cudaError_t e = cudaMemsetAsync(keys, 0, 32 * (size_t)nkeys, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "keys reset");
    k_leaf_boxes<<<(int)cdiv(nL, 128), 128, 0, c->stream>>>(xyz_dev, perm, nL, apl, r / 2.0f,
                                                           (float4*)c->pos4.p,
                                                           (int32_t*)c->idx.p, keys);
    c->launches++;
    if ((st = check_launch(c, "kept leaf boxes"))) return st;
    if ((st = build_internal_nodes(c, keys, (int32_t*)c->store.p, codes_sorted, nL, apl)))
        return st;
    out->n = n;
    out->nL = nL;
    out->apl = apl;
    out->codes = codes_sorted;
    out->perm = perm;
    out->pos4 = (const float4*)c->pos4.p;
    out->idx = (const int32_t*)c->idx.p;
    out->keys = keys;
    out->nkeys = nkeys;
    out->internal = true;
    return check_launch(c, "kept tree");
}

// bounding_volume_hierarchy!'s root-box overwrite on a built tree.
void root_overwrite(Ctx* c, float4* keys, int32_t nL) {
    k_root_overwrite<<<1, 1, 0, c->stream>>>(keys, nL);
    c->launches++;
}

// ==================================================================== scan

constexpr int SC_THREADS = 1024;
constexpr int SC_ITEMS = 4;
constexpr int SC_TILE = SC_THREADS * SC_ITEMS;

// Exclusive scan inside each tile; partial[] receives the tile sums.  A scan
// of one tile writes the grand total itself.
__global__ void __launch_bounds__(SC_THREADS)
    k_scan_tile(const int64_t* __restrict__ in, int64_t* __restrict__ out, int64_t n,
                int64_t* __restrict__ partial, int64_t* __restrict__ total) {
    __shared__ int64_t s_warp[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int64_t base = (int64_t)blockIdx.x * SC_TILE + (int64_t)t * SC_ITEMS;
    int64_t v[SC_ITEMS];
    int64_t sum = 0;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) {
        v[k] = (base + k < n) ? in[base + k] : 0;
        sum += v[k];
    }
    int64_t x = sum;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        int64_t y = __shfl_up_sync(0xffffffffu, x, s);
        if (lane >= s) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int64_t w = s_warp[lane];
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            int64_t y = __shfl_up_sync(0xffffffffu, w, s);
            if (lane >= s) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    int64_t run = (warp ? s_warp[warp - 1] : 0) + x - sum;
#pragma unroll
    for (int k = 0; k < SC_ITEMS; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (t == SC_THREADS - 1) {
        if (partial) partial[blockIdx.x] = s_warp[31];
        if (total) *total = s_warp[31];
    }
}

__global__ void k_scan_add(int64_t* __restrict__ out, int64_t n, const int64_t* __restrict__ add) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] += add[i / SC_TILE];
}

static nd_status scan_rec(Ctx* c, const int64_t* in, int64_t* out, int64_t n, int64_t* scratch,
                          size_t scratch_elems, int64_t* total) {
    int64_t nb = cdiv(n, SC_TILE);
    if (nb <= 1) {
        k_scan_tile<<<1, SC_THREADS, 0, c->stream>>>(in, out, n, nullptr, total);
        c->launches++;
        return check_launch(c, "scan");
    }
    if ((size_t)(2 * nb) > scratch_elems) return ND_ERR_INTERNAL;
    int64_t* part = scratch;
    int64_t* part_scan = scratch + nb;
    k_scan_tile<<<(unsigned)nb, SC_THREADS, 0, c->stream>>>(in, out, n, part, nullptr);
    c->launches++;
    nd_status st =
        scan_rec(c, part, part_scan, nb, scratch + 2 * nb, scratch_elems - 2 * nb, total);
    if (st) return st;
    k_scan_add<<<(unsigned)cdiv(n, 256), 256, 0, c->stream>>>(out, n, part_scan);
    c->launches++;
    return check_launch(c, "scan add");
}

nd_status scan_exclusive(Ctx* c, const int64_t* in, int64_t* out, int64_t n, int64_t* total_dev) {
    if (n <= 0) {
        cudaMemsetAsync(total_dev, 0, sizeof(int64_t), c->stream);
        return ND_OK;
    }
    size_t need = 4 * (size_t)cdiv(n, SC_TILE) + 64;
    nd_status st = ensure(c, c->partial, sizeof(int64_t) * need);
    if (st) return st;
    return scan_rec(c, in, out, n, (int64_t*)c->partial.p, need, total_dev);
}

// =============================================================== traversal

struct Node {
    float mnx, mny, mnz, mxx, mxy, mxz;
    int32_t left, skip;
};

__device__ __forceinline__ Node load_node(const float4* __restrict__ keys, int32_t k /*1-based*/) {
    float4 a = __ldg(&keys[2 * (int64_t)(k - 1)]);
    float4 b = __ldg(&keys[2 * (int64_t)(k - 1) + 1]);
    Node nd_;
    nd_.mnx = a.x; nd_.mny = a.y; nd_.mnz = a.z; nd_.mxx = a.w; nd_.mxy = b.x; nd_.mxz = b.y;
    nd_.left = __float_as_int(b.z);
    nd_.skip = __float_as_int(b.w);
    return nd_;
}

// aabb_overlap_test (BVHTraverse.jl:1094-1098), strict on all three axes.
__device__ __forceinline__ bool overlap(const Node& a, const Node& b) {
    return (a.mnx < b.mxx) & (a.mxx > b.mnx) & (a.mny < b.mxy) & (a.mxy > b.mny) &
           (a.mnz < b.mxz) & (a.mxz > b.mnz);
}

// Rounding slack of leaf a's box coordinates: 8 ulps of the largest.
__device__ __forceinline__ float leaf_slack(const Node& a) {
    const float mag = fmaxf(fmaxf(fmaxf(fabsf(a.mnx), fabsf(a.mxx)), fmaxf(fabsf(a.mny), fabsf(a.mxy))),
                            fmaxf(fabsf(a.mnz), fabsf(a.mxz)));
    return mag * 9.5367431640625e-7f;  // 8 * 2^-23
}

// The limit r2g of the gap filter below, computed once a launch: r^2 or the
// threshold on d^2 (above r^2 where r^2 underflows), widened a little, at the
// bottom of the range by a few of its steps.
static float gap_limit(float r, float r2) {
    return std::fma(std::fmax(r * r, r2), 1.0001f, 1e-44f);
}

// Whether two leaves whose key boxes (atom boxes -/+ r/2) overlap can hold a
// pair within r: the per-axis gaps of the atom boxes (key-box gap + r, each
// lowered by the rounding slack of the -/+ r/2) must have a Euclidean norm
// below r (r2g = gap_limit: a filter, the distance test decides).
// Boxes that overlap on every axis only bound each gap by r; this drops the
// leaf pairs diagonally apart.
__device__ __forceinline__ bool leaf_gap_ok(const Node& a, const Node& b, float r, float r2g,
                                            float slack) {
    const float gx = fmaxf(fmaxf(a.mnx - b.mxx, b.mnx - a.mxx) + r - slack, 0.0f);
    const float gy = fmaxf(fmaxf(a.mny - b.mxy, b.mny - a.mxy) + r - slack, 0.0f);
    const float gz = fmaxf(fmaxf(a.mnz - b.mxz, b.mnz - a.mxz) + r - slack, 0.0f);
    return gx * gx + gy * gy + gz * gz < r2g;
}

// Emission sinks of the walks: Count counts, Write and Triples write at a running
// cursor.
struct SinkCount {
    int64_t n = 0;
    __device__ __forceinline__ void push(int32_t, int32_t, float) { ++n; }
};
struct SinkWrite {
    int32_t* pi; int32_t* pj; float* pd;
    int64_t cur;
    __device__ __forceinline__ void push(int32_t i, int32_t j, float d) {
        pi[cur] = i; pj[cur] = j; pd[cur] = d; ++cur;
    }
};

struct SinkTriples {
    int32_t* out;
    int64_t cur;
    __device__ __forceinline__ void push(int32_t i, int32_t j, float d) {
        int32_t* o = out + 3 * cur++;
        o[0] = i; o[1] = j; o[2] = __float_as_int(d);
    }
};

// A rope walk visits every node at most once; a longer walk or a node index
// outside [1, 2nL-1] can only come from a corrupted tree and is reported
// instead of looping.
#define ND_WALK_GUARD(t, nnodes, visits, err, who)                          \
    if ((t) < 1 || (t) > (nnodes) || ++(visits) > (nnodes)) {               \
        set_error((err), ND_ERR_INTERNAL, (who));                           \
        break;                                                              \
    }

// neighbor_traverse (BVHTraverse.jl:1143-1181) for one query atom qi (1-based, sorted).
template <class Sink>
__device__ __forceinline__ void atom_query(int32_t qi, const float4* __restrict__ keys,
                                           const float4* __restrict__ pos, int32_t apl, float r2,
                                           int32_t nnodes, int32_t* err, Sink& s) {
    float4 p = __ldg(&pos[qi - 1]);
    int32_t t = (qi + apl - 1) / apl;
    int32_t visits = 0;
    while (t != 0) {
        ND_WALK_GUARD(t, nnodes, visits, err, qi)
        Node nd_ = load_node(keys, t);
        bool in = (nd_.mnx < p.x) & (p.x < nd_.mxx) & (nd_.mny < p.y) & (p.y < nd_.mxy) &
                  (nd_.mnz < p.z) & (p.z < nd_.mxz);
        if (in) {
            if (nd_.left == 0) {
                int32_t low = (t - 1) * apl + 1;
                for (int32_t e = 1; e <= apl; ++e) {
                    int32_t sidx = low + e - 1;
                    if (qi < e + low) {
                        float4 b = __ldg(&pos[sidx - 1]);
                        if (__float_as_int(p.w) != __float_as_int(b.w)) {
                            float d2 = dist2_ref(p.x, p.y, p.z, b.x, b.y, b.z);
                            if (d2 < r2) s.push(__float_as_int(p.w), __float_as_int(b.w), __fsqrt_rn(d2));
                        }
                    }
                }
                t = nd_.skip;
            } else {
                t = nd_.left;
            }
        } else {
            t = nd_.skip;
        }
    }
}

// ------------------------------------------- ordered emission, wide search
//
// leafneighbor_traverse visits the leaves after the query leaf q in index
// order and accepts those whose boxes overlap q's: a node's box holds its
// leaves' boxes exactly (min / max only), so a leaf overlapping q is reached
// whatever the topology above it.  The ordered list is therefore, for q
// ascending, the overlapping leaves t > q ascending, atoms of q outer, atoms
// of t inner, and any search that enumerates those leaves in order gives it.
// Here one warp searches for one query leaf over a 32-wide hierarchy of the
// sorted leaves (groups of 32 leaves, super-groups of 32 groups, and for many
// leaves two levels more, see kDirectSupers): 32 boxes are
// tested per step, one a lane, and the hits are taken in index order from the
// ballot.  A thread per leaf walking the binary tree's ropes, the form before,
// had 1 node load in flight a thread and wrote each thread's pairs to its own
// place: 262,144 atoms at density 0.83, r 2.5: count 237 and write 563 us, and
// 20,000 atoms in reference order (whose boxes overlap almost all others, no
// tree prunes them): 2.9 and 6.8 ms.

// The levels above nL leaves: groups of 32 leaves, super-groups of 32 groups,
// and so on.  Their boxes lie one level after the other, stored like leaf keys.
struct GroupLevels {
    int32_t ng, ns, n3, n4;
    __host__ __device__ explicit GroupLevels(int32_t nL)
        : ng((nL + 31) >> 5), ns((ng + 31) >> 5), n3((ns + 31) >> 5), n4((n3 + 31) >> 5) {}
    __host__ __device__ int64_t boxes() const { return (int64_t)ng + ns + n3 + n4; }
};

// Leaves above which an ordered list may come from rope walks (see sparse_leaves).
constexpr int32_t kWalkLeaves = 131072;

// Up to this many super-groups (262,144 leaves) they are tested 32 after 32;
// beyond, the two levels above them say which.  Testing them all grows with the
// square of the leaves: the ordered list of 4,194,304 points (density 0.83, r
// 1.3, four atoms a leaf) took 4.3 ms and takes 2.8, of 134,217,728 points (r
// 1.0) 2.5 s and 95 ms, the unordered one 96 and 39 ms.
constexpr int32_t kDirectSupers = 256;

// Boxes of the groups of 32 leaves at [0, ngroups) and of the super-groups of
// 32 groups after them, stored like leaf keys.  One warp per group, one block
// per super-group.
__global__ void __launch_bounds__(1024)
    k_group_boxes(const float4* __restrict__ keys, int32_t nL, float4* __restrict__ gbox) {
    __shared__ float s_b[32][6];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t ng = (nL + 31) >> 5, g = blockIdx.x * 32 + w;
    float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    const int64_t l = (int64_t)g * 32 + lane;
    if (l < nL) {
        const float4 a = __ldg(&keys[2 * l]), b = __ldg(&keys[2 * l + 1]);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y;
    }
    auto reduce = [&]() {
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                v[d] = fminf(v[d], __shfl_xor_sync(0xffffffffu, v[d], s));
                v[3 + d] = fmaxf(v[3 + d], __shfl_xor_sync(0xffffffffu, v[3 + d], s));
            }
    };
    reduce();
    if (lane == 0) {
        if (g < ng) {
            gbox[2 * (int64_t)g] = make_float4(v[0], v[1], v[2], v[3]);
            gbox[2 * (int64_t)g + 1] = make_float4(v[4], v[5], 0.f, 0.f);
        }
#pragma unroll
        for (int d = 0; d < 6; ++d) s_b[w][d] = v[d];
    }
    __syncthreads();
    if (w == 0) {
#pragma unroll
        for (int d = 0; d < 6; ++d) v[d] = s_b[lane][d];
        reduce();
        if (lane == 0) {
            const int64_t sb = ng + (int64_t)blockIdx.x;
            gbox[2 * sb] = make_float4(v[0], v[1], v[2], v[3]);
            gbox[2 * sb + 1] = make_float4(v[4], v[5], 0.f, 0.f);
        }
    }
}

// Boxes of the nodes of one level (nout of them at `out`) over 32 nodes each of
// the level below (nin at `in`).  One warp a node.
__global__ void __launch_bounds__(256)
    k_upper_boxes(const float4* __restrict__ in, int32_t nin, float4* __restrict__ out, int32_t nout) {
    const int lane = threadIdx.x & 31;
    const int32_t o = (int32_t)blockIdx.x * 8 + (int32_t)(threadIdx.x >> 5);
    if (o >= nout) return;  // whole warp
    float v[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
    const int64_t i = (int64_t)o * 32 + lane;
    if (i < nin) {
        const float4 a = __ldg(&in[2 * i]), b = __ldg(&in[2 * i + 1]);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            v[d] = fminf(v[d], __shfl_xor_sync(0xffffffffu, v[d], s));
            v[3 + d] = fmaxf(v[3 + d], __shfl_xor_sync(0xffffffffu, v[3 + d], s));
        }
    if (lane == 0) {
        out[2 * (int64_t)o] = make_float4(v[0], v[1], v[2], v[3]);
        out[2 * (int64_t)o + 1] = make_float4(v[4], v[5], 0.f, 0.f);
    }
}

// The boxes of the groups and super-groups, and (upper) of the levels above.
static void group_boxes(Ctx* c, const float4* keys, int32_t nL, float4* gbox, bool upper) {
    const GroupLevels v(nL);
    k_group_boxes<<<(unsigned)v.ns, 1024, 0, c->stream>>>(keys, nL, gbox);
    c->launches++;
    if (!upper) return;
    float4* sbox = gbox + 2 * (int64_t)v.ng;
    float4* box3 = sbox + 2 * (int64_t)v.ns;
    k_upper_boxes<<<(unsigned)cdiv(v.n3, 8), 256, 0, c->stream>>>(sbox, v.ns, box3, v.n3);
    k_upper_boxes<<<(unsigned)cdiv(v.n4, 8), 256, 0, c->stream>>>(box3, v.n3,
                                                                  box3 + 2 * (int64_t)v.n3, v.n4);
    c->launches += 2;
}

// Every group >= g0 that overlaps box q, in index order: hit(base, m) is called
// by the whole warp for 32 consecutive groups at a time, bit k of m telling
// whether group base + k overlaps.  DEEP: more than kDirectSupers super-groups.
template <bool DEEP, class F>
__device__ __forceinline__ void wide_groups(const Node& q, int32_t g0,
                                            const float4* __restrict__ gbox, int32_t nL, F&& hit) {
    const int lane = threadIdx.x & 31;
    const int32_t ng = (nL + 31) >> 5, ns = (ng + 31) >> 5;
    const int32_t s0 = g0 >> 5;
    // super-groups sb .. sb + 31
    auto supers = [&](int32_t sb) {
        const int32_t s = sb + lane;
        unsigned sm = __ballot_sync(0xffffffffu, s >= s0 && s < ns &&
                                                     overlap(q, load_node(gbox, ng + min(s, ns - 1) + 1)));
        while (sm) {
            const int32_t base = (sb + __ffs(sm) - 1) * 32, g = base + lane;
            sm &= sm - 1;
            hit(base, __ballot_sync(0xffffffffu, g >= g0 && g < ng &&
                                                     overlap(q, load_node(gbox, min(g, ng - 1) + 1))));
        }
    };
    if constexpr (!DEEP) {
        for (int32_t sb = s0; sb < ns; sb += 32) supers(sb);
    } else {
        const GroupLevels v(nL);
        const int32_t t0 = s0 >> 5, f0 = t0 >> 5;
        const float4* __restrict__ box3 = gbox + 2 * ((int64_t)ng + ns);
        const float4* __restrict__ box4 = box3 + 2 * (int64_t)v.n3;
        for (int32_t b4 = f0; b4 < v.n4; b4 += 32) {
            const int32_t f = b4 + lane;
            unsigned m4 = __ballot_sync(
                0xffffffffu, f < v.n4 && overlap(q, load_node(box4, min(f, v.n4 - 1) + 1)));
            while (m4) {
                const int32_t b3 = (b4 + __ffs(m4) - 1) * 32, t = b3 + lane;
                m4 &= m4 - 1;
                unsigned m3 = __ballot_sync(0xffffffffu,
                                            t >= t0 && t < v.n3 &&
                                                overlap(q, load_node(box3, min(t, v.n3 - 1) + 1)));
                while (m3) {
                    supers((b3 + __ffs(m3) - 1) * 32);
                    m3 &= m3 - 1;
                }
            }
        }
    }
}

// Every leaf t >= t0 (0-based) that overlaps box q, in index order: hit(t,
// box, in) is called by the whole warp for 32 consecutive leaves at a time,
// `in` telling whether this lane's leaf overlaps.
template <bool DEEP, class F>
__device__ __forceinline__ void wide_search(const Node& q, int32_t t0,
                                            const float4* __restrict__ keys,
                                            const float4* __restrict__ gbox, int32_t nL, F&& hit) {
    const int lane = threadIdx.x & 31;
    wide_groups<DEEP>(q, t0 >> 5, gbox, nL, [&](int32_t base, unsigned m) {
        while (m) {
            const int32_t t = (base + __ffs(m) - 1) * 32 + lane;
            m &= m - 1;
            const Node b = load_node(keys, min(t, nL - 1) + 1);
            hit(t, b, t >= t0 && t < nL && overlap(q, b));
        }
    });
}

// One warp per query leaf (DEEP: per leaf of `list`, of nq leaves, if there is
// one).  WRITE 0: counts[q] = its pairs; 1: its pairs at
// offsets[q] .. in three arrays (nothing when the total exceeds cap); 2: the
// same as triples of words in pi.
// APL 2 or 4: the overlapping leaves go through a queue of candidates so that
// 32 of them, one a lane, are tested together (in a box about 30 leaves
// overlap one, three of each group of 32): each lane has the APL x APL tests
// of its leaf as a bit mask, lane order and bit order are the list order, and
// the hits leave through shared memory as contiguous runs.  APL 0 (any other
// width): the warp runs the apl^2 tests of one leaf pair together, 32 at a
// time in list order.
template <int APL, int WRITE, bool DEEP>
__global__ void __launch_bounds__(128)
    k_leaf_wide(const float4* __restrict__ keys, const float4* __restrict__ gbox,
                const float4* __restrict__ pos, int32_t nL, int32_t apl, float r, float r2,
                float r2g, int64_t* __restrict__ counts, const int64_t* __restrict__ offsets,
                const int64_t* __restrict__ total, int64_t cap, int32_t* __restrict__ pi,
                int32_t* __restrict__ pj, float* __restrict__ pd, const int32_t* __restrict__ list,
                int32_t nq) {
    constexpr int BUF = APL > 0 && WRITE != 0 ? 32 * APL * APL : 1;
    __shared__ int2 sbij[4][BUF];
    __shared__ float sbd[4][BUF];
    __shared__ int32_t squeue[4][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t q = (int32_t)blockIdx.x * 4 + w;
    if (q >= (DEEP ? nq : nL)) return;  // whole warp
    if (DEEP && list) q = __ldg(&list[q]);
    int64_t cur = 0;
    if (WRITE) {
        if (*total > cap) return;
        cur = offsets[q];
    }
    const unsigned below = (1u << lane) - 1u;
    const Node ql = load_node(keys, q + 1);
    const float slack = leaf_slack(ql);
    if constexpr (APL > 0) {
        int32_t* queue = squeue[w];
        float4 qa[APL];
#pragma unroll
        for (int i = 0; i < APL; ++i) qa[i] = __ldg(&pos[(int64_t)q * APL + i]);
        int mine = 0;
        auto test = [&](int32_t nc) {
            unsigned mask = 0;
            float d2[APL * APL];
            float4 tb[APL];
            if (lane < nc) {
                const int32_t t = queue[lane];
#pragma unroll
                for (int j = 0; j < APL; ++j) tb[j] = __ldg(&pos[(int64_t)t * APL + j]);
#pragma unroll
                for (int k = 0; k < APL * APL; ++k) {
                    const int i = k / APL, j = k % APL;
                    d2[k] = dist2_ref(qa[i].x, qa[i].y, qa[i].z, tb[j].x, tb[j].y, tb[j].z);
                    if (d2[k] < r2 && (t != q || j > i)) mask |= 1u << k;
                }
            }
            const int n = __popc(mask);
            if constexpr (!WRITE) {
                mine += n;
            } else {
                int at = n;  // inclusive scan over the lanes
#pragma unroll
                for (int s = 1; s < 32; s <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, at, s);
                    if (lane >= s) at += y;
                }
                const int tot = __shfl_sync(0xffffffffu, at, 31);
                at -= n;
#pragma unroll
                for (int k = 0; k < APL * APL; ++k)
                    if ((mask >> k) & 1u) {
                        sbij[w][at] = make_int2(__float_as_int(qa[k / APL].w),
                                                __float_as_int(tb[k % APL].w));
                        sbd[w][at] = d2[k];
                        ++at;
                    }
                __syncwarp();
                if constexpr (WRITE == 1) {
                    for (int k = lane; k < tot; k += 32) {
                        const int2 ij = sbij[w][k];
                        pi[cur + k] = ij.x;
                        pj[cur + k] = ij.y;
                        pd[cur + k] = __fsqrt_rn(sbd[w][k]);
                    }
                } else {
                    // the run's words in order, one a lane
                    int32_t* __restrict__ out = pi + 3 * cur;
                    for (int m = lane; m < 3 * tot; m += 32) {
                        const int k = m / 3, f = m - 3 * k;
                        const int2 ij = sbij[w][k];
                        out[m] = f == 0 ? ij.x : f == 1 ? ij.y : __float_as_int(__fsqrt_rn(sbd[w][k]));
                    }
                }
                cur += tot;
            }
            __syncwarp();
        };
        if (lane == 0) queue[0] = q;  // the pairs inside the leaf come first
        int32_t qn = 1;
        wide_search<DEEP>(ql, q + 1, keys, gbox, nL, [&](int32_t t, const Node& b, bool in) {
            const bool want = in && leaf_gap_ok(ql, b, r, r2g, slack);
            const unsigned m = __ballot_sync(0xffffffffu, want);
            if (want) queue[qn + __popc(m & below)] = t;  // < 64: qn < 32 here
            qn += __popc(m);
            __syncwarp();
            if (qn >= 32) {
                test(32);
                const int32_t rest = lane < qn - 32 ? queue[32 + lane] : 0;
                __syncwarp();
                if (lane < qn - 32) queue[lane] = rest;
                qn -= 32;
                __syncwarp();
            }
        });
        __syncwarp();
        if (qn > 0) test(qn);
        if constexpr (!WRITE) {
            const unsigned n = __reduce_add_sync(0xffffffffu, (unsigned)mine);
            if (lane == 0) counts[q] = n;
        }
    } else {
        int64_t n = 0;
        const int64_t A = (int64_t)q * apl;
        const int64_t tests = (int64_t)apl * apl;
        auto leaf = [&](int32_t t) {
            const int64_t B = (int64_t)t * apl;
            for (int64_t k0 = 0; k0 < tests; k0 += 32) {
                const int64_t k = k0 + lane;
                const int32_t i = (int32_t)(k / apl), j = (int32_t)(k - (int64_t)i * apl);
                bool hit = k < tests && (t != q || j > i);
                float4 a, b;
                float d2 = 0.0f;
                if (hit) {
                    a = __ldg(&pos[A + i]);
                    b = __ldg(&pos[B + j]);
                    d2 = dist2_ref(a.x, a.y, a.z, b.x, b.y, b.z);
                    hit = d2 < r2;
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (WRITE && hit) {
                    const int64_t at = cur + __popc(m & below);
                    if (WRITE == 1) {
                        pi[at] = __float_as_int(a.w);
                        pj[at] = __float_as_int(b.w);
                        pd[at] = __fsqrt_rn(d2);
                    } else {
                        pi[3 * at] = __float_as_int(a.w);
                        pi[3 * at + 1] = __float_as_int(b.w);
                        pi[3 * at + 2] = __float_as_int(__fsqrt_rn(d2));
                    }
                }
                if (WRITE) cur += __popc(m);
                else n += __popc(m);
            }
        };
        leaf(q);
        wide_search<DEEP>(ql, q + 1, keys, gbox, nL, [&](int32_t t, const Node& b, bool in) {
            unsigned m =
                __ballot_sync(0xffffffffu, in && leaf_gap_ok(ql, b, r, r2g, slack));
            const int32_t base = t - lane;
            while (m) {
                leaf(base + __ffs(m) - 1);
                m &= m - 1;
            }
        });
        if (!WRITE && lane == 0) counts[q] = n;
    }
}

// ------------------------------------------- ordered emission, rope walks
//
// leafneighbor_traverse (BVHTraverse.jl:1236-1323) as it is, a thread a leaf: the
// ropes of the binary tree lead past what does not overlap.  Each thread writes
// its pairs to its own place, and the walk has one node load in flight; but a
// walk is short where few leaves overlap, and the search above spends a warp and
// its chain of loads on every leaf (see sparse_leaves).  Leaves whose atoms extend
// further than `widest` are left to the search: the walk of one that spans two
// clusters is as long as hundreds of others'.
__device__ __forceinline__ float leaf_extent(const Node& b, float r) {
    return fmaxf(fmaxf(fmaxf(b.mxx - b.mnx, b.mxy - b.mny), b.mxz - b.mnz) - r, 0.0f);
}
template <int APL, int WRITE>
__global__ void __launch_bounds__(128)
    k_leaf_walk(const float4* __restrict__ keys, const float4* __restrict__ pos, int32_t nL,
                int32_t apl, float r, float r2, float widest, int64_t* __restrict__ counts,
                const int64_t* __restrict__ offsets, const int64_t* __restrict__ total, int64_t cap,
                int32_t* pi, int32_t* pj, float* pd, int32_t* err) {
    const int32_t q = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x) + 1;
    if (q > nL || (WRITE && *total > cap)) return;
    const Node ql = load_node(keys, q);
    if (leaf_extent(ql, r) > widest) return;
    const int32_t na = APL > 0 ? APL : apl, nnodes = 2 * nL - 1;
    const int64_t A = (int64_t)(q - 1) * na;
    auto run = [&](auto& s) {
        [[maybe_unused]] float4 qa[APL > 0 ? APL : 1];
        if constexpr (APL > 0)
#pragma unroll
            for (int i = 0; i < APL; ++i) qa[i] = __ldg(&pos[A + i]);
        // the atoms of leaf t (tri: only those behind the query atom)
        auto leaf = [&](int32_t t, bool tri) {
            const int64_t B = (int64_t)(t - 1) * na;
            if constexpr (APL > 0) {
                float4 tb[APL];
#pragma unroll
                for (int j = 0; j < APL; ++j) tb[j] = __ldg(&pos[B + j]);
#pragma unroll
                for (int i = 0; i < APL; ++i)
#pragma unroll
                    for (int j = 0; j < APL; ++j) {
                        const float d2 = dist2_ref(qa[i].x, qa[i].y, qa[i].z, tb[j].x, tb[j].y, tb[j].z);
                        if (d2 < r2 && (!tri || j > i))
                            s.push(__float_as_int(qa[i].w), __float_as_int(tb[j].w), __fsqrt_rn(d2));
                    }
            } else {
                for (int32_t i = 0; i < apl; ++i) {
                    const float4 a = __ldg(&pos[A + i]);
                    for (int32_t j = tri ? i + 1 : 0; j < apl; ++j) {
                        const float4 b = __ldg(&pos[B + j]);
                        const float d2 = dist2_ref(a.x, a.y, a.z, b.x, b.y, b.z);
                        if (d2 < r2) s.push(__float_as_int(a.w), __float_as_int(b.w), __fsqrt_rn(d2));
                    }
                }
            }
        };
        leaf(q, true);
        int32_t visits = 0;
        for (int32_t t = ql.skip; t != 0;) {
            ND_WALK_GUARD(t, nnodes, visits, err, q)
            const Node nd_ = load_node(keys, t);
            const bool in = overlap(ql, nd_);
            if (in && nd_.left == 0) leaf(t, false);
            t = in && nd_.left != 0 ? nd_.left : nd_.skip;
        }
    };
    if constexpr (WRITE == 0) {
        SinkCount s;
        run(s);
        counts[q - 1] = s.n;
    } else if constexpr (WRITE == 1) {
        SinkWrite s{pi, pj, pd, offsets[q - 1]};
        run(s);
    } else {
        SinkTriples s{pi, offsets[q - 1]};
        run(s);
    }
}

// What the choice between search and walk looks at: the leaves behind the query
// leaf that overlap it, summed over kSampled query leaves spread over all and the
// most of one, and the largest and the summed extent of the leaves' atoms (their
// widest axis).
struct LeafSample {
    unsigned long long overlaps;
    unsigned most;
    float widest;
    double extents;
};
constexpr int kSampled = 512;
template <bool DEEP>
__global__ void __launch_bounds__(128)
    k_overlap_sample(const float4* __restrict__ keys, const float4* __restrict__ gbox, int32_t nL,
                     LeafSample* out) {
    const int32_t k = (int32_t)(blockIdx.x * 4 + (threadIdx.x >> 5));
    const int32_t q = (int32_t)((int64_t)k * nL / kSampled);
    const Node ql = load_node(keys, q + 1);
    unsigned n = 0;
    wide_search<DEEP>(ql, q + 1, keys, gbox, nL, [&](int32_t, const Node&, bool in) { n += in; });
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&out->overlaps, (unsigned long long)n);
        atomicMax(&out->most, n);
    }
}
__global__ void __launch_bounds__(256)
    k_leaf_extents(const float4* __restrict__ keys, int32_t nL, float r, LeafSample* out) {
    float widest = 0.0f, sum = 0.0f;
    for (int64_t l = blockIdx.x * 256 + threadIdx.x; l < nL; l += (int64_t)gridDim.x * 256) {
        const float e = leaf_extent(load_node(keys, (int32_t)l + 1), r);
        widest = fmaxf(widest, e);
        sum += e;
    }
    const unsigned w = __reduce_max_sync(0xffffffffu, __float_as_uint(widest));  // (not negative)
    double d = sum;
    for (int s = 16; s > 0; s >>= 1) d += __shfl_xor_sync(0xffffffffu, d, s);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(reinterpret_cast<unsigned*>(&out->widest), w);
        atomicAdd(&out->extents, d);
    }
}

__global__ void __launch_bounds__(256)
    k_wide_leaves(const float4* __restrict__ keys, int32_t nL, float r, float widest, int32_t cap,
                  int32_t* __restrict__ list, unsigned long long* count) {
    const int32_t l = (int32_t)(blockIdx.x * 256 + threadIdx.x);
    if (l >= nL || !(leaf_extent(load_node(keys, l + 1), r) > widest)) return;
    const unsigned long long k = atomicAdd(count, 1ull);
    if (k < (unsigned long long)cap) list[k] = l;
}

// One-pass emission, warp-cooperative (atomsperleaf 4; the pair multiset of
// leafneighbor_traverse in an order decided at run time).  A warp
// takes 32 consecutive query leaves and walks the tree ONCE, from the skip
// rope of its first leaf, pruning with the union of its lanes' boxes; at
// every leaf t it reaches, each lane runs leafneighbor_traverse's leaf test
// for its own leaf q (t > q, strict box overlap -- the leaves a rope walk
// from q's skip would accept, since a box overlapping t overlaps all of t's
// ancestors) and the 4 x 4 distance tests.  Lanes stay converged, node loads
// are broadcast, and the pairs are ballot-compacted into a shared-memory
// buffer per warp that is written out with one atomic reservation and
// coalesced stores.
constexpr int kWarpBuf = 512;  // buffered pairs per warp (one leaf visit adds at most 512)

__device__ __forceinline__ void warp_buf_flush(int2* bij, float* bd, int& nb,
                                               unsigned long long* cursor, int64_t cap,
                                               int32_t* pi, int32_t* pj, float* pd) {
    const int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    if (lane == 0 && nb) base = atomicAdd(cursor, (unsigned long long)nb);
    base = __shfl_sync(0xffffffffu, base, 0);
    if ((int64_t)(base + (unsigned long long)nb) <= cap) {
        // the whole run fits: 32-bit offsets from the run's first slot
        int32_t* __restrict__ qi = pi + base;
        int32_t* __restrict__ qj = pj + base;
        float* __restrict__ qd = pd + base;
        for (int k = lane; k < nb; k += 32) {
            const int2 ij = bij[k];
            qi[k] = ij.x;
            qj[k] = ij.y;
            qd[k] = __fsqrt_rn(bd[k]);
        }
    } else {
        for (int k = lane; k < nb; k += 32) {
            const unsigned long long w = base + (unsigned long long)k;
            if ((int64_t)w < cap) {
                const int2 ij = bij[k];
                pi[w] = ij.x;
                pj[w] = ij.y;
                pd[w] = __fsqrt_rn(bd[k]);
            }
        }
    }
    __syncwarp();
    nb = 0;
}

// Appends this lane's hits (bit k of mask = pair (ia[k / 4], ib[k % 4]) at
// squared distance d2[k], the value the test compared) to the warp's buffer
// in bit-major order: for each k, the lanes holding bit k take consecutive
// slots, so every store of the warp is contiguous (no shared-memory bank
// conflicts).  The buffer holds squared distances; the flush writes their
// square roots, every lane of the flush taking one.
__device__ __forceinline__ void warp_emit16(unsigned mask, const float (&d2)[16],
                                            const int32_t (&ia)[4], const int32_t (&ib)[4],
                                            int2* bij, float* bd, int& nb,
                                            unsigned long long* cursor, int64_t cap, int32_t* pi,
                                            int32_t* pj, float* pd) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)__popc(mask));
    if (total == 0) return;
    if (nb + (int)total > kWarpBuf) warp_buf_flush(bij, bd, nb, cursor, cap, pi, pj, pd);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const bool hit = (mask >> k) & 1u;
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int at = nb + __popc(bal & below);
            bij[at] = make_int2(ia[k >> 2], ib[k & 3]);
            bd[at] = d2[k];
        }
        nb += __popc(bal);
    }
    __syncwarp();
}

// The 16 tests of leaf pair (a, b) (a == b: the six pairs inside the leaf):
// squared distances and the hit mask.
__device__ __forceinline__ unsigned leaf_tests16(const float4 (&qa)[4], const float4 (&tb)[4],
                                                 bool self, float r2, float (&d2)[16]) {
    unsigned mask = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const int i = k >> 2, j = k & 3;
        d2[k] = dist2_ref(qa[i].x, qa[i].y, qa[i].z, tb[j].x, tb[j].y, tb[j].z);
        if ((!self || j > i) && d2[k] < r2) mask |= 1u << k;
    }
    return mask;
}

__global__ void __launch_bounds__(128, 6)
    k_leaf_warp4(const float4* __restrict__ keys, const float4* __restrict__ pos, int32_t nL,
                 float r, float r2, float r2g, unsigned long long* cursor, int64_t cap,
                 int32_t* pi, int32_t* pj, float* pd, int32_t* err) {
    constexpr int APL = 4;
    __shared__ int2 sbij[4][kWarpBuf];
    __shared__ float sbd[4][kWarpBuf];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t q0 = (int32_t)((blockIdx.x * 4 + w) * 32) + 1;
    if (q0 > nL) return;  // whole warp
    int2* bij = sbij[w];
    float* bd = sbd[w];
    const int32_t q = q0 + lane;
    const bool valid = q <= nL;
    Node ql;
    float4 qa[APL];
    if (valid) {
        ql = load_node(keys, q);
        const int64_t A = (int64_t)(q - 1) * APL;
#pragma unroll
        for (int i = 0; i < APL; ++i) qa[i] = __ldg(&pos[A + i]);
    } else {
        ql.mnx = ql.mny = ql.mnz = INFINITY;
        ql.mxx = ql.mxy = ql.mxz = -INFINITY;
        ql.left = ql.skip = 0;
#pragma unroll
        for (int i = 0; i < APL; ++i) qa[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float slack = valid ? leaf_slack(ql) : 0.0f;
    int nb = 0;
    int32_t ia[APL];
#pragma unroll
    for (int i = 0; i < APL; ++i) ia[i] = __float_as_int(qa[i].w);
    {
        // intra-leaf pairs (a before b in the leaf)
        float d2[16];
        unsigned mask = leaf_tests16(qa, qa, true, r2, d2);
        if (!valid) mask = 0;
        warp_emit16(mask, d2, ia, ia, bij, bd, nb, cursor, cap, pi, pj, pd);
    }
    // the warp's union box (invalid lanes contribute the empty box)
    Node un = ql;
    for (int sh = 16; sh > 0; sh >>= 1) {
        un.mnx = fminf(un.mnx, __shfl_xor_sync(0xffffffffu, un.mnx, sh));
        un.mny = fminf(un.mny, __shfl_xor_sync(0xffffffffu, un.mny, sh));
        un.mnz = fminf(un.mnz, __shfl_xor_sync(0xffffffffu, un.mnz, sh));
        un.mxx = fmaxf(un.mxx, __shfl_xor_sync(0xffffffffu, un.mxx, sh));
        un.mxy = fmaxf(un.mxy, __shfl_xor_sync(0xffffffffu, un.mxy, sh));
        un.mxz = fmaxf(un.mxz, __shfl_xor_sync(0xffffffffu, un.mxz, sh));
    }
    int32_t t = __shfl_sync(0xffffffffu, ql.skip, 0);
    int32_t visits = 0;
    const int32_t nnodes = 2 * nL - 1;
    while (t != 0) {
        if (t < 1 || t > nnodes || ++visits > nnodes) {
            if (lane == 0) set_error(err, ND_ERR_INTERNAL, q0);
            break;
        }
        const Node nd_ = load_node(keys, t);
        if (overlap(un, nd_)) {
            if (nd_.left == 0) {
                unsigned mask = 0;
                float d2[16];
                int32_t ib[APL] = {0, 0, 0, 0};
                if (valid && t > q && overlap(ql, nd_) && leaf_gap_ok(ql, nd_, r, r2g, slack)) {
                    const int64_t B = (int64_t)(t - 1) * APL;
                    float4 tb[APL];
#pragma unroll
                    for (int j = 0; j < APL; ++j) tb[j] = __ldg(&pos[B + j]);
                    mask = leaf_tests16(qa, tb, false, r2, d2);
#pragma unroll
                    for (int j = 0; j < APL; ++j) ib[j] = __float_as_int(tb[j].w);
                }
                warp_emit16(mask, d2, ia, ib, bij, bd, nb, cursor, cap, pi, pj, pd);
                t = nd_.skip;
            } else {
                t = nd_.left;
            }
        } else {
            t = nd_.skip;
        }
    }
    warp_buf_flush(bij, bd, nb, cursor, cap, pi, pj, pd);
}

__global__ void __launch_bounds__(128)
    k_atom_count(const float4* __restrict__ keys, const float4* __restrict__ pos, int32_t n,
                 int32_t apl, float r2, int64_t* __restrict__ counts, int32_t* err) {
    int32_t qi = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (qi > n) return;
    SinkCount s;
    if (qi <= n - 1) atom_query(qi, keys, pos, apl, r2, 2 * (n / apl) - 1, err, s);
    counts[qi - 1] = s.n;
}

__global__ void __launch_bounds__(128)
    k_atom_write(const float4* __restrict__ keys, const float4* __restrict__ pos, int32_t n,
                 int32_t apl, float r2, const int64_t* __restrict__ offsets,
                 const int64_t* __restrict__ total, int64_t cap, int32_t* pi, int32_t* pj,
                 float* pd, int32_t* err) {
    int32_t qi = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (qi > n - 1 || *total > cap) return;
    SinkWrite s{pi, pj, pd, offsets[qi - 1]};
    atom_query(qi, keys, pos, apl, r2, 2 * (n / apl) - 1, err, s);
}

// Unordered emission for callers that allow scratch memory.  First the pairs
// (g, h >= g) of groups of 32 leaves whose boxes overlap are listed: one warp
// per group searches the group boxes 32 at a time, super-groups first.  Then
// warps stride over these tasks.  A task tests the leaves of each group
// against the other group's box (one a lane), then takes the survivors of the
// shorter side one at a time against the other side's 32 lanes; leaf pairs
// that overlap and whose atoms can be within r go through a queue in shared
// memory, 32 at a time, one a lane, to the 4 x 4 distance tests, and the hits
// through a buffer in shared memory to the list.  A dense cluster only means
// more tasks, all of one size at most.
// The second kernel is bound by instruction issue and by the list's writes
// (12 bytes a pair).  In the form before, rope walks recorded subtrees, a
// second kernel scanned them leaf by leaf with every query leaf and recorded
// candidate leaf pairs, a third tested those: the walks' tail and the
// candidates' way through memory and the host are gone.  64 clusters in us,
// before and now: 131,072 points 336, 211; 1,048,576 points 1593, 1350;
// 4,194,304 points (2.97e9 pairs, 35.6 GB) 13707, 11490.  A buffer of 256 hits
// a warp (one reservation for 190 instead of 450) takes 14300; writing from a
// ring while its reservation is under way 13900 (more instructions).
constexpr int kTaskBuf = 128;  // tasks buffered per warp

template <bool DEEP>
__global__ void __launch_bounds__(128)
    k_group_tasks(const float4* __restrict__ gbox, int32_t nL, unsigned long long* tcursor,
                  int64_t tcap, int2* __restrict__ tasks) {
    __shared__ int32_t sbuf[4][kTaskBuf];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t g = (int32_t)blockIdx.x * 4 + w;
    if (g >= GroupLevels(nL).ng) return;  // whole warp
    int32_t* buf = sbuf[w];
    const Node un = load_node(gbox, g + 1);
    if (lane == 0) buf[0] = g;  // the pairs inside the group, whatever its box
    int nb = 1;
    auto flush = [&]() {
        __syncwarp();
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(tcursor, (unsigned long long)nb);
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int k = lane; k < nb; k += 32)
            if ((int64_t)(base + k) < tcap) tasks[base + k] = make_int2(g, buf[k]);
        __syncwarp();
        nb = 0;
    };
    wide_groups<DEEP>(un, g + 1, gbox, nL, [&](int32_t base, unsigned m) {
        if ((m >> lane) & 1u) buf[nb + __popc(m & ((1u << lane) - 1u))] = base + lane;
        nb += __popc(m);
        if (nb > kTaskBuf - 32) flush();
    });
    if (nb) flush();
}

constexpr int kPairBuf = 512;  // hits buffered per warp

// A warp's hits on their way to the list.  Squared distances are kept; the
// flush takes their roots with every lane busy.
struct PairBuf {
    int32_t i[kPairBuf], j[kPairBuf];
    float d2[kPairBuf];
};

__device__ __forceinline__ void pair_buf_flush(PairBuf& b, int& nb, unsigned long long* cursor,
                                               int64_t cap, int32_t* pi, int32_t* pj, float* pd) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0 && nb) base = atomicAdd(cursor, (unsigned long long)nb);
    base = __shfl_sync(0xffffffffu, base, 0);
    // entries of the run that fit (32-bit offsets from its first slot)
    const int64_t room = cap - (int64_t)base;
    const int n = room >= nb ? nb : room > 0 ? (int)room : 0;
    int32_t* __restrict__ qi = pi + base;
    int32_t* __restrict__ qj = pj + base;
    float* __restrict__ qd = pd + base;
    int k = lane;
    for (; k + 96 < n; k += 128) {
#pragma unroll
        for (int u = 0; u < 128; u += 32) {
            qi[k + u] = b.i[k + u];
            qj[k + u] = b.j[k + u];
            qd[k + u] = __fsqrt_rn(b.d2[k + u]);
        }
    }
    for (; k < n; k += 32) {
        qi[k] = b.i[k];
        qj[k] = b.j[k];
        qd[k] = __fsqrt_rn(b.d2[k]);
    }
    __syncwarp();
    nb = 0;
}

__global__ void __launch_bounds__(128, 6)
    k_group_pairs(const float4* __restrict__ keys, const float4* __restrict__ gbox,
                  const float4* __restrict__ pos, int32_t nL, float r, float r2, float r2g,
                  const unsigned long long* __restrict__ tcount, int64_t tcap,
                  const int2* __restrict__ tasks, unsigned long long* ticket,
                  unsigned long long* cursor, int64_t cap, int32_t* __restrict__ pi,
                  int32_t* __restrict__ pj, float* __restrict__ pd) {
    __shared__ PairBuf sbuf[4];
    __shared__ float4 sbox[4][2][64];  // leaf boxes of the task's groups, their slack beside
    __shared__ int2 squeue[4][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int64_t ntask = (int64_t)*tcount;
    if (ntask > tcap) return;  // the list of tasks has to grow first
    PairBuf& buf = sbuf[w];
    int2* queue = squeue[w];
    int nb = 0, qn = 0;
    auto put = [&](bool hit, float4 a, float4 b, float d2) {
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (hit) {
            const int at = nb + __popc(m & below);
            buf.i[at] = __float_as_int(a.w);
            buf.j[at] = __float_as_int(b.w);
            buf.d2[at] = d2;
        }
        nb += __popc(m);
    };
    auto room = [&]() {  // for 128 more
        if (nb > kPairBuf - 128) pair_buf_flush(buf, nb, cursor, cap, pi, pj, pd);
    };
    // the 4 x 4 tests of the first nc candidates, one a lane
    auto test = [&](int nc) {
        const int2 e = queue[lane < nc ? lane : 0];
        const float thr = lane < nc ? r2 : -1.0f;  // no squared distance is below -1
        float4 qa[4], tb[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) qa[i] = __ldg(&pos[(int64_t)e.x * 4 + i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) tb[j] = __ldg(&pos[(int64_t)e.y * 4 + j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            room();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float d2 = dist2_ref(qa[i].x, qa[i].y, qa[i].z, tb[j].x, tb[j].y, tb[j].z);
                put(d2 < thr, qa[i], tb[j], d2);
            }
        }
    };
    // this lane's leaf of group g (an empty box past the end) into side s
    auto load_side = [&](int s, int32_t g, Node& b, float& slack) {
        const int32_t l = g * 32 + lane;
        if (l < nL) {
            b = load_node(keys, l + 1);
            slack = leaf_slack(b);
        } else {
            b.mnx = b.mny = b.mnz = INFINITY;
            b.mxx = b.mxy = b.mxz = -INFINITY;
            slack = 0.0f;
        }
        __syncwarp();
        sbox[w][s][2 * lane] = make_float4(b.mnx, b.mny, b.mnz, b.mxx);
        sbox[w][s][2 * lane + 1] = make_float4(b.mxy, b.mxz, slack, 0.0f);
        __syncwarp();
    };
    int32_t g = -1;
    Node un, ql;
    float qslack = 0.0f;
    // Tasks are drawn a few in a row (they mostly share their first group) from
    // a counter, the next draw in flight: the tasks of a dense cluster hold a
    // hundred times those at its rim, and with a fixed share for each warp
    // half of the SM time went by idle.
    const int64_t chunk = min(max(ntask / ((int64_t)gridDim.x * 64), (int64_t)1), (int64_t)4);
    unsigned long long next = 0;
    if (lane == 0) next = atomicAdd(ticket, (unsigned long long)chunk);
    for (;;) {
        const int64_t k0 = (int64_t)__shfl_sync(0xffffffffu, next, 0);
        if (k0 >= ntask) break;
        if (lane == 0) next = atomicAdd(ticket, (unsigned long long)chunk);
        for (int64_t k = k0; k < min(k0 + chunk, ntask); ++k) {
            const int2 tk = __ldg(&tasks[k]);
            const int32_t h = tk.y;
            if (tk.x != g) {
                g = tk.x;
                un = load_node(gbox, g + 1);
                load_side(0, g, ql, qslack);
            }
            const Node uh = load_node(gbox, h + 1);
            Node tl;
            float tslack;
            load_side(1, h, tl, tslack);
            if (h == g) {  // the six pairs inside each leaf
                const bool valid = g * 32 + lane < nL;
                const int64_t A = (int64_t)(valid ? g * 32 + lane : 0) * 4;
                const float thr = valid ? r2 : -1.0f;
                float4 qa[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) qa[i] = __ldg(&pos[A + i]);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    room();
#pragma unroll
                    for (int j = i + 1; j < 4; ++j) {
                        const float d2 =
                            dist2_ref(qa[i].x, qa[i].y, qa[i].z, qa[j].x, qa[j].y, qa[j].z);
                        put(d2 < thr, qa[i], qa[j], d2);
                    }
                }
            }
            const unsigned mq = __ballot_sync(0xffffffffu, overlap(ql, uh));
            const unsigned mt = __ballot_sync(0xffffffffu, overlap(un, tl));
            // the shorter side goes one by one, the other one stays in the lanes
            const bool by_t = __popc(mt) <= __popc(mq);
            const Node own = by_t ? ql : tl;
            const float slack = by_t ? qslack : tslack;
            const bool in = ((by_t ? mq : mt) >> lane) & 1u;
            const float4* other = sbox[w][by_t ? 1 : 0];
            for (unsigned m = by_t ? mt : mq; m; m &= m - 1) {
                const int b = __ffs(m) - 1;
                const float4 b0 = other[2 * b], b1 = other[2 * b + 1];
                Node o;
                o.mnx = b0.x; o.mny = b0.y; o.mnz = b0.z;
                o.mxx = b0.w; o.mxy = b1.x; o.mxz = b1.y;
                const bool after = h > g || (by_t ? b > lane : lane > b);  // t > q
                const bool want = in && after && overlap(own, o) &&
                                  leaf_gap_ok(own, o, r, r2g, fmaxf(slack, b1.z));
                const unsigned c = __ballot_sync(0xffffffffu, want);
                if (!c) continue;
                if (want)
                    queue[qn + __popc(c & below)] =
                        make_int2(g * 32 + (by_t ? lane : b), h * 32 + (by_t ? b : lane));
                qn += __popc(c);
                __syncwarp();
                if (qn >= 32) {
                    test(32);
                    const int2 rest = queue[32 + (lane < qn - 32 ? lane : 0)];
                    __syncwarp();
                    if (lane < qn - 32) queue[lane] = rest;
                    qn -= 32;
                    __syncwarp();
                }
            }
        }
    }
    if (qn) test(qn);
    pair_buf_flush(buf, nb, cursor, cap, pi, pj, pd);
}

// The pair criterion as a threshold on the Float32 squared distance d2:
// ND_CRIT_SQUARED: d2 < r^2 (leafneighbor_traverse, BVHTraverse.jl:1048), the
// threshold fl(r * r); ND_CRIT_SQRT: sqrt(d2) < r (simdneighbor_traverse,
// ext/NaiveSIMD.jl:529,589), the smallest float T with sqrtf(T) >= r -- the
// square root is correctly rounded, hence monotonic, so sqrt(d2) < r exactly
// when d2 < T.  The kernels compare d2 with the threshold either way.
float pair_threshold(float r, int32_t criterion) {
    float t = r * r;
    if (criterion != ND_CRIT_SQRT) return t;
    while (t > 0.0f && std::sqrt(std::nextafter(t, 0.0f)) >= r) t = std::nextafter(t, 0.0f);
    while (std::sqrt(t) < r) t = std::nextafter(t, INFINITY);
    return t;
}

nd_status emit_unordered(Ctx* c, const TreeBuffers& t, float r, float r2, int32_t* pi,
                         int32_t* pj, float* pd, int64_t capacity, int64_t* total) {
    if (t.apl != 4) return ND_ERR_ARG;
    nd_status st;
    if ((st = ensure(c, c->misc, 64))) return st;
    unsigned long long* cursor = (unsigned long long*)c->misc.p;
    cudaError_t e;
    if (c->no_alloc) {
        // no scratch for candidate pairs: the one-pass walk
        cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), c->stream);
        k_leaf_warp4<<<(unsigned)cdiv(t.nL, 128), 128, 0, c->stream>>>(
            t.keys, t.pos4, t.nL, r, r2, gap_limit(r, r2), cursor, capacity, pi, pj, pd, c->d_err);
        c->launches++;
        if ((st = check_launch(c, "leaf pairs (unordered)"))) return st;
        unsigned long long tot = 0;
        e = cudaMemcpyAsync(&tot, cursor, sizeof(tot), cudaMemcpyDeviceToHost, c->stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "pair count");
        if ((st = sync_and_check(c, "leaf pairs (unordered)"))) return st;
        *total = (int64_t)tot;
        return ND_OK;
    }
    // run again with a longer task list while it overflowed
    unsigned long long* tcursor = cursor + 1;
    unsigned long long* ticket = cursor + 2;
    int nsm = 0, occ = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_group_pairs, 128, 0);
    const GroupLevels lev(t.nL);
    const int64_t ng = lev.ng;
    if ((st = ensure(c, c->store, 32 * (size_t)lev.boxes()))) return st;
    if ((st = ensure(c, c->tasks, sizeof(int2) * 128 * (size_t)ng))) return st;
    float4* gbox = (float4*)c->store.p;
    group_boxes(c, t.keys, t.nL, gbox, lev.ns > kDirectSupers);
    for (int attempt = 0;; ++attempt) {
        const int64_t tcap = (int64_t)(c->tasks.bytes / sizeof(int2));
        cudaMemsetAsync(cursor, 0, 3 * sizeof(unsigned long long), c->stream);
        const auto tasks_fn = lev.ns <= kDirectSupers ? k_group_tasks<false> : k_group_tasks<true>;
        tasks_fn<<<(unsigned)cdiv(ng, 4), 128, 0, c->stream>>>(gbox, t.nL, tcursor, tcap,
                                                               (int2*)c->tasks.p);
        k_group_pairs<<<(unsigned)(nsm * std::max(occ, 1)), 128, 0, c->stream>>>(
            t.keys, gbox, t.pos4, t.nL, r, r2, gap_limit(r, r2), tcursor, tcap,
            (const int2*)c->tasks.p, ticket, cursor, capacity, pi, pj, pd);
        c->launches += 2;
        if ((st = check_launch(c, "leaf pairs (unordered)"))) return st;
        unsigned long long h[2] = {0, 0};
        e = cudaMemcpyAsync(h, cursor, sizeof(h), cudaMemcpyDeviceToHost, c->stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "pair count");
        if ((st = sync_and_check(c, "leaf pairs (unordered)"))) return st;
        *total = (int64_t)h[0];
        if ((int64_t)h[1] <= tcap) return ND_OK;
        if (attempt == 2) {
            c->last_error = "overlapping leaf groups: buffer kept overflowing";
            return ND_ERR_INTERNAL;
        }
        if ((st = ensure(c, c->tasks, sizeof(int2) * (size_t)h[1]))) return st;
    }
}

// k_leaf_wide and k_leaf_walk for a tree's leaf width.
template <int WRITE>
static auto leaf_wide(const TreeBuffers& t, bool deep) {
    if (t.apl == 4) return deep ? k_leaf_wide<4, WRITE, true> : k_leaf_wide<4, WRITE, false>;
    if (t.apl == 2) return deep ? k_leaf_wide<2, WRITE, true> : k_leaf_wide<2, WRITE, false>;
    return deep ? k_leaf_wide<0, WRITE, true> : k_leaf_wide<0, WRITE, false>;
}
template <int WRITE>
static auto leaf_walk(const TreeBuffers& t) {
    return t.apl == 4 ? k_leaf_walk<4, WRITE> : t.apl == 2 ? k_leaf_walk<2, WRITE> : k_leaf_walk<0, WRITE>;
}

// The ordered list's group boxes: in place of the build's CAS slots, which it has
// no use for, or behind them where it may still build the tree.
static size_t group_box_at(int32_t nL) {
    return nL > kWalkLeaves ? (sizeof(int32_t) * (size_t)nL + 255) / 256 * 256 : 0;
}

// One pass (WRITE as in k_leaf_wide) over all query leaves.
template <int WRITE>
static void leaf_pass(Ctx* c, const TreeBuffers& t, float r, float r2, int64_t* counts,
                      const int64_t* offsets, const int64_t* total, int64_t cap, int32_t* pi,
                      int32_t* pj, float* pd) {
    const float4* gbox = (const float4*)((const char*)c->store.p + group_box_at(t.nL));
    if (t.walk) {
        leaf_walk<WRITE>(t)<<<(unsigned)cdiv(t.nL, 128), 128, 0, c->stream>>>(
            t.keys, t.pos4, t.nL, t.apl, r, r2, t.widest, counts, offsets, total, cap, pi, pj, pd,
            c->d_err);
        c->launches++;
        if (t.nwide == 0) return;
    }
    const int32_t nq = t.walk ? t.nwide : t.nL;
    const bool deep = t.walk || GroupLevels(t.nL).ns > kDirectSupers;
    leaf_wide<WRITE>(t, deep)<<<(unsigned)cdiv(nq, 4), 128, 0, c->stream>>>(
        t.keys, gbox, t.pos4, t.nL, t.apl, r, r2, gap_limit(r, r2), counts, offsets, total, cap, pi, pj,
        pd, t.walk ? (const int32_t*)c->tasks.p : nullptr, nq);
    c->launches++;
}

// Above kWalkLeaves leaves, where the search is bound by its warps' chains of
// loads, a sample of query leaves says how many leaves overlap one (behind it),
// and the walk is taken when the tests that makes are few: overlaps * width^2
// below 80 at 262,144 leaves on the mean, in proportion to the leaves up to 160,
// and below 1024 for every sampled leaf, as the longest walk sets the end (three
// atoms a leaf fill a third of the search's lanes: two and a half times these).
// The list of points at density 0.83, us, search and walk (overlaps): leaves of
// four, 1,048,576 points r 0.4 705 and 542 (2.5), r 0.7 747 and 703 (5.5), r 1.3
// 807 and 1005 (13); 4,194,304 points r 0.4 2453 and 1424, r 1.0 2749 and 2396 (9),
// r 1.7 3051 and 3735 (17); leaves of two, 2,097,152 points r 0.4 1690 and 815
// (1.0), r 1.7 2302 and 1946 (18), r 2.2 2536 and 2584 (32); leaves of eight,
// 4,194,304 points r 0.05 1296 and 1269 (1.0), r 0.4 2008 and 3212 (4.4).  64
// clusters of 32,768 points in all 2,097,152, leaves of four, r 0.2: 1471 and 4992
// (3.1, the most 88).  131,072 leaves: 342 and 296 at r 0.05, about what the sample
// takes.
static bool sparse_leaves(const LeafSample& h, const TreeBuffers& t) {
    const double tests = (double)t.apl * t.apl / (t.apl == 3 ? 2.5 : 1.0);
    return tests * h.overlaps / kSampled < std::min(160.0, 80.0 * t.nL / 262144) &&
           tests * h.most < 1024.0;
}

// Leaves that extend eight times as far as the mean leaf are left to the search
// (evenly spread points have none: the widest of 16.8 million is 5.5 times the
// mean), up to one leaf in 32.
constexpr double kWidest = 8.0;

// Whether the ordered list of t comes from rope walks (t.walk), and their tree.
static nd_status choose_walk(Ctx* c, TreeBuffers& t, float r, const float4* gbox) {
    if (t.nL <= kWalkLeaves || c->no_alloc) return ND_OK;
    nd_status st = ensure(c, c->misc, 64);
    if (st) return st;
    LeafSample* ds = (LeafSample*)c->misc.p;
    LeafSample h{};
    auto read = [&](void* dst, size_t bytes) {
        cudaError_t e = cudaMemcpyAsync(dst, c->misc.p, bytes, cudaMemcpyDeviceToHost, c->stream);
        return e == cudaSuccess ? cudaStreamSynchronize(c->stream) : e;
    };
    cudaMemsetAsync(ds, 0, sizeof(h), c->stream);
    const bool deep = GroupLevels(t.nL).ns > kDirectSupers;
    (deep ? k_overlap_sample<true> : k_overlap_sample<false>)<<<kSampled / 4, 128, 0, c->stream>>>(
        t.keys, gbox, t.nL, ds);
    k_leaf_extents<<<152 * 4, 256, 0, c->stream>>>(t.keys, t.nL, r, ds);
    c->launches += 2;
    cudaError_t e = read(&h, sizeof(h));
    if (e != cudaSuccess) return cuda_fail(c, e, "leaf sample");
    if (!sparse_leaves(h, t)) return ND_OK;
    t.widest = (float)(kWidest * h.extents / t.nL);
    t.nwide = 0;
    if (h.widest > t.widest) {
        const int32_t cap = t.nL / 32;
        if ((st = ensure(c, c->tasks, sizeof(int32_t) * (size_t)cap))) return st;
        unsigned long long n = 0;
        cudaMemsetAsync(ds, 0, sizeof(n), c->stream);
        k_wide_leaves<<<(unsigned)cdiv(t.nL, 256), 256, 0, c->stream>>>(
            t.keys, t.nL, r, t.widest, cap, (int32_t*)c->tasks.p, (unsigned long long*)ds);
        c->launches++;
        if ((e = read(&n, sizeof(n))) != cudaSuccess) return cuda_fail(c, e, "wide leaves");
        if (n > (unsigned long long)cap) return ND_OK;
        t.nwide = (int32_t)n;
    }
    t.walk = true;
    if (t.internal) return ND_OK;
    t.internal = true;
    return build_internal_nodes(c, t.keys, (int32_t*)c->store.p, t.codes, t.nL, t.apl);
}

// Ordered emission: per-query counts, their scan, then the pairs at their
// places.  total_dev receives the number of pairs (device); the write pass
// reads it and writes nothing when it exceeds the capacity, so no host round
// trip lies between the two passes.
nd_status count_pairs(Ctx* c, TreeBuffers& t, float r, float r2, int kind, int64_t* total_dev) {
    nd_status st;
    int64_t nq = (kind == 0) ? t.nL : t.n;
    if ((st = ensure(c, c->counts, sizeof(int64_t) * (size_t)(nq + 1)))) return st;
    if ((st = ensure(c, c->offsets, sizeof(int64_t) * (size_t)(nq + 2)))) return st;
    int64_t* counts = (int64_t*)c->counts.p;
    int64_t* offsets = (int64_t*)c->offsets.p;
    if (kind == 0) {
        const size_t at = group_box_at(t.nL);
        if ((st = ensure(c, c->store, at + 32 * (size_t)GroupLevels(t.nL).boxes()))) return st;
        float4* gbox = (float4*)((char*)c->store.p + at);
        group_boxes(c, t.keys, t.nL, gbox, t.nL > kWalkLeaves);
        if ((st = choose_walk(c, t, r, gbox))) return st;
        leaf_pass<0>(c, t, r, r2, counts, nullptr, nullptr, 0, nullptr, nullptr, nullptr);
    } else {
        k_atom_count<<<(unsigned)cdiv(nq, 128), 128, 0, c->stream>>>(t.keys, t.pos4, t.n, t.apl, r2,
                                                                     counts, c->d_err);
        c->launches++;
    }
    if ((st = check_launch(c, "pair count"))) return st;
    return scan_exclusive(c, counts, offsets, nq, total_dev);
}

nd_status write_pairs(Ctx* c, const TreeBuffers& t, float r, float r2, int kind,
                      const int64_t* total_dev, int64_t cap, int32_t* pi, int32_t* pj, float* pd) {
    const int64_t* offsets = (const int64_t*)c->offsets.p;
    if (kind == 0) {
        leaf_pass<1>(c, t, r, r2, nullptr, offsets, total_dev, cap, pi, pj, pd);
    } else {
        k_atom_write<<<(unsigned)cdiv(t.n, 128), 128, 0, c->stream>>>(
            t.keys, t.pos4, t.n, t.apl, r2, offsets, total_dev, cap, pi, pj, pd, c->d_err);
        c->launches++;
    }
    return check_launch(c, "pair write");
}

// The list as its caller keeps it.  Three arrays had to be put together entry by
// entry on the host, and a length not known beforehand cost a second call with
// a second tree: 2.36 of 2.99 ms for 20,000 atoms (now 0.63 with the copies).
nd_status write_pair_triples(Ctx* c, const TreeBuffers& t, float r, float r2,
                             const int64_t* total_dev, int64_t cap, int32_t* out) {
    leaf_pass<2>(c, t, r, r2, nullptr, (const int64_t*)c->offsets.p, total_dev, cap, out, nullptr,
                 nullptr);
    return check_launch(c, "pair write");
}

__global__ void k_unpack_positions(const float4* __restrict__ pos4, int32_t n,
                                   float* __restrict__ out) {
    const int64_t m = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (m < 3 * (int64_t)n) out[m] = reinterpret_cast<const float*>(pos4)[4 * (m / 3) + m % 3];
}

void unpack_positions(Ctx* c, const float4* pos4, int32_t n, float* out) {
    k_unpack_positions<<<(unsigned)cdiv(3 * (int64_t)n, 256), 256, 0, c->stream>>>(pos4, n, out);
    c->launches++;
}

// ================================================================ pair hash

__global__ void k_pair_hash(const int32_t* __restrict__ pi, const int32_t* __restrict__ pj,
                            const float* __restrict__ pd, int64_t np,
                            unsigned long long* out) {
    uint64_t h0 = 0, h1 = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < np;
         k += (int64_t)gridDim.x * blockDim.x)
        pair_hash_one(pi[k], pj[k], pd[k], h0, h1);
    for (int s = 16; s > 0; s >>= 1) {
        h0 += __shfl_xor_sync(0xffffffffu, h0, s);
        h1 += __shfl_xor_sync(0xffffffffu, h1, s);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&out[0], (unsigned long long)h0);
        atomicAdd(&out[1], (unsigned long long)h1);
    }
}

nd_status pair_hash(Ctx* c, const int32_t* pi, const int32_t* pj, const float* pd, int64_t np,
                    uint64_t out[2]) {
    nd_status st = ensure(c, c->hash, 16);
    if (st) return st;
    cudaMemsetAsync(c->hash.p, 0, 16, c->stream);
    if (np > 0) {
        int blocks = (int)std::min<int64_t>(cdiv(np, 256), 152 * 16);
        k_pair_hash<<<blocks, 256, 0, c->stream>>>(pi, pj, pd, np, (unsigned long long*)c->hash.p);
        c->launches++;
    }
    cudaError_t e = cudaMemcpyAsync(out, c->hash.p, 16, cudaMemcpyDeviceToHost, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "hash copy");
    return sync_and_check(c, "pair hash");
}

}  // namespace nd
