// Bug-compatible forms of the reference's force calls (src/Forces.jl), for
// scripts written against their actual results rather than the intended
// physics that the engine computes:
//
//   force_lennardjones!(force, pairslist, position)   Forces.jl:6-45
//     force zeroed; for each pair (i, j, d) in list order
//       force[i] .+= (24 eps / d) * ((2 sigma / d)^12 - (sigma / d)^6)
//     with eps = -1f10 (Float32) and sigma = 0.0001 (Float64) hard-coded, the
//     scalar added to all three components, nothing added to force[j];
//   force_coulomb!(force, pairslist, charge)           Forces.jl:46-66
//     force zeroed; for each pair in list order
//       force[i] .+= k q_i q_j / d^2  (k = 1);  force[j] .-= force[i]
//     -- the running total of force[i], an order-dependent recurrence.
//
// Precision follows Julia's promotion rules: Float32 pair distance and
// charges, 24 eps / d in Float32, the powers of sigma / d in Float64 (sigma is
// a Float64 literal), their product with the Float32 factor in Float64, added
// to the Float32 accumulator in Float64 and rounded back to Float32.  Julia's
// x^n for Float64 x and integer-valued exponent is the compensated power by
// squaring of Base.Math (pow_body), restated in jl_pow_int.
//
//   simulate!(sys, spec, clct)                         Simulator.jl:154-256
//     over the all-pairs list, Float32 state, integer stepwidth (compat_simulate).
//
// LJ: each atom's additions are independent of other atoms' -- the pairs are
// sorted by i (stable, so each atom keeps its list order) and one thread per
// atom adds its run.  Coulomb: every update reads the result of earlier ones
// through force[i] and force[j]; for an arbitrary list the recurrence runs on
// one thread in list order, for the all-pairs order of unique_pairs its columns
// flow through bands of rows (compat_simulate).
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "nd_bands.cuh"
#include "nd_internal.cuh"

namespace nd {

namespace {

// Julia's Base.Math.pow_body(x::Float64, n::Integer) for n >= 4: power by
// squaring with the low parts of each product kept (two_mul) and folded in
// with fused multiply-adds (Julia's muladd, fused on the hosts the reference
// targets).  Every other operation is rounded on its own (__d*_rn: nothing is
// contracted).
__device__ inline double jl_pow_int(double x, int n) {
    double y = 1.0, xnlo = 0.0, ynlo = 0.0;
    while (n > 1) {
        if (n & 1) {
            const double err = fma(y, xnlo, __dmul_rn(x, ynlo));
            const double yy = __dmul_rn(x, y);
            ynlo = __dadd_rn(fma(x, y, -yy), err);
            y = yy;
        }
        const double err = __dmul_rn(__dmul_rn(x, 2.0), xnlo);
        const double xx = __dmul_rn(x, x);
        xnlo = __dadd_rn(fma(x, x, -xx), err);
        x = xx;
        n >>= 1;
    }
    const double err = fma(y, xnlo, __dmul_rn(x, ynlo));
    return (isfinite(x) && isfinite(err)) ? fma(x, y, err) : __dmul_rn(x, y);
}

// lennardjones_interior (Forces.jl:6-13) for one pair distance d: the value
// added to each component of force[i].
__device__ inline double lj_compat_term(float d) {
    const float eps = -1e10f;
    const double sigma = 0.0001;
    const float a = __fdiv_rn(__fmul_rn(24.0f, eps), d);  // 24 * eps: Int times Float32
    const double b = jl_pow_int(__ddiv_rn(__dmul_rn(2.0, sigma), (double)d), 12);
    const double c = jl_pow_int(__ddiv_rn(sigma, (double)d), 6);
    return __dmul_rn((double)a, __dsub_rn(b, c));
}

__global__ void k_compat_runs(const uint32_t* __restrict__ key, int64_t np, int32_t* start,
                              int32_t* end) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    const uint32_t k = key[p];  // 1-based atom index
    if (p == 0 || key[p - 1] != k) start[k - 1] = (int32_t)p;
    if (p == np - 1 || key[p + 1] != k) end[k - 1] = (int32_t)p + 1;
}

__global__ void k_compat_lj(const int32_t* __restrict__ order, const float* __restrict__ pd,
                            const int32_t* __restrict__ start, const int32_t* __restrict__ end,
                            int32_t n, float* __restrict__ force) {
    const int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    float f = 0.0f;
    for (int32_t p = start[a]; p < end[a]; ++p)
        f = (float)__dadd_rn((double)f, lj_compat_term(__ldg(&pd[__ldg(&order[p])])));
    force[3 * (int64_t)a] = f;
    force[3 * (int64_t)a + 1] = f;
    force[3 * (int64_t)a + 2] = f;
}

__global__ void k_compat_coulomb(const int32_t* __restrict__ pi, const int32_t* __restrict__ pj,
                                 const float* __restrict__ pd, int64_t np,
                                 const float* __restrict__ q, float* F, int32_t n,
                                 int32_t* err) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int64_t p = 0; p < np; ++p) {
        const int32_t i = pi[p] - 1, j = pj[p] - 1;
        if (i < 0 || i >= n || j < 0 || j >= n) { set_error(err, ND_ERR_ARG, (int32_t)p); return; }
        const float d = pd[p];
        // k * charge[i] * charge[j] ./ (d .^ 2), k = 1
        F[i] = __fadd_rn(F[i], __fdiv_rn(__fmul_rn(q[i], q[j]), __fmul_rn(d, d)));
        F[j] = __fsub_rn(F[j], F[i]);
    }
}

__global__ void k_compat_spread(const float* __restrict__ F, int32_t n, float* __restrict__ force) {
    const int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= n) return;
    const float f = F[a];
    force[3 * (int64_t)a] = f;
    force[3 * (int64_t)a + 1] = f;
    force[3 * (int64_t)a + 2] = f;
}

__global__ void k_iota(int32_t* v, int64_t n) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) v[p] = (int32_t)p;
}

// ------------------------------------------------ simulate! as written
// The all-pairs list of unique_pairs (AllToAll.jl:65-80) holds (i, j) for
// i < j, row by row (row i: j = i + 1 .. n - 1, 0-based).  Nothing of it is
// stored in that order: the Lennard-Jones terms are used as they are computed,
// the Coulomb terms lie in the order the recurrence reads them.

// force_lennardjones! over the whole list and over threshold_pairs(list,
// 0.01): atom i's terms are its row, added in order to Float32 accumulators,
// each addition through Float64 as Julia's promotion does: fa <- Float32(
// Float64(fa) + t).  The terms follow from the pair distances of
// update_pairslist! (AllToAll.jl:7-62): d = sqrt(sum((a[i] .- a[j]).^2)), the
// sum left to right.
//
// GB300 has few Float64 units (a term takes about 60 Float64 operations, an
// addition three on a dependent chain: the term and sum kernels before took
// 1,060 and 1,085 us at 4,096 atoms), so both run on Float32 pairs with a
// bound on their error, and whatever the bound cannot decide is done again in
// Float64 as written:
//  * a term t = a c (4096 c - 1), c = (sigma / d)^6, a = Float32(24 eps / d)
//    (the 12th power is 4096 c^2), as th + tl with a relative error below
//    2^-41 against the Float64 value (the largest of 220,000 distances in each
//    binade) for distances in [2^-10, 2^9]; outside, th = NaN;
//  * an addition: s = fa + th and its error e (TwoSum); the sum lies within
//    err = 2^-38 |th| + 2^-44 |s| + 1e-42 of s + (e + tl), which covers the
//    term's error, the roundings here and the rounding to Float64.  Rounding
//    to Float64 and then Float32 is monotonic, so when s + (r - err) and s +
//    (r + err) round to the same Float32 that is the result; when not (about
//    one addition in 10^5, and terms out of the range above) that addition is
//    done in Float64.
// A block serves 32 atoms: eight warps compute the terms of 64 columns at a
// time into shared memory (a lane per atom, a column at a time), one warp adds
// them up, a lane per atom; the chain of additions bounds it.
constexpr int kLjCols = 64;  // columns per buffer: eight per producing warp

__device__ __forceinline__ float compat_dist(const float3& a, const float* __restrict__ x,
                                             int32_t j) {
    const float dx = __fsub_rn(a.x, __ldg(&x[3 * (int64_t)j]));
    const float dy = __fsub_rn(a.y, __ldg(&x[3 * (int64_t)j + 1]));
    const float dz = __fsub_rn(a.z, __ldg(&x[3 * (int64_t)j + 2]));
    return __fsqrt_rn(
        __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
}

// (h, l) <- (ah, al) (bh, bl) as Float32 pairs.
__device__ __forceinline__ void pair_mul(float ah, float al, float bh, float bl, float& h,
                                         float& l) {
    h = __fmul_rn(ah, bh);
    l = __fadd_rn(__fmaf_rn(ah, bh, -h), __fmaf_rn(ah, bl, __fmul_rn(al, bh)));
}

// lj_compat_term(d) as th + tl.
__device__ __forceinline__ float2 lj_pair_term(float d) {
    if (!(d >= 0x1p-10f && d <= 0x1p9f)) return make_float2(__int_as_float(0x7fffffff), 0.0f);
    const double s6 = 0.0001 * 0.0001 * 0.0001 * 0.0001 * 0.0001 * 0.0001;
    const float s6h = (float)s6, s6l = (float)(s6 - (double)s6h);
    const float a = __fdiv_rn(__fmul_rn(24.0f, -1e10f), d);
    const float ih = __frcp_rn(d);  // 1 / d = ih + il
    const float il = __fmul_rn(ih, __fmaf_rn(-d, ih, 1.0f));
    float zh, zl, wh, wl, vh, vl, ch, cl, uh, ul, ph, pl, th, tl;
    pair_mul(ih, il, ih, il, zh, zl);
    pair_mul(zh, zl, zh, zl, wh, wl);
    pair_mul(wh, wl, zh, zl, vh, vl);    // d^-6
    pair_mul(vh, vl, s6h, s6l, ch, cl);  // (sigma / d)^6
    const float gh = __fmaf_rn(4096.0f, ch, -1.0f);
    const float gl = __fmaf_rn(4096.0f, cl, __fmaf_rn(4096.0f, ch, -__fadd_rn(gh, 1.0f)));
    pair_mul(a, 0.0f, s6h, s6l, uh, ul);
    pair_mul(uh, ul, vh, vl, ph, pl);
    pair_mul(ph, pl, gh, gl, th, tl);
    return make_float2(th, tl);
}

__global__ void __launch_bounds__(288) k_cs_lj(const float* __restrict__ x, int32_t n, float thr,
                                               float* __restrict__ ljthr,
                                               float* __restrict__ ljall) {
    __shared__ float2 st[2][kLjCols][32];
    __shared__ unsigned char snear[2][32][8];  // bit m of [row][w]: column 8 w + m is near
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int32_t i0 = (int32_t)blockIdx.x * 32, i = i0 + lane;
    float3 p = make_float3(0.f, 0.f, 0.f);
    if (i < n)
        p = make_float3(x[3 * (int64_t)i], x[3 * (int64_t)i + 1], x[3 * (int64_t)i + 2]);
    const int32_t jb = i0 + 1;  // the first column of any row of the block
    const int32_t nchunk = (n - jb + kLjCols - 1) / kLjCols;
    float fa = 0.0f, ft = 0.0f;
    auto produce = [&](int32_t c) {
        const int32_t j0 = jb + c * kLjCols + 8 * w;
        unsigned near = 0;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int32_t j = j0 + m;
            if (j < n) {
                const float d = compat_dist(p, x, j);
                st[c & 1][8 * w + m][lane] = lj_pair_term(d);
                if (d < thr && j > i) near |= 1u << m;
            }
        }
        snear[c & 1][lane][w] = (unsigned char)near;
    };
    // fa + t through Float64, decided in Float32: false when it cannot be
    auto add = [](float& f, const float2& t) -> bool {
        const float s = __fadd_rn(f, t.x);
        const float b = __fsub_rn(s, f);
        const float e = __fadd_rn(__fsub_rn(f, __fsub_rn(s, b)), __fsub_rn(t.x, b));
        const float r = __fadd_rn(e, t.y);
        const float err = __fmaf_rn(fabsf(t.x), 0x1p-38f, __fmaf_rn(fabsf(s), 0x1p-44f, 1e-42f));
        const float up = __fadd_rn(s, __fadd_rn(r, err));
        const bool sure = up == __fadd_rn(s, __fsub_rn(r, err));
        f = up;
        return sure;
    };
    auto consume = [&](int32_t c) {
        if (i0 >= n) return;
        for (int g = 0; g < 8; ++g) {
            const int32_t j0 = jb + c * kLjCols + 8 * g;
            if (j0 >= n) break;
            const float f0 = fa;
            bool good = j0 > i0 + 31 && j0 + 7 < n;  // every column belongs to every row
            if (good) {
#pragma unroll
                for (int m = 0; m < 8; ++m) {
                    const bool sure = add(fa, st[c & 1][8 * g + m][lane]);
                    good = good && sure;
                }
            }
            // a NaN stays one (and an infinity, whatever finite term is added)
            if (!good && i < n && f0 == f0) {
                fa = f0;
                for (int m = 0; m < 8; ++m) {
                    const int32_t j = j0 + m;
                    if (j <= i || j >= n || fa != fa) continue;
                    const float2 t = st[c & 1][8 * g + m][lane];
                    float f = fa;
                    if (add(f, t))
                        fa = f;
                    else if (!(isinf(fa) && isfinite(t.x)))
                        fa = __double2float_rn(
                            __dadd_rn((double)fa, lj_compat_term(compat_dist(p, x, j))));
                }
            }
            unsigned near = snear[c & 1][lane][g];
            while (near) {
                const int32_t j = j0 + __ffs(near) - 1;
                near &= near - 1;
                ft = __double2float_rn(
                    __dadd_rn((double)ft, lj_compat_term(compat_dist(p, x, j))));
            }
        }
    };
    if (w < 8 && nchunk > 0) produce(0);
    __syncthreads();
    for (int32_t c = 0; c < nchunk; ++c) {
        if (w == 8) consume(c);
        else if (c + 1 < nchunk) produce(c + 1);
        __syncthreads();
    }
    if (w == 8 && i < n) {
        ljthr[i] = ft;
        ljall[i] = fa;
    }
}

// force_coulomb! over the all-pairs list.  Pair (i, j) depends on the pairs
// before it that touch i or j: in this list order those are (i, j - 1) (or
// (i - 1, i)) and (i - 1, j).  Any schedule that keeps the two orders (along
// a row, and down a column) and runs each pair's two updates as written gives
// every atom the same sequence of roundings as the sequential loop.
//
// Bands (kLevelAtoms < n <= kBandMaxAtoms): a warp owns 256 consecutive rows, eight a
// lane, whose running forces stay in registers; the columns flow through its
// lanes, four at a time.  At step t lane l takes the four columns 256 b + 4 (t -
// l) .. + 3 from lane l - 1 by shuffles, adds the pair terms to its rows' forces
// and subtracts those from the columns'; a row starts from its own column's
// value when that arrives (j == i).  Columns pass from a band to the next
// through an array in shared memory, each value with the number of bands it
// has passed in the same 64-bit word (so no fence is needed); bands are spread
// over a cluster of up to eight blocks, the last band of a block writing into
// the next block's array.  The time is the dependence's: 95 steps a band, a step
// of about 180 ns (64 dependent-in-pairs additions, shuffles, 4 KB of terms)
// wherever the band lies.  4,096 atoms: 2,882 us a force evaluation with one
// block running the anti-diagonals i + j behind a barrier each (the form
// before), about 360 us so; one column and four rows a lane and step 460 us.
//
// The pair terms k q_i q_j / d^2 do not depend on the recurrence: they are
// computed beforehand in the order the lanes read them, 4 KB a step.  Where a
// lane has no pair the term is -0, which adds nothing to any value (signed
// zeros included).
__device__ __forceinline__ float coulomb_term(float xi, float yi, float zi, float qi, float xj,
                                              float yj, float zj, float qj) {
    const float dx = __fsub_rn(xi, xj), dy = __fsub_rn(yi, yj), dz = __fsub_rn(zi, zj);
    const float d = __fsqrt_rn(
        __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
    // k * charge[i] * charge[j] ./ (d .^ 2), k = 1
    return __fdiv_rn(__fmul_rn(qi, qj), __fmul_rn(d, d));
}

__global__ void __launch_bounds__(256)
    k_cs_band_terms(const float* __restrict__ x, const float* __restrict__ q, int32_t n, int32_t P,
                    float4* __restrict__ cterm) {
    const int32_t b = blockIdx.y, lane = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int32_t t = (int32_t)blockIdx.x;
    if (t >= P - 64 * b) return;
    const int32_t i = band_row(b, lane, r), j0 = band_col(b, lane, t);
    float c[4] = {-0.0f, -0.0f, -0.0f, -0.0f};
    if (band_tile_has_pair(i, j0, n)) {
        const float xi = __ldg(&x[3 * (int64_t)i]), yi = __ldg(&x[3 * (int64_t)i + 1]),
                    zi = __ldg(&x[3 * (int64_t)i + 2]), qi = __ldg(&q[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int32_t j = j0 + k;
            if (j > i && j < n)
                c[k] = coulomb_term(xi, yi, zi, qi, __ldg(&x[3 * (int64_t)j]),
                                    __ldg(&x[3 * (int64_t)j + 1]), __ldg(&x[3 * (int64_t)j + 2]),
                                    __ldg(&q[j]));
        }
    }
    cterm[(band_off(b, P) + t) * 256 + threadIdx.x] = make_float4(c[0], c[1], c[2], c[3]);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* m) {
    asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(m)) : "memory");
}
// One bulk copy of `bytes` contiguous bytes (16-byte aligned on both sides),
// completing on mbarrier m.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes,
                                          unsigned long long* m) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(m)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(m))
        : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long* m, unsigned phase) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_addr(m)), "r"(phase)
        : "memory");
    return ok != 0;
}

// One cluster of blocks; warp w of block k runs band k * warps + w.  RING: the
// terms come through a ring of 2^ldepth copies of kBandCopy steps a warp in
// shared memory, filled by bulk copies that far ahead (registers cannot hold
// enough loads to cover their latency); otherwise (more warps than rings fit
// beside the columns) straight into registers, a step ahead.
template <bool RING, int THREADS>
__global__ void __launch_bounds__(THREADS, 1)
    k_cs_coulomb_bands(const float4* __restrict__ cterm, int32_t n, int32_t P, int32_t ldepth,
                       float* __restrict__ F, int32_t* err) {
    // columns (bands passed << 32 | value, column j at j + kBandPad), the
    // rings, their barriers
    extern __shared__ __align__(128) unsigned char sband[];
    unsigned long long* scol = reinterpret_cast<unsigned long long*>(sband);
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int32_t b = (int32_t)rank * W + w;
    const int32_t ncol = band_col_bytes(n) / 8, depth = 1 << ldepth;
    constexpr int CP = kBandCopy;
    float4* ring = reinterpret_cast<float4*>(sband + 8 * ncol) + (w << ldepth) * CP * 256;
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(
                                  sband + 8 * ncol + ((int64_t)W << ldepth) * CP * 4096) +
                              (w << ldepth);
    for (int32_t k = threadIdx.x; k < ncol; k += blockDim.x) scol[k] = 0ull;
    if (RING && lane == 0) {
        for (int32_t k = 0; k < depth; ++k) mbar_init(bar + k);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster.sync();
    const int32_t row0 = kBandRows * b;
    if (row0 < n) {
        constexpr int32_t kPolls = 1 << 22;  // a tenth of a second or more: never in a sound run
        unsigned long long* out = scol;
        if (w == W - 1 && rank + 1 < cluster.num_blocks())
            out = cluster.map_shared_rank(scol, rank + 1);
        const int32_t T = P - 64 * b, ncp = T / CP;  // P is a multiple of CP
        const float4* __restrict__ C = cterm + band_off(b, P) * 256;
        float a[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) a[r] = 0.0f;
        bool lost = false;
        float4 buf[2][8];
        auto issue = [&](int32_t c) {
            bulk_load(ring + (c & (depth - 1)) * CP * 256, C + (int64_t)c * CP * 256, CP * 4096,
                      bar + (c & (depth - 1)));
        };
        if (RING && lane == 0)
            for (int32_t c = 0; c < min(depth, ncp); ++c) issue(c);
        const float4* src = ring + lane;
        auto load = [&](float4 (&dst)[8], int32_t t) {
            if (t >= T) return;
            if constexpr (RING) {
                if ((t & (CP - 1)) == 0) {
                    const int32_t c = t / CP, slot = c & (depth - 1);
                    for (int32_t polls = 0; !mbar_try(bar + slot, (unsigned)(c >> ldepth) & 1u); ++polls)
                        if (polls > kPolls) {
                            lost = true;
                            if (lane == 0) set_error(err, ND_ERR_INTERNAL, b);
                            break;
                        }
                    src = ring + slot * CP * 256 + lane;
                    __syncwarp();
                    // every lane has read the copy before: its slot takes a later one
                    if (lane == 0 && c > 0 && c - 1 + depth < ncp) issue(c - 1 + depth);
                }
#pragma unroll
                for (int r = 0; r < 8; ++r) dst[r] = src[r * 32];
                src += 256;
            } else {
#pragma unroll
                for (int r = 0; r < 8; ++r) dst[r] = __ldg(&C[(int64_t)t * 256 + r * 32 + lane]);
            }
        };
        // columns row0 + 4 t .. + 3 and the bands they have passed (every lane
        // reads the same words)
        unsigned long long in[4] = {0, 0, 0, 0};
        auto peek = [&](int32_t t) {
            const unsigned at = smem_addr(scol + row0 + 4 * t + kBandPad);
            asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                         : "=l"(in[0]), "=l"(in[1])
                         : "r"(at)
                         : "memory");
            asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                         : "=l"(in[2]), "=l"(in[3])
                         : "r"(at + 16)
                         : "memory");
        };
        auto missing = [&]() {
            const unsigned g = (unsigned)b;
            return (((unsigned)(in[0] >> 32) ^ g) | ((unsigned)(in[1] >> 32) ^ g) |
                    ((unsigned)(in[2] >> 32) ^ g) | ((unsigned)(in[3] >> 32) ^ g)) != 0u;
        };
        const int32_t tin = b > 0 ? T - 31 : 0;  // steps at which columns come in
        if (tin > 0) peek(0);
        float up[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // the columns from the lane below
        unsigned long long* o = out + row0 - 4 * 31 + kBandPad;
        const unsigned long long tag = (unsigned long long)(b + 1) << 32;
        auto tile = [&](const float4 (&cc)[8], int32_t t) {
            // this step's columns for lane 0 were looked at a step ago: a band
            // that follows closely falls back by one step and then never waits
            if (t < tin) {
                for (int32_t polls = 0; missing() && !lost; ++polls) {
                    peek(t);
                    if (polls > kPolls) {
                        lost = true;
                        if (lane == 0) set_error(err, ND_ERR_INTERNAL, b);
                    }
                }
                __syncwarp();
            }
            float f[4], t4[8][4];
#pragma unroll
            for (int k = 0; k < 4; ++k) f[k] = lane == 0 ? __uint_as_float((unsigned)in[k]) : up[k];
            if (t + 1 < tin) peek(t + 1);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                t4[r][0] = cc[r].x; t4[r][1] = cc[r].y; t4[r][2] = cc[r].z; t4[r][3] = cc[r].w;
            }
            // a row starts from its own column: row r of the lane at column
            // r % 4 of its tile t - lane - 2 lane = r / 4
            const bool s0 = t == 3 * lane, s1 = t == 3 * lane + 1;
            // the tile by anti-diagonals, whose cells do not depend on one
            // another: a cell adds its term to its row's force and subtracts
            // that from its column's; a finished column leaves at once
#pragma unroll
            for (int s = 0; s < 11; ++s) {
                float fi[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int r = s - k;
                    if (r >= 0 && r < 8) fi[k] = __fadd_rn(a[r], t4[r][k]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int r = s - k;
                    if (r >= 0 && r < 8) {
                        a[r] = (r & 3) == k && (r < 4 ? s0 : s1) ? f[k] : fi[k];
                        f[k] = __fsub_rn(f[k], fi[k]);
                        if (r == 7) up[k] = __shfl_up_sync(0xffffffffu, f[k], 1);
                    }
                }
            }
            // the columns that left lane 31 (also those no later band reads)
            asm volatile(
                "{\n.reg .pred p;\nsetp.eq.s32 p, %0, 31;\n"
                "@p st.volatile.v2.u64 [%1], {%2, %3};\n"
                "@p st.volatile.v2.u64 [%1+16], {%4, %5};\n}" ::"r"(lane),
                "l"(o), "l"(tag | __float_as_uint(f[0])), "l"(tag | __float_as_uint(f[1])),
                "l"(tag | __float_as_uint(f[2])), "l"(tag | __float_as_uint(f[3]))
                : "memory");
            o += 4;
        };
        load(buf[0], 0);
        for (int32_t t = 0; t < T; t += 2) {  // T is even
            load(buf[1], t + 1);
            tile(buf[0], t);
            load(buf[0], t + 2);
            tile(buf[1], t + 1);
        }
        const int32_t i0 = row0 + 8 * lane;
#pragma unroll
        for (int r = 0; r < 8; ++r)
            if (i0 + r < n) F[i0 + r] = a[r];
    }
    cluster.sync();  // the next block's array is written until here
}

// Up to kLevelAtoms and beyond kBandMaxAtoms: the pairs with i + j = s form one
// level whose pairs touch distinct atoms, and level s follows level s - 1; one
// block runs the levels in order.  The pair terms are stored level by level (level s at
// level_off(s); its pairs by increasing i).

__host__ __device__ inline int32_t level_lo(int32_t s, int32_t n) { return max(0, s - (n - 1)); }
__host__ __device__ inline int32_t level_count(int32_t s, int32_t n) {
    return (s - 1) / 2 - level_lo(s, n) + 1;
}
// Pairs in the levels before s: level t <= n - 1 holds ceil(t / 2) pairs, so
// floor(s^2 / 4) for s <= n; the map (i, j) -> (n-1-j, n-1-i) reverses the
// levels, which gives P - floor((2n - 1 - s)^2 / 4) for s >= n - 1.
__host__ __device__ inline int64_t level_off(int32_t s, int32_t n) {
    if (s <= n) return (int64_t)s * s / 4;
    const int64_t r = 2 * (int64_t)n - 1 - s;
    return (int64_t)n * (n - 1) / 2 - r * r / 4;
}

// The pair terms of one level per block, from the positions with the same
// operations as update_pairslist! (so the same d).
__global__ void k_cs_cterms(const float* __restrict__ x, const float* __restrict__ q, int32_t n,
                            float* __restrict__ cterm) {
    const int32_t s = blockIdx.x + 1;
    const int32_t ilo = level_lo(s, n), cnt = level_count(s, n);
    float* out = cterm + level_off(s, n);
    for (int32_t k = threadIdx.x; k < cnt; k += blockDim.x) {
        const int32_t i = ilo + k, j = s - i;
        out[k] = coulomb_term(x[3 * (int64_t)i], x[3 * (int64_t)i + 1], x[3 * (int64_t)i + 2], q[i],
                              x[3 * (int64_t)j], x[3 * (int64_t)j + 1], x[3 * (int64_t)j + 2], q[j]);
    }
}

// The bands take 32 steps and a cluster launch at least, whatever the size.  us a
// step of simulate!, levels and bands: 1 atom 10.4 and 23.9, 4 atoms 15.1 and
// 22.1, 16 atoms 21.2 and 23.8, 24 atoms 27.4 and 23.1.
constexpr int kLevelAtoms = 16;

constexpr int kLevelThreads = 128;  // fewest warps paying the per-level overhead (measured: 128 of 32-1024)

// The recurrence by levels, accumulators in global memory (any n): the
// block's own writes are visible to it after each barrier.  The first item of
// the next level is loaded ahead.
__global__ void __launch_bounds__(kLevelThreads, 1)
    k_cs_coulomb_global(const float* __restrict__ cterm, int32_t n, float* F) {
    for (int32_t k = threadIdx.x; k < n; k += blockDim.x) F[k] = 0.0f;
    __syncthreads();
    const int32_t smax = 2 * n - 3;
    auto first = [&](int32_t s) -> float {
        if (s > smax || (int32_t)threadIdx.x >= level_count(s, n)) return 0.0f;
        return __ldg(&cterm[level_off(s, n) + threadIdx.x]);
    };
    float cn = first(1);
    for (int32_t s = 1; s <= smax; ++s) {
        const float c0 = cn;
        cn = first(s + 1);
        const int32_t ilo = level_lo(s, n), ihi = (s - 1) / 2;
        const float* cc = cterm + level_off(s, n);
        for (int32_t i = ilo + (int32_t)threadIdx.x; i <= ihi; i += blockDim.x) {
            const int32_t j = s - i;
            const float c = i == ilo + (int32_t)threadIdx.x ? c0 : __ldg(&cc[i - ilo]);
            const float fi = __fadd_rn(F[i], c);
            F[i] = fi;
            F[j] = __fsub_rn(F[j], fi);
        }
        __syncthreads();
    }
}

// One step's per-atom part (Simulator.jl:183-228): sum_forces!, the position
// update with a(t), the velocity update with a(t) + a(t - dt) (Fnext, the
// previous step's all-pairs forces), boundary_reflect! (:81-111), and the
// forces carried to the next step.  Every operation rounds to Float32 as in
// Julia (Float32 times Int64 promotes to Float32).
__global__ void k_cs_step(float* __restrict__ x, float* __restrict__ v, float* __restrict__ force,
                          float* __restrict__ fnext, const float* __restrict__ mass,
                          const float* __restrict__ ljthr, const float* __restrict__ ljall,
                          const float* __restrict__ cf, int32_t n, float dt, float dt2,
                          float3 lo, float3 hi, float* __restrict__ frame) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float m = mass[i];
    const float at = __fdiv_rn(__fadd_rn(ljthr[i], cf[i]), m);  // accels_t
    const float fn = __fadd_rn(ljall[i], cf[i]);                // force_nextstep
    const float l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int64_t e = 3 * (int64_t)i + k;
        float xk = x[e], vk = v[e];
        // position .+= velocity .* dt .+ ((accels_t .* dt ^ 2) ./ 2)
        xk = __fadd_rn(xk, __fadd_rn(__fmul_rn(vk, dt), __fdiv_rn(__fmul_rn(at, dt2), 2.0f)));
        const float atdt = __fdiv_rn(fnext[e], m);  // accels_t_dt
        // velocity .+= (accels_t .+ accels_t_dt) .* dt / 2
        vk = __fadd_rn(vk, __fdiv_rn(__fmul_rn(__fadd_rn(at, atdt), dt), 2.0f));
        if (l[k] > xk) {
            vk = __fmul_rn(vk, -1.0f);
            xk = l[k];
        }
        if (h[k] < xk) {
            vk = __fmul_rn(vk, -1.0f);
            xk = h[k];
        }
        x[e] = xk;
        v[e] = vk;
        force[e] = fn;
        fnext[e] = fn;
        if (frame) frame[e] = xk;
    }
}

// rescale_velocity!(velocity, Tf, gamma, mass, objectcount) (Simulator.jl:
// 119-144): Ti += (2 / (3 objects kb)) * |v_i| * m_i / 2 in Float32, in atom
// order; beta = (1 + gamma (Tf / Ti - 1))^0.5 in Float64 (Float32 ^ Float64
// promotes; the square root correctly rounded); v .*= beta through Float64.
// A negative radicand raises ND_ERR_ARG and leaves v unchanged.  One block.
__global__ void __launch_bounds__(1024) k_cs_rescale(float* __restrict__ v,
                                                     const float* __restrict__ mass, int32_t n,
                                                     float c, float Tf, float gamma,
                                                     float* __restrict__ term, int32_t* err) {
    __shared__ double beta;
    __shared__ int ok;
    for (int32_t k = threadIdx.x; k < n; k += blockDim.x) {
        const float a = v[3 * (int64_t)k], b = v[3 * (int64_t)k + 1], z = v[3 * (int64_t)k + 2];
        const float s = __fadd_rn(__fadd_rn(__fmul_rn(a, a), __fmul_rn(b, b)), __fmul_rn(z, z));
        term[k] = __fdiv_rn(__fmul_rn(__fmul_rn(c, __fsqrt_rn(s)), mass[k]), 2.0f);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float Ti = 0.0f;
        for (int32_t k = 0; k < n; ++k) Ti = __fadd_rn(Ti, term[k]);
        const float r = __fadd_rn(1.0f, __fmul_rn(gamma, __fsub_rn(__fdiv_rn(Tf, Ti), 1.0f)));
        ok = !(r < 0.0f);
        if (ok) beta = __dsqrt_rn((double)r);
        else set_error(err, ND_ERR_ARG, 1);
    }
    __syncthreads();
    if (!ok) return;
    for (int64_t e = threadIdx.x; e < 3 * (int64_t)n; e += blockDim.x)
        v[e] = __double2float_rn(__dmul_rn((double)v[e], beta));
}

}  // namespace

nd_status compat_simulate(Ctx* c, const nd_compat_sim* spec, int32_t n, float* x, float* v,
                          float* force, const float* mass, const float* q, float* poslog) {
    if (!spec || !x || !v || !force || !mass || !q) return ND_ERR_ARG;
    if (n < 1 || n > 65536 || spec->duration < 0) {
        c->last_error = "nd_compat_simulate: 1 <= n <= 65536 and duration >= 0";
        return ND_ERR_ARG;
    }
    const size_t n3 = 3 * (size_t)n;
    const int64_t P = (int64_t)n * (n - 1) / 2;
    // device log: a chunk of frames, flushed to the host when full
    const int64_t frame_bytes = (int64_t)(n3 * sizeof(float));
    int64_t chunk_frames = (256ll << 20) / frame_bytes;
    // test hooks: a smaller log chunk (several flushes) and the global-memory
    // Coulomb form at any size; both compute the same results
    if (const char* ev = getenv("NAIVEGPU_COMPAT_LOG_CHUNK")) chunk_frames = atoll(ev);
    const bool force_global = getenv("NAIVEGPU_COMPAT_GLOBAL") != nullptr;
    const int64_t chunk =
        poslog ? std::max<int64_t>(1, std::min<int64_t>(spec->duration, chunk_frames)) : 0;
    nd_status st;
    // Coulomb terms: in band order, or by level for the global-memory form
    const bool bands = !force_global && n > kLevelAtoms && n <= kBandMaxAtoms;
    const int32_t nband = (int32_t)cdiv(n, kBandRows), P4 = band_steps(n);
    const int32_t nlev = std::max(2 * n - 3, 0);
    const size_t ncterm =
        bands ? 1024 * (size_t)band_off(nband, P4) : (size_t)std::max<int64_t>(P, 1);
    if ((st = ensure(c, c->leafpairs, sizeof(float) * ncterm))) return st;
    const size_t small = sizeof(float) * (4 * n3 + 6 * (size_t)n);
    if ((st = ensure(c, c->compat, small + (size_t)(chunk * frame_bytes)))) return st;
    float* cterm = (float*)c->leafpairs.p;  // Coulomb pair terms
    float* dx = (float*)c->compat.p;
    float* dv = dx + n3;
    float* dF = dv + n3;
    float* dFn = dF + n3;
    float* dm = dFn + n3;
    float* dq = dm + n;
    float* ljthr = dq + n;
    float* ljall = ljthr + n;
    float* cf = ljall + n;
    float* term = cf + n;
    float* dlog = term + n;
    cudaStream_t s = c->stream;
    cudaError_t e = cudaMemcpyAsync(dx, x, n3 * sizeof(float), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dv, v, n3 * sizeof(float), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)  // force_nextstep = deepcopy(sys.force)
        e = cudaMemcpyAsync(dFn, force, n3 * sizeof(float), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dF, force, n3 * sizeof(float), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dm, mass, n * sizeof(float), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dq, q, n * sizeof(float), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return cuda_fail(c, e, "compat simulate upload");

    // bands over one cluster of up to eight blocks, the rings as deep as the
    // shared memory beside the columns allows
    const unsigned nblk = (unsigned)std::min(nband, 8), nwarp = (unsigned)cdiv(nband, nblk);
    const void* band_fn = (const void*)k_cs_coulomb_bands<true, 160>;
    size_t band_smem = (size_t)band_col_bytes(n);
    int32_t ldepth = 3;
    if (bands) {
        int maxsm = 0;
        cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
        auto ring = [&](int32_t l) { return ((size_t)nwarp * (kBandCopy * 4096 + 8)) << l; };
        while (ldepth > 0 && (band_smem + ring(ldepth) > (size_t)maxsm || nwarp > 5)) --ldepth;
        if (ldepth > 0) band_smem += ring(ldepth);
        else band_fn = (const void*)k_cs_coulomb_bands<false, 320>;
        // one limit whatever the size: the attribute belongs to the process
        e = cudaFuncSetAttribute(band_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, maxsm);
        if (e != cudaSuccess) return cuda_fail(c, e, "compat simulate smem");
    }
    // Two chains per step, both from the list of the previous step's
    // positions: force_coulomb! (update_pairslist!'s Coulomb terms, then the
    // recurrence on up to eight SMs) on the context's stream, and
    // force_lennardjones! on a side stream over the other SMs.  The step kernel waits for both; the side chain of
    // the next step waits for the step kernel.
    struct Side {
        cudaStream_t s2 = nullptr;
        cudaEvent_t moved = nullptr, lj = nullptr;
        ~Side() {
            if (s2) cudaStreamSynchronize(s2);
            if (moved) cudaEventDestroy(moved);
            if (lj) cudaEventDestroy(lj);
            if (s2) cudaStreamDestroy(s2);
        }
    } side;
    e = cudaStreamCreateWithFlags(&side.s2, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&side.moved, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&side.lj, cudaEventDisableTiming);
    if (e != cudaSuccess) return cuda_fail(c, e, "compat simulate streams");
    cudaStream_t s2 = side.s2;
    auto coulomb_terms = [&]() {
        if (bands) {
            k_cs_band_terms<<<dim3((unsigned)P4, (unsigned)nband), 256, 0, s>>>(
                dx, dq, n, P4, (float4*)cterm);
            c->launches++;
        } else if (n > 1) {
            k_cs_cterms<<<nlev, 256, 0, s>>>(dx, dq, n, cterm);
            c->launches++;
        }
    };
    auto coulomb = [&]() -> cudaError_t {
        c->launches++;
        if (!bands) {
            k_cs_coulomb_global<<<1, kLevelThreads, 0, s>>>(cterm, n, cf);
            return cudaSuccess;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(nblk);
        cfg.blockDim = dim3(32 * nwarp);
        cfg.dynamicSmemBytes = band_smem;
        cfg.stream = s;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nblk;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        const float4* ct = (const float4*)cterm;
        int32_t nn = n, pp = P4, ld = ldepth;
        float* ff = cf;
        int32_t* ee = c->d_err;
        void* args[] = {&ct, &nn, &pp, &ld, &ff, &ee};
        return cudaLaunchKernelExC(&cfg, band_fn, args);
    };
    // after the positions of stream `after` moved: the LJ sums on s2
    auto lj_chain = [&](cudaStream_t after) -> cudaError_t {
        cudaError_t ee = cudaEventRecord(side.moved, after);
        if (ee == cudaSuccess) ee = cudaStreamWaitEvent(s2, side.moved, 0);
        if (ee != cudaSuccess) return ee;
        k_cs_lj<<<(unsigned)cdiv(n, 32), 288, 0, s2>>>(dx, n, 0.01f, ljthr, ljall);
        c->launches++;
        return cudaEventRecord(side.lj, s2);
    };
    const float dt = (float)spec->stepwidth;
    const float dt2 = (float)(int64_t)((uint64_t)spec->stepwidth * (uint64_t)spec->stepwidth);
    const float3 lo = make_float3(spec->min_dim[0], spec->min_dim[1], spec->min_dim[2]);
    const float3 hi = make_float3(spec->max_dim[0], spec->max_dim[1], spec->max_dim[2]);
    // rescale_velocity!: 2 / (3 * objects * kb), objects = Float32(objectnumber), kb = 1
    const float cT = 2.0f / ((3.0f * (float)spec->objectnumber) * 1.0f);
    const unsigned ga = (unsigned)cdiv(n, 256);

    // pairslist = unique_pairs(position)
    coulomb_terms();
    if ((e = lj_chain(s)) != cudaSuccess) return cuda_fail(c, e, "compat simulate streams");
    int64_t pending = 0;  // frames in the device chunk not yet copied out
    int64_t first = 1;    // step of the chunk's first frame
    auto flush = [&]() -> nd_status {
        if (pending == 0) return ND_OK;
        cudaError_t ee = cudaMemcpyAsync(poslog + first * (int64_t)n3, dlog,
                                         (size_t)(pending * frame_bytes), cudaMemcpyDeviceToHost, s);
        if (ee != cudaSuccess) return cuda_fail(c, ee, "compat simulate log");
        ee = cudaStreamSynchronize(s);
        if (ee != cudaSuccess) return cuda_fail(c, ee, "compat simulate log");
        first += pending;
        pending = 0;
        return ND_OK;
    };
    for (int64_t step = 1; step <= spec->duration; ++step) {
        // force_coulomb! runs twice per step on the same list and charges: one
        // evaluation gives both results; so does force_lennardjones!'s pass
        // over the whole list and its threshold_pairs part
        if ((e = coulomb()) != cudaSuccess) return cuda_fail(c, e, "compat simulate (Coulomb)");
        float* frame = poslog ? dlog + pending * (int64_t)n3 : nullptr;
        e = cudaStreamWaitEvent(s, side.lj, 0);
        if (e != cudaSuccess) return cuda_fail(c, e, "compat simulate streams");
        k_cs_step<<<ga, 256, 0, s>>>(dx, dv, dF, dFn, dm, ljthr, ljall, cf, n, dt, dt2, lo, hi,
                                      frame);
        c->launches++;
        if (step < spec->duration) {  // update_pairslist! (unused after the last step)
            coulomb_terms();
            if ((e = lj_chain(s)) != cudaSuccess) return cuda_fail(c, e, "compat simulate streams");
        }
        if (step % 10 == 0) {
            k_cs_rescale<<<1, 1024, 0, s>>>(dv, dm, n, cT, spec->temperature,
                                             spec->velocity_dampening, term, c->d_err);
            c->launches++;
            if ((st = sync_and_check(c, "compat simulate (rescale_velocity!)"))) {
                // the reference throws here: hand back the state it holds
                cudaMemcpyAsync(x, dx, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
                cudaMemcpyAsync(v, dv, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
                cudaMemcpyAsync(force, dF, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
                cudaStreamSynchronize(s);
                c->last_error = "rescale_velocity!: negative radicand (DomainError)";
                return st;
            }
        }
        if (poslog && ++pending == chunk && (st = flush())) return st;
        if ((st = check_launch(c, "compat simulate"))) return st;
    }
    if (poslog && (st = flush())) return st;
    e = cudaMemcpyAsync(x, dx, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(v, dv, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(force, dF, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess && poslog)  // poslog[1] is sys.position itself
        e = cudaMemcpyAsync(poslog, dx, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return cuda_fail(c, e, "compat simulate download");
    return sync_and_check(c, "compat simulate");
}

namespace {

// ------------------------------------------------ collect_objects
// collect_objects(::GenericRandomCollector) (MDInput.jl:305-369) with a
// counter-based stream in place of Julia's global RNG: draw k of stream c is
// mix64(seed ^ mix64(c << 56 ^ k)).  Uniform(a, b) as Distributions draws it:
// a + (b - a) * u with u in [0, 1) (53 bits), stored as Float32; rand(Float32)
// for the velocity split: 24 bits.

__host__ __device__ inline uint64_t cobj_bits(uint64_t seed, uint64_t stream, uint64_t k) {
    return mix64(seed ^ mix64((stream << 56) ^ k));
}
__host__ __device__ inline float cobj_uniform(uint64_t seed, uint64_t stream, uint64_t k, float a,
                                              float b) {
    const double u = (double)(cobj_bits(seed, stream, k) >> 11) * 0x1.0p-53;
    return (float)((double)a + (double)(b - a) * u);
}
__host__ __device__ inline float cobj_rand32(uint64_t seed, uint64_t stream, uint64_t k) {
    return (float)(cobj_bits(seed, stream, k) >> 40) * 0x1.0p-24f;
}

// mass, charge, position (generate_positions, MDInput.jl:175-190) and the
// velocity split draws of every atom.
__global__ void k_cobj_draw(nd_collector cl, uint64_t seed, int32_t n, float* __restrict__ x,
                            float* __restrict__ m, float* __restrict__ q,
                            float* __restrict__ vd) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    m[i] = cobj_uniform(seed, 0, i, cl.minmass, cl.maxmass);
    q[i] = cobj_uniform(seed, 1, i, cl.mincharge, cl.maxcharge);
    for (int d = 0; d < 3; ++d) {
        x[3 * (int64_t)i + d] = cobj_uniform(seed, 2 + d, i, cl.min_dim[d], cl.max_dim[d]);
        vd[(int64_t)d * n + i] = cobj_rand32(seed, 5 + d, i);
    }
}

// sum(veldist) per dimension in a fixed order: 256-element chunks reduced as
// a binary tree (stride 128, 64, .., 1), then the chunk sums in chunk order.
__global__ void __launch_bounds__(256) k_cobj_chunks(const float* __restrict__ vd, int32_t n,
                                                     int32_t nchunk, float* __restrict__ part) {
    __shared__ float t[256];
    const int d = blockIdx.y;
    const int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x;
    t[threadIdx.x] = k < n ? vd[(int64_t)d * n + k] : 0.0f;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) t[threadIdx.x] = __fadd_rn(t[threadIdx.x], t[threadIdx.x + w]);
        __syncthreads();
    }
    if (threadIdx.x == 0) part[(int64_t)d * nchunk + blockIdx.x] = t[0];
}

__global__ void k_cobj_total(const float* __restrict__ part, int32_t nchunk, float* sum) {
    const int d = threadIdx.x;
    if (d >= 3) return;
    float s = 0.0f;
    for (int32_t c = 0; c < nchunk; ++c) s = __fadd_rn(s, part[(int64_t)d * nchunk + c]);
    sum[d] = s;
}

// velocity[i][d] = T * veldist[i] * 3 * N * kb / mass[i] with veldist ./=
// sum(veldist), or T / N * 3 * N * kb / mass[i] (kb = 1), in Float32.
__global__ void k_cobj_velocity(nd_collector cl, int32_t n, const float* __restrict__ m,
                                const float* __restrict__ vd, const float* __restrict__ sum,
                                float* __restrict__ v) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float N = (float)cl.objectnumber;
    for (int d = 0; d < 3; ++d) {
        float a;
        if (cl.randomvelocity) {
            const float vn = __fdiv_rn(vd[(int64_t)d * n + i], sum[d]);
            a = __fmul_rn(__fmul_rn(__fmul_rn(cl.temperature, vn), 3.0f), N);
        } else {
            a = __fmul_rn(__fmul_rn(__fdiv_rn(cl.temperature, N), 3.0f), N);
        }
        v[3 * (int64_t)i + d] = __fdiv_rn(__fmul_rn(a, 1.0f), m[i]);
    }
}

// unique_pairs_prune (MDInput.jl:228-259) as written: for i in 1:N-1, j in
// i+1:N-1 (the last atom is never compared), sqrt(dx^2 + dy^2 + dz^2) <
// minimumdistance fills a[i] with Inf.  A filled a[i] meets nothing after,
// and every a[j] compared is still the drawn one, so atom i is filled exactly
// when some j in (i, N-1) lies within the distance of it: one thread per i,
// the candidates staged through shared memory.
__global__ void __launch_bounds__(256) k_cobj_prune(const float* __restrict__ x, int32_t n,
                                                    float dmin, unsigned char* __restrict__ hit) {
    __shared__ float3 tile[256];
    const int32_t i = blockIdx.x * 256 + threadIdx.x;
    const int32_t jmax = n - 2;  // last compared atom, 0-based
    float3 a = make_float3(0.f, 0.f, 0.f);
    if (i < n) a = make_float3(x[3 * (int64_t)i], x[3 * (int64_t)i + 1], x[3 * (int64_t)i + 2]);
    bool found = false;
    for (int32_t j0 = blockIdx.x * 256; j0 <= jmax; j0 += 256) {
        const int32_t jl = j0 + threadIdx.x;
        if (jl <= jmax)
            tile[threadIdx.x] =
                make_float3(x[3 * (int64_t)jl], x[3 * (int64_t)jl + 1], x[3 * (int64_t)jl + 2]);
        __syncthreads();
        if (!found && i < jmax) {
            const int32_t kend = min(256, jmax - j0 + 1);
            for (int k = max(0, i + 1 - j0); k < kend; ++k) {
                const float dx = __fsub_rn(a.x, tile[k].x), dy = __fsub_rn(a.y, tile[k].y),
                            dz = __fsub_rn(a.z, tile[k].z);
                const float d = __fsqrt_rn(
                    __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
                if (d < dmin) {
                    found = true;
                    break;
                }
            }
        }
        __syncthreads();
    }
    if (i < n) hit[i] = found;
}

__global__ void k_cobj_fill(float* __restrict__ x, const unsigned char* __restrict__ hit, int32_t n,
                            unsigned long long* count) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !hit[i]) return;
    x[3 * (int64_t)i] = x[3 * (int64_t)i + 1] = x[3 * (int64_t)i + 2] = __int_as_float(0x7f800000);
    atomicAdd(count, 1ull);
}

}  // namespace

nd_status collect_objects(Ctx* c, const nd_collector* cl, uint64_t seed, float* x, float* v,
                          float* m, float* q, int64_t* pruned) {
    if (!cl || !x || !v || !m || !q) return ND_ERR_ARG;
    // the pruning compares every pair (as the reference does): 2^20 atoms
    // are 5e11 comparisons, about a second
    if (cl->objectnumber < 1 || cl->objectnumber > (1 << 20)) {
        c->last_error = "nd_collect_objects: 1 <= objectnumber <= 2^20";
        return ND_ERR_ARG;
    }
    const int32_t n = (int32_t)cl->objectnumber;
    const size_t n3 = 3 * (size_t)n;
    const int32_t nchunk = (int32_t)cdiv(n, 256);
    nd_status st;
    // [count (16 B)] [x, v, m, q, veldist, chunk sums, sums (Float32)] [hit (bytes)]
    const size_t nf = 2 * n3 + 2 * (size_t)n + n3 + 3 * (size_t)nchunk + 4;
    if ((st = ensure(c, c->compat, 16 + sizeof(float) * nf + (size_t)n))) return st;
    unsigned long long* cnt = (unsigned long long*)c->compat.p;
    float* dx = (float*)((char*)c->compat.p + 16);
    float* dv = dx + n3;
    float* dm = dv + n3;
    float* dq = dm + n;
    float* vd = dq + n;
    float* part = vd + n3;
    float* sum = part + 3 * (size_t)nchunk;
    unsigned char* hit = (unsigned char*)(sum + 4);
    cudaStream_t s = c->stream;
    const unsigned g = (unsigned)cdiv(n, 256);
    cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), s);
    k_cobj_draw<<<g, 256, 0, s>>>(*cl, seed, n, dx, dm, dq, vd);
    if (cl->randomvelocity) {
        k_cobj_chunks<<<dim3((unsigned)nchunk, 3), 256, 0, s>>>(vd, n, nchunk, part);
        k_cobj_total<<<1, 32, 0, s>>>(part, nchunk, sum);
        c->launches += 2;
    }
    k_cobj_velocity<<<g, 256, 0, s>>>(*cl, n, dm, vd, sum, dv);
    k_cobj_prune<<<g, 256, 0, s>>>(dx, n, cl->minimumdistance, hit);
    k_cobj_fill<<<g, 256, 0, s>>>(dx, hit, n, cnt);
    c->launches += 4;
    if ((st = check_launch(c, "collect_objects"))) return st;
    unsigned long long h_cnt = 0;
    cudaError_t e = cudaMemcpyAsync(x, dx, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(v, dv, n3 * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(m, dm, n * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(q, dq, n * sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&h_cnt, cnt, sizeof(h_cnt), cudaMemcpyDeviceToHost, s);
    if (e != cudaSuccess) return cuda_fail(c, e, "collect_objects download");
    if ((st = sync_and_check(c, "collect_objects"))) return st;
    if (pruned) *pruned = (int64_t)h_cnt;
    return ND_OK;
}

nd_status compat_forces(Ctx* c, int kind, int32_t n, const int32_t* pi, const int32_t* pj,
                        const float* pd, int64_t np, const float* q, float* force) {
    if (n <= 0 || np < 0 || !force || (np > 0 && (!pi || !pj || !pd)) || (kind == 1 && !q))
        return ND_ERR_ARG;
    if (np > INT32_MAX) return ND_ERR_ARG;
    for (int64_t p = 0; p < np; ++p)
        if (pi[p] < 1 || pi[p] > n || pj[p] < 1 || pj[p] > n) return ND_ERR_ARG;
    const size_t nx = 3 * (size_t)n;
    nd_status st;
    if ((st = ensure(c, c->pairs_i, sizeof(int32_t) * (size_t)std::max<int64_t>(np, 1)))) return st;
    if ((st = ensure(c, c->pairs_j, sizeof(int32_t) * (size_t)std::max<int64_t>(np, 1)))) return st;
    if ((st = ensure(c, c->pairs_d, sizeof(float) * (size_t)std::max<int64_t>(np, 1)))) return st;
    if ((st = ensure(c, c->counts, sizeof(float) * (nx + (size_t)n) + 2 * sizeof(int32_t) * n))) return st;
    int32_t* dpi = (int32_t*)c->pairs_i.p;
    int32_t* dpj = (int32_t*)c->pairs_j.p;
    float* dpd = (float*)c->pairs_d.p;
    float* dforce = (float*)c->counts.p;
    float* dF = dforce + nx;  // Coulomb accumulators, or LJ run starts / ends
    int32_t* start = (int32_t*)(dF + n);
    int32_t* end = start + n;
    cudaError_t e = cudaSuccess;
    if (np > 0) {
        e = cudaMemcpyAsync(dpi, pi, sizeof(int32_t) * np, cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dpj, pj, sizeof(int32_t) * np, cudaMemcpyHostToDevice, c->stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(dpd, pd, sizeof(float) * np, cudaMemcpyHostToDevice, c->stream);
    }
    if (e != cudaSuccess) return cuda_fail(c, e, "compat forces upload");
    cudaMemsetAsync(dforce, 0, sizeof(float) * nx, c->stream);
    const unsigned ga = (unsigned)cdiv(n, 256);
    if (kind == 0 && np > 0) {
        // stable sort of the pairs by i: keys i (1-based), values the list positions
        if ((st = ensure(c, c->codes, sizeof(uint32_t) * np))) return st;
        if ((st = ensure(c, c->perm, sizeof(int32_t) * np))) return st;
        uint32_t* key = (uint32_t*)c->codes.p;
        int32_t* order = (int32_t*)c->perm.p;
        e = cudaMemcpyAsync(key, pi, sizeof(int32_t) * np, cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "compat forces upload");
        k_iota<<<(unsigned)cdiv(np, 256), 256, 0, c->stream>>>(order, np);
        int bits = 1;
        while (bits < 31 && ((uint32_t)n >> bits) != 0) ++bits;
        if ((st = radix_sort_pairs(c, key, order, (int32_t)np, bits))) return st;
        cudaMemsetAsync(start, 0, sizeof(int32_t) * n, c->stream);
        cudaMemsetAsync(end, 0, sizeof(int32_t) * n, c->stream);
        k_compat_runs<<<(unsigned)cdiv(np, 256), 256, 0, c->stream>>>(key, np, start, end);
        k_compat_lj<<<ga, 256, 0, c->stream>>>(order, dpd, start, end, n, dforce);
        c->launches += 3;
    } else if (kind == 1) {
        float* dq = dF + n;  // charges after the accumulators (reuse of the run arrays)
        e = cudaMemcpyAsync(dq, q, sizeof(float) * n, cudaMemcpyHostToDevice, c->stream);
        if (e != cudaSuccess) return cuda_fail(c, e, "compat forces upload");
        cudaMemsetAsync(dF, 0, sizeof(float) * n, c->stream);
        if (np > 0) {
            k_compat_coulomb<<<1, 32, 0, c->stream>>>(dpi, dpj, dpd, np, dq, dF, n, c->d_err);
            c->launches++;
        }
        k_compat_spread<<<ga, 256, 0, c->stream>>>(dF, n, dforce);
        c->launches++;
    }
    if ((st = check_launch(c, "compat forces"))) return st;
    e = cudaMemcpyAsync(force, dforce, sizeof(float) * nx, cudaMemcpyDeviceToHost, c->stream);
    if (e != cudaSuccess) return cuda_fail(c, e, "compat forces download");
    return sync_and_check(c, "compat forces");
}

}  // namespace nd
