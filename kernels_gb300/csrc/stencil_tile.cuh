// The TMA tile kernel, templated on pattern, radius, storage form and temporal depth.
//
// One CTA per TH x TW tile of the grid, as many resident per SM as shared memory allows. The elected
// thread issues two 2D TMA loads that complete on one mbarrier: the `in` tile with its halo and the
// `out` tile. The halo is R rows above and below and RA >= R columns either side, RA rounded up to
// 16 bytes so every TMA x coordinate is 16-byte aligned; the hardware zero-fills what lies outside
// the grid. The resident CTAs of an SM overlap one another's loads and evaluation. (A persistent
// variant with a ring of stages per CTA measured slower here: fewer warps per SM to evaluate each
// tile, and CTAs drifting apart in the raster order.)
//
// In a tile, lane l owns CPT adjacent columns (one 16-byte vector) and warp w owns the ROWS
// consecutive rows from w * ROWS, so that the rows of a thread share their vertical taps in
// registers. in_next and out go straight to HBM with 16-byte stores.
//
// Temporal depth STEPS: the tile applies STEPS consecutive applications before writing back.
// `in` evolves pointwise (in_{k+1} = in_k + 1, Cxx11/stencil-openmp.cc:208-218), so the copy in
// shared memory, halo included, is advanced in place with the same rounded +1 the reference
// applies, and the halo never grows. Every application reads the current `in` values and applies
// every tap. `out` stays in registers and is rounded after each application as the reference
// rounds it. HBM traffic per application drops by STEPS. STEPS = 0 takes the depth at run time
// (`depth`, any count): a whole run in one launch per tile, as the host-buffer path uses it on
// bands of rows. STEPS = OPERATOR is the reference operator alone: out += S(in), no in_next.
//
// Evaluation, chosen per tile from its values; FP64 gives the bits of the reference's order on every route:
//   FP64, star R=1,2 and grid R=1   whole numbers: FP32 or integer arithmetic (prk_fixed.cuh); else binary64,
//                  the power-of-two products joined to the adds
//   FP64, the others   whole numbers of a small range: products from tables, the chain in fixed point (the
//                  64-bit narrow form, else 96 bits); other whole numbers: products on the integer pipes;
//                  reals: products shared between taps or joined to the adds; else every product and add
//                  in binary64
//   FP32C          whole numbers near one another: the taps times the weights' common denominator, exact in
//                  FP32 (the integer route); else paired differences summed per weight group (the operator
//                  form: one product per tap), split weights, TwoSum, two-float out (prk_arith.cuh)
#pragma once

#include <cuda.h>

#include <type_traits>

#include "prk_arith.cuh"
#include "prk_fixed.cuh"
#include "prk_internal.cuh"
#include "prk_ptx.cuh"

namespace prk {
namespace tile {

constexpr int THREADS = 256;
constexpr int WARPS = THREADS / 32;

// Tile shape per storage form: TW columns (CPT per lane, one 16-byte vector) by TH rows (TH/8 per
// warp). TH is the tile-height variant the autotuner chooses between (32: 4 rows per thread; 64: 8).
template <int DT, int TH_ = 32>
struct Cfg;
template <int TH_>
struct Cfg<FP64, TH_> {
    using T = double;
    static constexpr int TW = 64, TH = TH_, CPT = 2, VEC = 2;
};
template <int TH_>
struct Cfg<FP32C, TH_> {
    using T = float;
    static constexpr int TW = 128, TH = TH_, CPT = 4, VEC = 4;
};
constexpr int TH_DEFAULT = 32;
constexpr int TH_TALL = 64;
// STEPS of the operator form: one application of out += S(in), in untouched and no in_next. It takes
// the same tiles and routes as the fused form and stores no in_next, so a power-of-two stencil moves 24
// bytes per point at the copy rate: at n=8192, FP64, star R=2 2049 us on the generic kernels, 229 us
// here (7.0 TB/s); grid R=4 18273 against 2134 us; FP32C star R=2 369 against 193 us, grid R=5 1677
// against 365 us (reals: 1571).
constexpr int OPERATOR = -1;
constexpr bool one_application(int steps) { return steps == 1 || steps == OPERATOR; }
// Deepest run-time depth for which the FP32 route holds: 15 * (2^20 + 65536) < 2^24.
constexpr int FP32_MAX_STEPS = 65536;

constexpr int SMEM_PER_SM = 228 * 1024;
constexpr int SMEM_PER_CTA_MAX = 227 * 1024;
constexpr int SMEM_DEFAULT_MAX = 48 * 1024;  // without cudaFuncAttributeMaxDynamicSharedMemorySize

template <int DT, int R, int TH_ = 32>
struct Geo {
    using C = Cfg<DT, TH_>;
    using T = typename C::T;
    static constexpr int RA = ((R + C::VEC - 1) / C::VEC) * C::VEC;  // halo columns, 16-byte multiple
    static constexpr int SW = C::TW + 2 * RA;                        // in-tile row length = TMA box x
    static constexpr int SH = C::TH + 2 * R;                         // in-tile rows = TMA box y
    static constexpr int IN_BYTES = SW * SH * static_cast<int>(sizeof(T));
    static constexpr int OUT_BYTES = C::TW * C::TH * 8;
    static constexpr int OUT_OFF = (IN_BYTES + 127) / 128 * 128;     // out tile
    static constexpr int RED_OFF = OUT_OFF + OUT_BYTES;              // per-warp words of the certification
    static constexpr int BAR_OFF = RED_OFF + WARPS * 8;
    static constexpr int SMEM = BAR_OFF + 8;
    static constexpr int CTAS_FIT = SMEM_PER_SM / (SMEM + 1024);     // 1 KB per CTA is reserved
    static constexpr int CTAS = CTAS_FIT > 8 ? 8 : CTAS_FIT;         // resident CTAs per SM
    static constexpr int ELEMS = SW * SH;
    static constexpr int ROWS = C::TH / WARPS;
    static_assert(SMEM <= SMEM_PER_CTA_MAX && CTAS >= 1, "the tile must fit in shared memory");
    static_assert(SW <= 256 && SH <= 256 && C::TW <= 256, "TMA box dimensions are at most 256");
    static_assert((SW * sizeof(T)) % 16 == 0, "TMA box rows must be 16-byte multiples");
    static_assert(C::TH % WARPS == 0 && C::TW == 32 * C::CPT, "thread layout");
};

// Everything a launch needs besides the template arguments.
struct Launch {
    CUtensorMap tm_in;
    CUtensorMap tm_out;
    int64_t n;
    void* in_next;
    void* out;
    unsigned* status;
    cudaStream_t stream;
    int depth;     // applications per launch for the run-time-depth kernels (STEPS = 0)
    int64_t row0;  // first array row of the launch's tiles
    int64_t rows;  // array rows covered from row0 (0: to the last row of the arrays)
    int64_t nr;    // rows the arrays hold (0: n, a whole grid); the tensor maps cover nr x n
    int64_t goff;  // grid row of the arrays' row 0
};

// ---------------------------------------------------------------------------------------------
// 16-byte vector access helpers

__device__ __forceinline__ void st_vec(double* p, const double (&v)[2])
{
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void st_vec(float* p, const float (&v)[4])
{
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// N consecutive floats from 16-byte-aligned shared memory.
template <int N>
__device__ __forceinline__ void ld_seg(const float* p, float (&v)[N])
{
    static_assert(N % 4 == 0, "segment is whole float4 vectors");
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const float4 t = reinterpret_cast<const float4*>(p)[q];
        v[4 * q] = t.x;
        v[4 * q + 1] = t.y;
        v[4 * q + 2] = t.z;
        v[4 * q + 3] = t.w;
    }
}

// N consecutive fixed-point words from 16-byte-aligned shared memory, narrowed to I.
template <int N, typename I>
__device__ __forceinline__ void ld_seg_i(const int64_t* p, I (&v)[N])
{
    static_assert(N % 2 == 0, "segment is whole 16-byte vectors");
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
        const longlong2 t = reinterpret_cast<const longlong2*>(p)[q];
        v[2 * q] = static_cast<I>(t.x);
        v[2 * q + 1] = static_cast<I>(t.y);
    }
}

// ---------------------------------------------------------------------------------------------
// FP32C: the stencil sums of CPT points of one row. s points at in(r, c0) in the smem tile.

// The taps of a PRK stencil share few distinct weights: star R has R (1/(2kR) on the k-th ring of
// the cross), grid R has 2R (the sides and the diagonal of each ring). Group g collects the paired
// differences whose weight is +-c_g: D_g = sum of sign * (in[p+d] - in[p-d]). Every tap's two values
// are read and differenced; the sums within a group are exact for integer fields (they stay below
// 2^24), and the weights then enter through NG compensated products instead of one per tap.
template <int P, int R>
__host__ __device__ constexpr int group_count() { return P == STAR ? R : 2 * R; }

// Group of the positive tap (dc, dr) (dr > 0, or dr == 0 and dc > 0) and the sign of its weight.
template <int P, int R>
__host__ __device__ constexpr int group_of(int dc, int dr)
{
    const int adc = dc > 0 ? dc : -dc, adr = dr > 0 ? dr : -dr;
    const int m = adc > adr ? adc : adr;
    if (P == STAR) return m - 1;
    return (adc == m && adr == m) ? R + m - 1 : m - 1;  // diagonal of ring m, else its sides
}

// |weight| of group g, as a (hi, lo) float pair.
template <int P, int R>
__host__ __device__ constexpr double group_weight(int g)
{
    if (P == STAR) return weight(STAR, R, 0, g + 1);
    return g < R ? weight(GRID, R, 0, g + 1) : weight(GRID, R, g - R + 1, g - R + 1);
}

// Every positive tap's |weight| is its group's weight (checked at compile time for all stencils).
template <int P, int R>
__host__ __device__ constexpr bool groups_ok()
{
    for (int dr = 0; dr <= R; ++dr)
        for (int dc = -R; dc <= R; ++dc) {
            if (dr == 0 && dc <= 0) continue;
            const double w = weight(P, R, dc, dr);
            if (w != 0.0 && (w > 0 ? w : -w) != group_weight<P, R>(group_of<P, R>(dc, dr))) return false;
        }
    return true;
}
static_assert(groups_ok<STAR, 1>() && groups_ok<STAR, 2>() && groups_ok<STAR, 3>() && groups_ok<STAR, 4>() &&
                  groups_ok<STAR, 5>() && groups_ok<GRID, 1>() && groups_ok<GRID, 2>() && groups_ok<GRID, 3>() &&
                  groups_ok<GRID, 4>() && groups_ok<GRID, 5>(),
              "weight groups");

template <int P, int R, int CPT, int RA>
__device__ __forceinline__ void fp32c_points(const float* s, int ld, float (&sh)[CPT], float (&sl)[CPT])
{
    constexpr int SEG = CPT + 2 * RA;
    constexpr int NG = group_count<P, R>();
    float D[NG][CPT];
    bool seen[NG];  // a group's sum starts from its first difference (known once the loops unroll)
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        seen[g] = false;
#pragma unroll
        for (int k = 0; k < CPT; ++k) D[g][k] = 0.0f;
    }
    {
        float m0[SEG];
        ld_seg<SEG>(s - RA, m0);
#pragma unroll
        for (int dc = 1; dc <= R; ++dc) {
            constexpr int dr = 0;
            const int g = group_of<P, R>(dc, dr);
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const float d = __fsub_rn(m0[k + RA + dc], m0[k + RA - dc]);
                D[g][k] = seen[g] ? __fadd_rn(D[g][k], d) : d;
            }
            seen[g] = true;
        }
    }
#pragma unroll
    for (int dr = 1; dr <= R; ++dr) {
        if constexpr (P == STAR) {
            float up[CPT], dn[CPT];
            ld_seg<CPT>(s + dr * ld, up);
            ld_seg<CPT>(s - dr * ld, dn);
            const int g = group_of<P, R>(0, dr);
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const float d = __fsub_rn(up[k], dn[k]);
                D[g][k] = seen[g] ? __fadd_rn(D[g][k], d) : d;
            }
            seen[g] = true;
        } else {
            float up[SEG], dn[SEG];
            ld_seg<SEG>(s + dr * ld - RA, up);
            ld_seg<SEG>(s - dr * ld - RA, dn);
#pragma unroll
            for (int dc = -R; dc <= R; ++dc) {
                const int sg = weight_sign(P, R, dc, dr);
                if (sg != 0) {
                    const int g = group_of<P, R>(dc, dr);
#pragma unroll
                    for (int k = 0; k < CPT; ++k) {
                        const float d = __fsub_rn(up[k + RA + dc], dn[k + RA - dc]);
                        if (seen[g])
                            D[g][k] = sg > 0 ? __fadd_rn(D[g][k], d) : __fsub_rn(D[g][k], d);
                        else
                            D[g][k] = sg > 0 ? d : -d;
                    }
                    seen[g] = true;
                }
            }
        }
    }
    // S = sum over groups of c_g * D_g: products with split weights and their errors through FMA,
    // the sum through TwoSum, giving (hi, lo)
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const double w = group_weight<P, R>(g);
        const float wh = split_hi(w), wl = split_lo(w);
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const float p = __fmul_rn(wh, D[g][k]);
            float pe = __fmaf_rn(wh, D[g][k], -p);
            pe = __fmaf_rn(wl, D[g][k], pe);
            if (g == 0) {
                sh[k] = p;
                sl[k] = pe;
            } else {
                float t, e;
                two_sum(sh[k], p, t, e);
                sh[k] = t;
                sl[k] = __fadd_rn(sl[k], __fadd_rn(e, pe));
            }
        }
    }
}

// The same sums with one compensated product per tap (fp32c_point's terms, row by row so that every
// row segment is read once as vectors): each tap's difference enters with its own product, so no
// difference is rounded twice.
template <int P, int R, int CPT, int RA>
__device__ __forceinline__ void fp32c_taps(const float* s, int ld, float (&sh)[CPT], float (&sl)[CPT])
{
    constexpr int SEG = CPT + 2 * RA;
    bool first = true;  // known once the loops unroll
    auto tap = [&](double w, const float (&d)[CPT]) {
        const float wh = split_hi(w), wl = split_lo(w);
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const float p = __fmul_rn(wh, d[k]);
            float pe = __fmaf_rn(wh, d[k], -p);
            pe = __fmaf_rn(wl, d[k], pe);
            if (first) {
                sh[k] = p;
                sl[k] = pe;
            } else {
                float t, e;
                two_sum(sh[k], p, t, e);
                sh[k] = t;
                sl[k] = __fadd_rn(sl[k], __fadd_rn(e, pe));
            }
        }
        first = false;
    };
    {
        float m0[SEG];
        ld_seg<SEG>(s - RA, m0);
#pragma unroll
        for (int dc = 1; dc <= R; ++dc) {
            float d[CPT];
#pragma unroll
            for (int k = 0; k < CPT; ++k) d[k] = __fsub_rn(m0[k + RA + dc], m0[k + RA - dc]);
            tap(weight(P, R, dc, 0), d);
        }
    }
#pragma unroll
    for (int dr = 1; dr <= R; ++dr) {
        constexpr int PAD = P == STAR ? 0 : RA;
        float up[CPT + 2 * PAD], dn[CPT + 2 * PAD];
        ld_seg<CPT + 2 * PAD>(s + dr * ld - PAD, up);
        ld_seg<CPT + 2 * PAD>(s - dr * ld - PAD, dn);
#pragma unroll
        for (int dc = P == STAR ? 0 : -R; dc <= (P == STAR ? 0 : R); ++dc) {
            const double w = weight(P, R, dc, dr);
            if (w != 0.0) {
                float d[CPT];
#pragma unroll
                for (int k = 0; k < CPT; ++k) d[k] = __fsub_rn(up[k + PAD + dc], dn[k + PAD - dc]);
                tap(w, d);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// FP32C, the integer route. Every PRK weight is +-1/den, so with M the common denominator of a
// stencil M * S is a sum of integer coefficients times values. On a tile of whole numbers within B of
// one another that sum is an integer small enough for FP32 arithmetic to be exact in any order, so the
// taps cost one FMA each and the division by M, with its remainder, comes once, after every application
// of the launch has been summed: no TwoSum and no split-weight products per group and application, and
// a smaller error (one division's). The tile holds u = in - ref, ref a value of the tile, to keep the
// partial sums small; in += 1 advances u. A thread's rows share every row segment it reads.
// Bound by the FMA pipe (grid R >= 3) and by shared memory (about 28 bytes per point and application);
// the group sums were bound by FP32 issue (star R=4, eight applications: FMA pipe 68%, issue 78%). At
// n=8192, us per application of whole runs of 16, group sums and this route: star R=2 87 and 48, star R=4
// 138 and 61, star R=5 171 and 78, grid R=3 262 and 98, grid R=5 502 and 227; one application, grid R=5 589
// and 374. Tiles off the route run as fast as without it (their loops share no registers with it).

__host__ __device__ constexpr int gcd_of(int a, int b) { return b == 0 ? a : gcd_of(b, a % b); }

// Common denominator M of the weights.
template <int P, int R>
__host__ __device__ constexpr int common_den()
{
    int m = 1;
    for (int dc = -R; dc <= R; ++dc)
        for (int dr = -R; dr <= R; ++dr) {
            const int d = weight_den(P, R, dc, dr);
            if (d != 0) m = m / gcd_of(m, d) * d;
        }
    return m;
}

// M * weight of every tap, c[R + dr][R + dc]. A table made at compile time: evaluated per tap in the
// unrolled loops, the weights' divisions stayed in the code of some stencils.
template <int P, int R>
struct IntCoefs {
    int c[2 * R + 1][2 * R + 1];
    int l1;
};

template <int P, int R>
__host__ __device__ constexpr IntCoefs<P, R> make_int_coefs()
{
    IntCoefs<P, R> t{};
    for (int dc = -R; dc <= R; ++dc)
        for (int dr = -R; dr <= R; ++dr) {
            const int d = weight_den(P, R, dc, dr);
            if (d == 0) continue;
            t.c[R + dr][R + dc] = weight_sign(P, R, dc, dr) * (common_den<P, R>() / d);
            t.l1 += common_den<P, R>() / d;
        }
    return t;
}

// Range of the tile's values, |u| < B at the launch's first application: 128, which a PRK field's tiles
// keep (their values lie within 110 of the middle one), or the stencil's largest.
constexpr int INT_NEAR = 128;

template <int P, int R>
__host__ __device__ constexpr int int_wide()
{
    int b = INT_NEAR;
    while (b < (1 << 17) && static_cast<int64_t>(8) * b * make_int_coefs<P, R>().l1 < (1 << 24)) b *= 2;
    return b;
}

// Applications whose sums one FP32 accumulator takes, and applications a launch may make on the route.
// An application's M * S is at most L1 (B - 1) (its taps in pairs of opposite weight, each difference at
// most 2 (B - 1)); while it forms, its partial sums reach L1 (B + t) for |u| < B + t. Together they stay
// below 2^24 for SUMS applications in a row and STEPS in all, and the sum over STEPS below 2^31.
template <int P, int R, int B>
struct IntBound {
    static constexpr int64_t L1 = make_int_coefs<P, R>().l1, LIMIT = (1 << 24) - 1;
    static constexpr int64_t MAX_S = L1 * (B - 1);
    static constexpr int64_t SUMS0 = LIMIT / 2 / MAX_S + 1;
    static constexpr int SUMS = static_cast<int>(SUMS0 > 16 ? 16 : SUMS0);
    static constexpr int64_t STEPS0 = (LIMIT - (SUMS - 1) * MAX_S) / L1 - B;
    static constexpr int64_t STEPS1 = ((1ll << 31) - 1) / MAX_S;
    static constexpr int STEPS = static_cast<int>(STEPS0 < STEPS1 ? STEPS0 : STEPS1);
    static_assert(SUMS >= 1 && STEPS >= INT_NEAR && STEPS + B < (1 << 23),
                  "integer route bounds");
};

// Launches that try the integer route: all on the TMA tiles (PLAIN false), where one fused application is
// bound by HBM on either route and grid R >= 3 gains (n=8192, grid R=4: 373 to 300 us). On the plain-staged
// and batched tiles one application of the others keeps the group sums, which cost it no check (n=8189, star
// R=1: 274 us, 307 with the check), and so do the batched launches of two, four and eight of the stencils
// with power-of-two weights (32 grids of star R=1, 2 and grid R=1 in twos: 791 against 954 us), whose group
// sums of whole numbers are exact as well. Where the exact sum is no FP32 pair the last bits differ between
// the routes, so there they may depend on the depth.
template <int P, int R, int DT, int STEPS, bool PLAIN>
__host__ __device__ constexpr bool int_route()
{
    return DT == FP32C && (!PLAIN || (STEPS > 0 ? (STEPS == 1 ? P == GRID && R >= 3 : !pow2_weights(P, R)) : true));
}

// Whether a staged FP32C tile takes the integer route, and its ref: checked while it was staged by plain
// loads (known), or to be checked in the evaluation. sums: IntBound::SUMS of its range, 0 off the route.
struct IntTile {
    bool known = false;
    int sums = 0;
    float ref = 0.0f;
};

// |x| < 2^22 and whole.
__device__ __forceinline__ bool whole_f32(float x) { return __fsub_rn(__fadd_rn(x, 12582912.0f), 12582912.0f) == x; }

// The tile's values: in whole, and the largest |u|, u = in - ref. Asked of in, not of u: the difference of
// a small value and a whole ref rounds to a whole number. With ref whole and in below 2^22, u is exact.
struct IntCheck {
    bool whole = true;
    float most = 0.0f;
    // Whether three of the tile's values let it take the route, asked before all of them are: a tile of reals
    // or of whole numbers far apart then does without the check and its vote.
    template <int P, int R>
    static __device__ __forceinline__ bool hopeful(float ref, float v, float w)
    {
        const float far = fmaxf(fabsf(__fsub_rn(v, ref)), fabsf(__fsub_rn(w, ref)));
        return whole_f32(ref) && whole_f32(v) && whole_f32(w) && far < static_cast<float>(int_wide<P, R>());
    }
    __device__ __forceinline__ void add(float v, float u)
    {
        whole = whole && whole_f32(v);
        most = fmaxf(most, fabsf(u));
    }
    // The block's verdict (a barrier, or two where the values are not near): IntTile::sums.
    template <int P, int R>
    __device__ __forceinline__ int sums(float ref, int nsteps) const
    {
        using Near = IntBound<P, R, INT_NEAR>;
        using Wide = IntBound<P, R, int_wide<P, R>()>;
        // |in| < |ref| + 2^17 <= 2^22 where |u| < B, as whole_f32 needs; in + steps stays below 2^24
        static_assert(int_wide<P, R>() <= (1 << 17), "in below 2^22");
        const bool ok = whole && fabsf(ref) <= 4194304.0f - 131072.0f && rintf(ref) == ref;
        if (__syncthreads_and(ok && most < static_cast<float>(INT_NEAR) && nsteps <= Near::STEPS)) return Near::SUMS;
        if (int_wide<P, R>() > INT_NEAR &&
            __syncthreads_and(ok && most < static_cast<float>(int_wide<P, R>()) && nsteps <= Wide::STEPS))
            return Wide::SUMS;
        return 0;
    }
};

// S[rr][k] += M * S of the thread's CPT points of ROWS consecutive rows; u points at (r0, c0) of the tile.
// Row by row of the tile: each row segment is read once and enters every output row it is a tap of. own
// (when given) gets the values of the thread's points.
template <int P, int R, int CPT, int ROWS, int RA>
__device__ __forceinline__ void int_rows(const float* u, int ld, float (&S)[ROWS][CPT], float (*own)[CPT] = nullptr)
{
    constexpr IntCoefs<P, R> C = make_int_coefs<P, R>();
#pragma unroll
    for (int q = -R; q < ROWS + R; ++q) {
        auto taps = [&](auto pad, const auto& seg) {
            constexpr int PAD = decltype(pad)::value;
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                const int dr = q - rr;
#pragma unroll
                for (int dc = -PAD; dc <= PAD; ++dc) {
                    const int c = dr >= -R && dr <= R && dc >= -R && dc <= R ? C.c[R + dr][R + dc] : 0;
                    if (c != 0) {
#pragma unroll
                        for (int k = 0; k < CPT; ++k)
                            S[rr][k] = __fmaf_rn(static_cast<float>(c), seg[k + PAD + dc], S[rr][k]);
                    }
                }
            }
        };
        if (P == GRID || (q >= 0 && q < ROWS)) {
            float seg[CPT + 2 * RA];
            ld_seg<CPT + 2 * RA>(u + q * ld - RA, seg);
            if (own && q >= 0 && q < ROWS) {
#pragma unroll
                for (int k = 0; k < CPT; ++k) own[q][k] = seg[k + RA];
            }
            taps(std::integral_constant<int, RA>{}, seg);
        } else {  // star: a row above or below the thread's is a vertical tap only
            float seg[CPT];
            ld_seg<CPT>(u + q * ld, seg);
            taps(std::integral_constant<int, 0>{}, seg);
        }
    }
}

// (o_hi, o_lo) += (t + tl) / M, renormalised, for whole t and tl (t a float's 24 bits, |tl| far smaller):
// q = t / M rounded (one correction of t * (1 / M)), the remainder t - q M exact (a small multiple of q's
// last bit), and the remainder's share of the quotient as the low word. Exact where M divides t, as it
// does for a PRK field; within 2^-46.9 of the quotient otherwise.
template <int P, int R>
__device__ __forceinline__ void int_add(uint64_t& o, float t, float tl)
{
    constexpr int M = common_den<P, R>();
    constexpr float INV = static_cast<float>(1.0 / M);
    const float q0 = __fmul_rn(t, INV);
    const float q = __fmaf_rn(__fmaf_rn(-q0, static_cast<float>(M), t), INV, q0);
    const float rem = __fmaf_rn(-q, static_cast<float>(M), t);
    float oh = __uint_as_float(static_cast<uint32_t>(o)), ol = __uint_as_float(static_cast<uint32_t>(o >> 32));
    df_add(oh, ol, q, __fmul_rn(__fadd_rn(rem, tl), INV));
    o = static_cast<uint64_t>(__float_as_uint(oh)) | (static_cast<uint64_t>(__float_as_uint(ol)) << 32);
}

// ---------------------------------------------------------------------------------------------
// FP64 exact route: integer coefficients c = w * 2^shift of a power-of-two stencil.

template <int P, int R>
__device__ __forceinline__ constexpr int coef(int dc, int dr)
{
    const int d = weight_den(P, R, dc, dr);
    return d == 0 ? 0 : weight_sign(P, R, dc, dr) * ((1 << pow2_shift(P, R)) / d);
}

// sum of c * (V[p+d] - V[p-d]) over the positive taps for CPT points of a row; v points at V(r, c0).
template <int P, int R, int CPT, int RA, typename I>
__device__ __forceinline__ void fx_points(const int64_t* v, int ld, I (&S)[CPT])
{
    constexpr int SEG = CPT + 2 * RA;
#pragma unroll
    for (int k = 0; k < CPT; ++k) S[k] = 0;
    {
        I m0[SEG];
        ld_seg_i<SEG>(v - RA, m0);
#pragma unroll
        for (int dc = 1; dc <= R; ++dc) {
            const int cc = coef<P, R>(dc, 0);
#pragma unroll
            for (int k = 0; k < CPT; ++k) S[k] += static_cast<I>(cc) * (m0[k + RA + dc] - m0[k + RA - dc]);
        }
    }
#pragma unroll
    for (int dr = 1; dr <= R; ++dr) {
        if constexpr (P == STAR) {
            I up[CPT], dn[CPT];
            ld_seg_i<CPT>(v + dr * ld, up);
            ld_seg_i<CPT>(v - dr * ld, dn);
            const int cc = coef<P, R>(0, dr);
#pragma unroll
            for (int k = 0; k < CPT; ++k) S[k] += static_cast<I>(cc) * (up[k] - dn[k]);
        } else {
            I up[SEG], dn[SEG];
            ld_seg_i<SEG>(v + dr * ld - RA, up);
            ld_seg_i<SEG>(v - dr * ld - RA, dn);
#pragma unroll
            for (int dc = -R; dc <= R; ++dc) {
                const int cc = coef<P, R>(dc, dr);
                if (cc != 0) {
#pragma unroll
                    for (int k = 0; k < CPT; ++k) S[k] += static_cast<I>(cc) * (up[k + RA + dc] - dn[k + RA - dc]);
                }
            }
        }
    }
}

// N consecutive floats from 8-byte-aligned shared memory (float2 loads).
template <int N>
__device__ __forceinline__ void ld_seg2(const float* p, float (&v)[N])
{
    static_assert(N % 2 == 0, "segment is whole float2 vectors");
#pragma unroll
    for (int q = 0; q < N / 2; ++q) {
        const float2 t = reinterpret_cast<const float2*>(p)[q];
        v[2 * q] = t.x;
        v[2 * q + 1] = t.y;
    }
}

// The integer route in FP32: every value of the tile is an integer below 2^20, so the differences,
// the products by the small integer coefficients and every partial sum are integers below 2^24 and
// FP32 arithmetic is exact. Sum of c * (V[p+d] - V[p-d]) for CPT points; v points at V(r, c0).
template <int P, int R, int CPT, int RA>
__device__ __forceinline__ void fexact_points(const float* v, int ld, float (&S)[CPT])
{
    constexpr int SEG = CPT + 2 * RA;
#pragma unroll
    for (int k = 0; k < CPT; ++k) S[k] = 0.0f;
    {
        float m0[SEG];
        ld_seg2<SEG>(v - RA, m0);
#pragma unroll
        for (int dc = 1; dc <= R; ++dc) {
            const float cc = static_cast<float>(coef<P, R>(dc, 0));
#pragma unroll
            for (int k = 0; k < CPT; ++k) S[k] = __fmaf_rn(cc, __fsub_rn(m0[k + RA + dc], m0[k + RA - dc]), S[k]);
        }
    }
#pragma unroll
    for (int dr = 1; dr <= R; ++dr) {
        if constexpr (P == STAR) {
            float up[CPT], dn[CPT];
            ld_seg2<CPT>(v + dr * ld, up);
            ld_seg2<CPT>(v - dr * ld, dn);
            const float cc = static_cast<float>(coef<P, R>(0, dr));
#pragma unroll
            for (int k = 0; k < CPT; ++k) S[k] = __fmaf_rn(cc, __fsub_rn(up[k], dn[k]), S[k]);
        } else {
            float up[SEG], dn[SEG];
            ld_seg2<SEG>(v + dr * ld - RA, up);
            ld_seg2<SEG>(v - dr * ld - RA, dn);
#pragma unroll
            for (int dc = -R; dc <= R; ++dc) {
                const int c = coef<P, R>(dc, dr);
                if (c != 0) {
#pragma unroll
                    for (int k = 0; k < CPT; ++k)
                        S[k] = __fmaf_rn(static_cast<float>(c), __fsub_rn(up[k + RA + dc], dn[k + RA - dc]), S[k]);
                }
            }
        }
    }
}

// fexact_points for the ROWS consecutive rows of a thread at once: S[rr] for the CPT points of row
// r0 + rr, v pointing at V(r0, c0); own[rr] gets the values of those points. Every row segment
// (star: every column strip) is read from shared memory once and serves every row it is a tap of.
// The arithmetic is exact, so the order of the terms does not matter.
template <int P, int R, int CPT, int ROWS, int RA>
__device__ __forceinline__ void fexact_rows(const float* v, int ld, float (&S)[ROWS][CPT], float (&own)[ROWS][CPT])
{
    constexpr int SEG = CPT + 2 * RA;
    constexpr int NR = ROWS + 2 * R;  // rows r0 - R .. r0 + ROWS - 1 + R
    if constexpr (P == STAR) {
        float col[NR][CPT];
#pragma unroll
        for (int q = 0; q < NR; ++q)
            if (q < R || q >= R + ROWS) ld_seg2<CPT>(v + (q - R) * ld, col[q]);
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            float m[SEG];
            ld_seg2<SEG>(v + rr * ld - RA, m);
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                col[rr + R][k] = m[k + RA];
                own[rr][k] = m[k + RA];
                S[rr][k] = 0.0f;
            }
#pragma unroll
            for (int dc = 1; dc <= R; ++dc) {
                const float cc = static_cast<float>(coef<P, R>(dc, 0));
#pragma unroll
                for (int k = 0; k < CPT; ++k)
                    S[rr][k] = __fmaf_rn(cc, __fsub_rn(m[k + RA + dc], m[k + RA - dc]), S[rr][k]);
            }
        }
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr)
#pragma unroll
            for (int dr = 1; dr <= R; ++dr) {
                const float cc = static_cast<float>(coef<P, R>(0, dr));
#pragma unroll
                for (int k = 0; k < CPT; ++k)
                    S[rr][k] = __fmaf_rn(cc, __fsub_rn(col[rr + R + dr][k], col[rr + R - dr][k]), S[rr][k]);
            }
    } else {
        float seg[NR][SEG];
#pragma unroll
        for (int q = 0; q < NR; ++q) ld_seg2<SEG>(v + (q - R) * ld - RA, seg[q]);
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                S[rr][k] = 0.0f;
                own[rr][k] = seg[rr + R][k + RA];
            }
#pragma unroll
            for (int dr = 0; dr <= R; ++dr)
#pragma unroll
                for (int dc = -R; dc <= R; ++dc) {
                    if (dr == 0 && dc <= 0) continue;
                    const int c = coef<P, R>(dc, dr);
                    if (c != 0) {
#pragma unroll
                        for (int k = 0; k < CPT; ++k)
                            S[rr][k] = __fmaf_rn(static_cast<float>(c),
                                                 __fsub_rn(seg[rr + R + dr][k + RA + dc], seg[rr + R - dr][k + RA - dc]),
                                                 S[rr][k]);
                    }
                }
        }
    }
}

// binary64 encoding of f * 2^adj for an integer-valued f (|f| < 2^24): exponent rebias and a
// mantissa shift, no conversion instruction (those run on the binary64 pipe).
__device__ __forceinline__ uint64_t f2d(float f, int adj)
{
    const uint32_t u = __float_as_uint(f);
    const uint64_t mag = u & 0x7FFFFFFFu;
    const uint64_t d = (static_cast<uint64_t>(u & 0x80000000u) << 32) |
                       ((mag + (static_cast<uint64_t>(896 + adj) << 23)) << 29);
    return mag == 0 ? 0ull : d;
}

// binary64 encoding of x * 2^unit for a 32-bit x (exact).
__device__ __forceinline__ uint64_t from_fixed32(int32_t x, int unit)
{
    if (x == 0) return 0;
    const uint64_t s = x < 0 ? fx::SIGN : 0;
    const uint32_t a = x < 0 ? static_cast<uint32_t>(-x) : static_cast<uint32_t>(x);
    const int msb = 31 - __clz(a);
    const uint64_t m = static_cast<uint64_t>(a) << (52 - msb);
    return s | ((static_cast<uint64_t>(msb + unit + 1022) << 52) + m);
}

// binary64 encoding of a whole number |v| < 2^22, through the float it is exactly: a magic number's
// mantissa takes the integer and one FP32 subtraction normalises it, where from_fixed32 searches for
// the leading bit and shifts 64 bits.
__device__ __forceinline__ uint64_t whole_bits(int32_t v)
{
    return f2d(__fsub_rn(__uint_as_float(0x4B400000u + static_cast<uint32_t>(v)), 12582912.0f), 0);
}

// out = V * 2^-shift for an integer V with |V| < 2^21, read from the binary64 encoding (+-0 give 0);
// false for any other value. With M the 53-bit significand, V = M >> (k + 32) for
// k = 1043 - shift - (biased exponent), an integer below 2^21 exactly when 0 <= k <= 20 and the
// k + 32 bits shifted out are zero. Subnormals, infinities and NaNs fall outside that range of k.
__device__ __forceinline__ bool out_units(uint64_t b, int shift, int32_t& V)
{
    const uint32_t hi = static_cast<uint32_t>(b >> 32), lo = static_cast<uint32_t>(b);
    const uint32_t mag = hi & 0x7FFFFFFFu;
    const int k = 1043 - shift - static_cast<int>(mag >> 20);
    const uint32_t m = (mag & 0xFFFFFu) | 0x100000u;
    const bool zero = (mag | lo) == 0u;
    const bool ok = zero || (lo == 0u && k >= 0 && k <= 20 && (m & ((1u << (k & 31)) - 1u)) == 0u);
    const int32_t a = static_cast<int32_t>(m >> (k & 31));
    V = zero ? 0 : ((hi >> 31) ? -a : a);
    return ok;
}

__device__ __forceinline__ double as_dbl(uint64_t b) { return __longlong_as_double(static_cast<long long>(b)); }
__device__ __forceinline__ uint64_t as_bits(double d) { return static_cast<uint64_t>(__double_as_longlong(d)); }

// in += 1 over the whole staged tile, halo included, as 16-byte vectors (the tile starts at the
// 128-byte aligned stage and its element count is a multiple of four): FP32 values (the FP32 route
// and FP32C), integers in fixed-point units (one = 1.0 in those units) or binary64 values.
template <int ELEMS>
__device__ __forceinline__ void advance_f32(float* p)
{
    constexpr int NV = ELEMS / 4;
#pragma unroll
    for (int q = 0; q < (NV + THREADS - 1) / THREADS; ++q) {
        const int idx = threadIdx.x + q * THREADS;
        if (NV % THREADS == 0 || idx < NV) {
            float4 v = reinterpret_cast<float4*>(p)[idx];
            v.x = __fadd_rn(v.x, 1.0f);
            v.y = __fadd_rn(v.y, 1.0f);
            v.z = __fadd_rn(v.z, 1.0f);
            v.w = __fadd_rn(v.w, 1.0f);
            reinterpret_cast<float4*>(p)[idx] = v;
        }
    }
}

// dst = src + 1 over the halo of a staged FP32 tile only (the R rows above and below, the RA
// columns either side): the interior points are advanced by the threads that own them. Rows as
// 16-byte vectors, side columns as 8-byte pairs.
template <int SW, int SH, int R, int RA>
__device__ __forceinline__ void advance_halo_f32(const float* src, float* dst)
{
    static_assert(SW % 4 == 0 && RA % 2 == 0, "halo vectors");
    constexpr int ROWV = SW / 4;               // 16-byte vectors in a row
    constexpr int NROW = 2 * R * ROWV;         // top and bottom halo rows
    constexpr int PER_SIDE = RA / 2;           // 8-byte pairs per side of a row
    constexpr int NSIDE = (SH - 2 * R) * 2 * PER_SIDE;
#pragma unroll
    for (int q = 0; q < (NROW + NSIDE + THREADS - 1) / THREADS; ++q) {
        const int h = threadIdx.x + q * THREADS;
        if (h < NROW) {
            const int r = h / ROWV, v = h - r * ROWV;
            const int row = r < R ? r : SH - 2 * R + r;  // rows 0..R-1, then SH-R..SH-1
            float4 x = reinterpret_cast<const float4*>(src + row * SW)[v];
            x.x = __fadd_rn(x.x, 1.0f);
            x.y = __fadd_rn(x.y, 1.0f);
            x.z = __fadd_rn(x.z, 1.0f);
            x.w = __fadd_rn(x.w, 1.0f);
            reinterpret_cast<float4*>(dst + row * SW)[v] = x;
        } else if (h < NROW + NSIDE) {
            const int i = h - NROW;
            const int row = R + i / (2 * PER_SIDE), p = i - (i / (2 * PER_SIDE)) * (2 * PER_SIDE);
            const int col = p < PER_SIDE ? 2 * p : SW - RA + 2 * (p - PER_SIDE);
            float2 x = *reinterpret_cast<const float2*>(src + row * SW + col);
            x.x = __fadd_rn(x.x, 1.0f);
            x.y = __fadd_rn(x.y, 1.0f);
            *reinterpret_cast<float2*>(dst + row * SW + col) = x;
        }
    }
}

template <int ELEMS>
__device__ __forceinline__ void advance_i64(int64_t* p, int64_t one)
{
    constexpr int NV = ELEMS / 2;
#pragma unroll
    for (int q = 0; q < (NV + THREADS - 1) / THREADS; ++q) {
        const int idx = threadIdx.x + q * THREADS;
        if (NV % THREADS == 0 || idx < NV) {
            longlong2 v = reinterpret_cast<longlong2*>(p)[idx];
            v.x += one;
            v.y += one;
            reinterpret_cast<longlong2*>(p)[idx] = v;
        }
    }
}

template <int ELEMS>
__device__ __forceinline__ void advance_f64(double* p)
{
    constexpr int NV = ELEMS / 2;
#pragma unroll
    for (int q = 0; q < (NV + THREADS - 1) / THREADS; ++q) {
        const int idx = threadIdx.x + q * THREADS;
        if (NV % THREADS == 0 || idx < NV) {
            double2 v = reinterpret_cast<double2*>(p)[idx];
            v.x = inc_exact(v.x);
            v.y = inc_exact(v.y);
            reinterpret_cast<double2*>(p)[idx] = v;
        }
    }
}

// binary64 encoding of a constexpr double (normal or zero), by exact scaling by powers of two
// (C++17 has no bit_cast in constant expressions).
__host__ __device__ constexpr uint64_t encode(double w)
{
    if (w == 0.0) return 0;
    uint64_t sign = 0;
    if (w < 0) {
        sign = fx::SIGN;
        w = -w;
    }
    int e = 0;
    while (w >= 2.0) {
        w /= 2.0;
        ++e;
    }
    while (w < 1.0) {
        w *= 2.0;
        --e;
    }
    const uint64_t frac = static_cast<uint64_t>((w - 1.0) * 4503599627370496.0);  // exact: 52 bits
    return sign | (static_cast<uint64_t>(e + 1023) << 52) | frac;
}
static_assert(encode(1.0) == 0x3FF0000000000000ull && encode(-0.125) == 0xBFC0000000000000ull &&
                  encode(1.0 / 6.0) == 0x3FC5555555555555ull,
              "constexpr binary64 encoding");

// The taps of a stencil in the generator's order (column offset outer, row offset inner, zero
// weights left out), with their offsets in a tile of row length LD and their weights split for
// fx::mul_whole20_split: the significand's low 32 bits, its high 21 bits with the hidden bit, and
// the sign and exponent field of the encoding's high word. One 16-byte entry per tap.
template <int P, int R, int LD>
struct TapTable {
    struct alignas(16) Tap {
        int off;
        uint32_t w1, w2, hib;
    } tap[tap_count(P, R)];
};

template <int P, int R, int LD>
constexpr TapTable<P, R, LD> make_taps()
{
    TapTable<P, R, LD> t{};
    int k = 0;
    for (int dc = -R; dc <= R; ++dc)
        for (int dr = -R; dr <= R; ++dr) {
            const double w = weight(P, R, dc, dr);
            if (w != 0.0) {
                const uint64_t wb = encode(w);
                t.tap[k].off = dr * LD + dc;
                t.tap[k].w1 = static_cast<uint32_t>(wb);
                t.tap[k].w2 = static_cast<uint32_t>((wb >> 32) & 0xFFFFFu) | 0x100000u;
                t.tap[k].hib = static_cast<uint32_t>(wb >> 32) & 0xFFF00000u;
                ++k;
            }
        }
    return t;
}

template <int P, int R, int LD>
__constant__ TapTable<P, R, LD> c_taps = make_taps<P, R, LD>();

// fp64_point for CPT adjacent points of a tile of whole numbers |v| < 2^20 held as int32: every
// product comes from fx::mul_whole20_split on the integer pipes (the same bits as __dmul_rn), every sum is
// the same binary64 add in the same order, so the binary64 pipe issues one instruction per tap
// instead of two. The taps come from constant memory in a loop, which keeps the code small.
template <int P, int R, int LD, int CPT>
__device__ __forceinline__ void fp64_points_whole(const int32_t* s, double (&acc)[CPT])
{
    constexpr int N = tap_count(P, R);
    const auto& T = c_taps<P, R, LD>;
    {
        const auto tp = T.tap[0];
#pragma unroll
        for (int k = 0; k < CPT; ++k)
            acc[k] = __longlong_as_double(
                static_cast<long long>(fx::mul_whole20_split(tp.w1, tp.w2, tp.hib, s[tp.off + k])));
    }
#pragma unroll 2
    for (int t = 1; t < N; ++t) {
        const auto tp = T.tap[t];
#pragma unroll
        for (int k = 0; k < CPT; ++k)
            acc[k] = __dadd_rn(acc[k], __longlong_as_double(static_cast<long long>(
                                           fx::mul_whole20_split(tp.w1, tp.w2, tp.hib, s[tp.off + k]))));
    }
}

// The reference's chain with binary64 instructions throughout, for two adjacent points: the tiles no other
// route takes (subnormals, infinities, NaNs and values near the ends of the exponent range). Bound by the
// binary64 pipe and unrolled, so that the two points share the products of the values that they weigh alike
// (as a loop over the taps, n=4096, one application: grid R=2 1332 us against 1221, grid R=5 7122 against
// 6364).
template <int P, int R, int LD>
__device__ __forceinline__ double2 fp64_pair_strict(const double* s)
{
    return make_double2(fp64_point<P, R>(s, LD), fp64_point<P, R>(s + 1, LD));
}

// in += 1 over a staged tile of int32 whole numbers, as 16-byte vectors.
template <int ELEMS>
__device__ __forceinline__ void advance_i32(int32_t* p)
{
    constexpr int NV = ELEMS / 4;
#pragma unroll
    for (int q = 0; q < (NV + THREADS - 1) / THREADS; ++q) {
        const int idx = threadIdx.x + q * THREADS;
        if (NV % THREADS == 0 || idx < NV) {
            int4 v = reinterpret_cast<int4*>(p)[idx];
            v.x += 1;
            v.y += 1;
            v.z += 1;
            v.w += 1;
            reinterpret_cast<int4*>(p)[idx] = v;
        }
    }
}

// Where process_tile finds `out`: the out tile loaded into shared memory next to `in` (TMA path), or
// HBM, read in the evaluation row by row (batched path) or with every row's words requested before
// the first row is evaluated (plain-staged path; used for the FP64 power-of-two stencils at one
// application, where it measured faster, and like OUT_HBM otherwise).
constexpr int OUT_SMEM = 0, OUT_HBM = 1, OUT_HBM_AHEAD = 2;

// ---------------------------------------------------------------------------------------------
// FP64 stencils whose weights are not powers of two, on whole-number tiles of small range: the
// table route.
//
// Every product and every partial sum of the reference's chain rounds, and GB300 issues binary64
// adds at a small fraction of its integer rate, so the route moves work off the binary64 pipe
// without changing a bit:
//  - Products from a table. A tile whose values all lie in [base, base + TBL_L) takes each product
//    fl(|w| * v) from a shared-memory table of every weight group and every such v, built once per
//    tile with fx::mul_whole20 (the weight's sign enters as an add or a subtract). Every tap still
//    reads its own in value, and indexes the table with it.
//  - Most adds of each point's chain run in fixed point on the integer pipes, the exact sum rounded to
//    53 bits, nearest-even: the binary64 add's result bit for bit on these values. In 64 bits where a
//    window's values allow it (the narrow form), else in 96 (fx::fx96_acc_round). The rest, and the add
//    into out, run on the binary64 pipe.
// Lane l evaluates columns l and l + 32 of its warp's rows, so a warp's table reads are consecutive
// entries; the results go into the shared-memory out tile, which the stores then read in their own
// layout. Applications of a multi-application launch write in + 1 to the other half of the stage
// (the int32 tile takes half of it), and the tables are rebuilt at a new base when the values outgrow
// them.

constexpr int TBL_L = 128;  // consecutive values one product table covers

// The tables follow the TMA kernel's own shared memory (16-byte aligned).
template <int DT, int R, int TH_>
__host__ __device__ constexpr int table_offset()
{
    return (Geo<DT, R, TH_>::SMEM + 15) / 16 * 16;
}

template <int P, int R>
struct StrictTaps {
    int dc[tap_count(P, R)], dr[tap_count(P, R)], g[tap_count(P, R)], neg[tap_count(P, R)];
};

// The taps in the generator's order (column offset outer, row offset inner, zeros left out), each
// with its weight group and sign.
template <int P, int R>
constexpr StrictTaps<P, R> make_strict_taps()
{
    StrictTaps<P, R> t{};
    int k = 0;
    for (int dc = -R; dc <= R; ++dc)
        for (int dr = -R; dr <= R; ++dr) {
            const double w = weight(P, R, dc, dr);
            if (w != 0.0) {
                t.dc[k] = dc;
                t.dr[k] = dr;
                t.g[k] = group_of<P, R>(dc, dr);
                t.neg[k] = w < 0.0 ? 1 : 0;
                ++k;
            }
        }
    return t;
}

// Every tap's |weight| is its group's (checked for the stencils the route serves).
template <int P, int R>
constexpr bool strict_taps_ok()
{
    constexpr StrictTaps<P, R> t = make_strict_taps<P, R>();
    for (int k = 0; k < tap_count(P, R); ++k) {
        const double w = weight(P, R, t.dc[k], t.dr[k]);
        if ((w < 0.0 ? -w : w) != group_weight<P, R>(t.g[k])) return false;
    }
    return true;
}
static_assert(strict_taps_ok<STAR, 3>() && strict_taps_ok<STAR, 4>() && strict_taps_ok<STAR, 5>() &&
                  strict_taps_ok<GRID, 2>() && strict_taps_ok<GRID, 3>() && strict_taps_ok<GRID, 4>() &&
                  strict_taps_ok<GRID, 5>(),
              "strict tap groups");

// Sixteenths of each chain that run in fixed point in the 96-bit form (the rest on the binary64 pipe),
// per stencil and form (ONE: one application per launch; else several), as measured at n=16384 on tiles
// that all took this form: star R=3, 4 11/16 and R=5 12/16 at one application, 14/16 and 13/16 at
// several; grid R=2 11/16, R=3 12/16, R=4 13/16, R=5 15/16 at one, 12/16, 12/16, 14/16 and 13/16 at
// several.
template <int P, int R, bool ONE>
__host__ __device__ constexpr int fixed_sixteenths()
{
    if (P == STAR) {
        if (ONE) return R == 5 ? 12 : 11;
        return R == 3 ? 14 : 13;
    }
    if (ONE) return R == 2 ? 11 : (R == 3 ? 12 : (R == 4 ? 13 : 15));
    return R <= 3 ? 12 : (R == 4 ? 14 : 13);
}

// Taps of each chain whose adds run in fixed point (at least the first).
template <int P, int R, bool ONE>
__host__ __device__ constexpr int fixed_taps()
{
    const int k = tap_count(P, R) * fixed_sixteenths<P, R, ONE>() / 16;
    return k < 1 ? 1 : (k > tap_count(P, R) ? tap_count(P, R) : k);
}

template <int P, int R, int DT>
__host__ __device__ constexpr bool table_route()
{
    return DT == FP64 && !pow2_weights(P, R);
}

// Shared memory of the tables: per weight group TBL_L binary64 products, then TBL_L 96-bit images or
// TBL_L 64-bit images of either sign (the narrow form), then one descriptor per tap (the narrow form).
template <int P, int R, int DT>
__host__ __device__ constexpr int table_bytes()
{
    return table_route<P, R, DT>() ? group_count<P, R>() * TBL_L * (8 + 16) + tap_count(P, R) * 16 : 0;
}

// Tiles of the table route resident per SM: four where their shared memory allows it (star R=3, 4, grid
// R=2; 64 registers), else three (80).
template <int P, int R>
__host__ __device__ constexpr int strict_tiles()
{
    return 4 * (table_offset<FP64, R, 32>() + table_bytes<P, R, FP64>() + 1024) <= SMEM_PER_SM ? 4 : 3;
}

// Dynamic shared memory of the TMA kernel: its tile stages, and the tables where the route applies.
template <int P, int R, int DT, int TH_>
__host__ __device__ constexpr int tile_smem()
{
    return table_offset<DT, R, TH_>() + table_bytes<P, R, DT>();
}

// Fill the tables for the values [base, base + TBL_L): T64[g * TBL_L + u] = fl(|w_g| * (base + u))
// and T96 its fixed-point image. Values at or beyond 2^20 in magnitude (never read) get 0.
template <int P, int R>
__device__ __forceinline__ void build_tables(uint64_t* T64, uint4* T96, int base)
{
    constexpr int NG = group_count<P, R>();
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        const uint64_t wb = encode(group_weight<P, R>(g));
        for (int u = threadIdx.x; u < TBL_L; u += THREADS) {
            const int v = base + u;
            const uint64_t p = (v > -(1 << 20) && v < (1 << 20)) ? fx::mul_whole20(wb, v) : 0ull;
            uint32_t x0, x1, x2;
            fx::fx96_from_bits(p, x0, x1, x2);
            T64[g * TBL_L + u] = p;
            T96[g * TBL_L + u] = make_uint4(x0, x1, x2, 0u);
        }
    }
}

// Whether a row of the table route's tile holds points to update (row-uniform). The 96-bit form skips the
// other rows; the narrow form takes a thread's eight points together and drops those outside, and skips a
// warp's rows only where none has any.
__device__ __forceinline__ bool table_row_active(bool has_out, int64_t gi, int64_t gg, int64_t row_end, int64_t n, int R)
{
    return has_out && gi < row_end && gg >= R && gg < n - R;
}

// The narrow form of the table route: the chain in 64-bit fixed point, its rounding positions known
// per tap before the points are evaluated.
//
// In a window [base, top] of values, all of one sign, every product is a multiple of 2^L, L the lowest
// bit of the smallest one, and so is every rounded partial sum. The partial sum after tap t lies within
// W_t * mid +- A_t * half of the window's middle and half width (W_t, A_t the prefix sums of the weights
// and of their magnitudes), so
//  - where that stays below 2^62 units the sums are 64-bit integers, two words instead of three;
//  - where it stays inside one binade, as it does unless the window straddles a power of two, the
//    rounding position is the same for every point and comes from the tap's descriptor: no search for
//    the leading bit, no per-point masks. The other taps find it per point (bfind).
// Over the tiles of a PRK field at n=16384, 96% of the taps of star R=3 and 93% of grid R=5's have one
// rounding position; at n=4096 88% and 78%. Windows that hold zero, or span too many binades, take the
// 96-bit form (table_rows).
//
// A tap is a loop iteration over eight points of a thread, which share its constants and descriptor, so
// the code stays small at 110 taps; the tile holds table offsets instead of values, so a point's two
// reads need no address arithmetic between them. What bounds it (ncu, grid R=5, n=8192, four
// applications): shared memory 86% of its wavefronts (one for the offset, two for the product, per 32
// points and tap) and the integer ALU 79%, 12.3 instructions per point and tap. At n=8192, us per
// application, against the 96-bit form for every tile: one per launch, star R=3 925 to 663, grid R=2
// 1296 to 851, grid R=5 6389 to 3137; whole runs of 16, star R=3 678 to 426, grid R=5 5342 to 2894.
// Slower: two products prefetched a tap ahead (grid R=2 888 and 722 at 24 warps), indices of four rows
// packed in a word (grid R=5 3106: fewer wavefronts, more ALU instructions), the tie found through a
// carry of the lowest kept bit (7 instructions, 3088).

// Taps of each chain whose adds run in fixed point; the ones after them, at least one, run on the
// binary64 pipe beside the integer pipes. Measured at n=8192 (us per application): one application per
// launch, star one tap (R=3: 646 against 681 with two), grid R=2 two (842; 848 with one, 870 with
// three), grid R=3..5 three for each ring past the second (R=5: 3128 with nine, 3154 with twelve, 3180
// with six); several applications per launch, one (grid R=5 whole run 2901; 2939 with five).
template <int P, int R, bool ONE>
__host__ __device__ constexpr int narrow_taps()
{
    return tap_count(P, R) - (!ONE || P == STAR ? 1 : R == 2 ? 2 : 3 * (R - 2));
}

struct alignas(16) NarrowTap {
    int off;        // offset in the int32 tile
    uint32_t t64;   // byte offset of the tap's binary64 products in the tables
    uint32_t fix;   // byte offset of its signed 64-bit images
    uint32_t sign;  // 0x80000000 for a negative weight
};

template <int P, int R, int SW>
struct NarrowTaps {
    NarrowTap tap[tap_count(P, R)];
    float w[tap_count(P, R)], a[tap_count(P, R)];  // W_t and A_t
    double gw[group_count<P, R>()];                // |weight| of each group
};

template <int P, int R, int SW>
constexpr NarrowTaps<P, R, SW> make_narrow_taps()
{
    constexpr StrictTaps<P, R> s = make_strict_taps<P, R>();
    constexpr int NG = group_count<P, R>();
    NarrowTaps<P, R, SW> t{};
    double w = 0.0, a = 0.0;
    for (int k = 0; k < tap_count(P, R); ++k) {
        t.tap[k].off = s.dr[k] * SW + s.dc[k];
        t.tap[k].t64 = static_cast<uint32_t>(s.g[k] * TBL_L * 8);
        t.tap[k].fix = static_cast<uint32_t>((NG + (s.neg[k] ? NG : 0) + s.g[k]) * TBL_L * 8);
        t.tap[k].sign = s.neg[k] ? 0x80000000u : 0u;
        const double wk = weight(P, R, s.dc[k], s.dr[k]);
        w += wk;
        a += wk < 0.0 ? -wk : wk;
        t.w[k] = static_cast<float>(w);
        t.a[k] = static_cast<float>(a);
    }
    for (int g = 0; g < NG; ++g) t.gw[g] = group_weight<P, R>(g);
    return t;
}

template <int P, int R, int SW>
__constant__ NarrowTaps<P, R, SW> c_narrow = make_narrow_taps<P, R, SW>();

// Smallest weight group: its products have the lowest bits.
template <int P, int R>
__host__ __device__ constexpr double smallest_weight()
{
    double m = group_weight<P, R>(0);
    for (int g = 1; g < group_count<P, R>(); ++g)
        if (group_weight<P, R>(g) < m) m = group_weight<P, R>(g);
    return m;
}

// floor(log2 x) of a positive normal float.
__device__ __forceinline__ int log2_floor(float x) { return static_cast<int>(__float_as_uint(x) >> 23) - 127; }

// Build the narrow form's tables and descriptors for the window [base, top] (top - base < TBL_L).
// Returns false (block-uniform, through a barrier) when the window holds zero or both signs or a
// partial sum may reach 2^62 units; *unit is L otherwise. The tables are complete on return.
template <int P, int R, int SW, bool ONE>
__device__ __forceinline__ bool build_narrow(unsigned char* tbl, int base, int top, int* unit)
{
    constexpr int NG = group_count<P, R>(), KF = narrow_taps<P, R, ONE>();
    const int amin = base > 0 ? base : -top, amax = base > 0 ? top : -base;
    if (amin <= 0 || amax >= (1 << 20)) return false;
    const int L = static_cast<int>(fx::mul_whole20(encode(smallest_weight<P, R>()), amin) >> 52) - 1075;
    uint64_t* T64 = reinterpret_cast<uint64_t*>(tbl);
    const auto& T = c_narrow<P, R, SW>;
#pragma unroll 1
    for (int k = threadIdx.x; k < NG * TBL_L; k += THREADS) {
        const int v = base + k % TBL_L;
        const uint64_t p =
            v <= top ? as_bits(__dmul_rn(T.gw[k / TBL_L], as_dbl(whole_bits(v)))) : 0ull;  // v is not 0
        // p = m * 2^(e - 1075); as an integer of 2^L units m << (e - 1075 - L). The shift lies in 0..11
        // for every product of a window that passes the check below.
        const uint64_t m = (p & fx::MANT) | fx::HIDDEN;
        const int sh = min(static_cast<int>((p >> 52) & 0x7FFu) - 1075 - L, 11);
        int64_t x = p == 0 ? 0 : static_cast<int64_t>(m << (sh & 63));
        if (p & fx::SIGN) x = -x;
        T64[k] = p;
        T64[NG * TBL_L + k] = static_cast<uint64_t>(x);
        T64[2 * NG * TBL_L + k] = static_cast<uint64_t>(-x);
    }
    bool ok = true;
    uint4* desc = reinterpret_cast<uint4*>(tbl + NG * TBL_L * 24);
    for (int t = threadIdx.x; t < KF; t += THREADS) {
        // every partial sum lies in [|W mid| - r, |W mid| + r]; the slack covers the float arithmetic
        // and the roundings of the sum itself
        const float mid = 0.5f * static_cast<float>(base + top), half = 0.5f * static_cast<float>(top - base);
        const float c = fabsf(T.w[t] * mid), r = T.a[t] * (half + 1e-5f * static_cast<float>(amax));
        const int bhi = max(log2_floor(c + r) - 52 - L, 0);
        const int blo = c - r > 1e-3f ? max(log2_floor(c - r) - 52 - L, 0) : 0;
        ok = ok && log2_floor(c + r) - L < 62;
        const int b = bhi & 31;
        desc[t] = make_uint4((1u << b) >> 1, b ? 1u << b : 0u, b ? ~((2u << b) - 1u) : ~0u, bhi != blo ? 1u : 0u);
    }
    *unit = L;
    return __syncthreads_and(ok) != 0;
}

// binary64 encoding of x * 2^unit for a 64-bit x with at most 53 significant bits (0 gives +0).
__device__ __forceinline__ uint64_t fx64_to_bits(uint32_t x0, uint32_t x1, int unit)
{
    const int64_t x = static_cast<int64_t>((static_cast<uint64_t>(x1) << 32) | x0);
    if (x == 0) return 0;
    const uint64_t a = x < 0 ? static_cast<uint64_t>(-x) : static_cast<uint64_t>(x);
    const int lead = fx::clz64(a);
    return (static_cast<uint64_t>(x1 >> 31) << 63) |
           ((static_cast<uint64_t>(63 - lead + unit + 1022) << 52) + ((a << lead) >> 11));
}

// The int32 tile as byte offsets into a table of the window: 8 (v - base), and back. In place, as
// 16-byte vectors; each thread its own.
template <int ELEMS, bool TO>
__device__ __forceinline__ void offsets_tile(int32_t* p, int base)
{
    constexpr int NV = ELEMS / 4;
    auto f = [&](int v) { return TO ? (v - base) * 8 : (v >> 3) + base; };
#pragma unroll 1
    for (int idx = threadIdx.x; idx < NV; idx += THREADS) {
        int4 v = reinterpret_cast<int4*>(p)[idx];
        v.x = f(v.x);
        v.y = f(v.y);
        v.z = f(v.z);
        v.w = f(v.w);
        reinterpret_cast<int4*>(p)[idx] = v;
    }
}

// The chains of a thread's eight points: rows r, r + QR, r + 2 QR, r + 3 QR (q >> 1) of columns c and
// c + 32 (q & 1); sp points at (r, c) of the tile of table offsets. The add of tap t rounds the 64-bit sum to a
// multiple of 2^b, nearest-even, b from the descriptor (.x = 2^(b-1), .y = 2^b, .z = the bits above b; 0,
// 0 and all ones for b = 0): plus half a unit, then the bits below b cut (halves round up), and bit b
// cleared on a tie. A tie leaves zeros below b, so subtracting 1 turns bit b over exactly then: bit b of
// s & (s - 1) is the even neighbour's, and no carry leaves the low word (b <= 9).
template <int P, int R, int SW, int QR, bool ONE>
__device__ __forceinline__ void narrow_chain(const int32_t* sp, const unsigned char* tbl, int unit, double (&d)[8])
{
    constexpr int N = tap_count(P, R), KF = narrow_taps<P, R, ONE>(), NG = group_count<P, R>(), NQ = 8;
    static_assert(N >= KF + 1 && KF >= 2, "at least one tap on the binary64 pipe");
    const auto& T = c_narrow<P, R, SW>;
    const uint4* desc = reinterpret_cast<const uint4*>(tbl + NG * TBL_L * 24);
    auto load_v = [&](int t, uint32_t (&v)[NQ]) {
        const int32_t* s = sp + T.tap[t].off;
#pragma unroll
        for (int q = 0; q < NQ; ++q) v[q] = static_cast<uint32_t>(s[(q >> 1) * QR * SW + 32 * (q & 1)]);
    };
    auto load_p = [&](uint32_t table, const uint32_t (&v)[NQ], uint2 (&p)[NQ]) {
        const unsigned char* tf = tbl + table;
#pragma unroll
        for (int q = 0; q < NQ; ++q) p[q] = *reinterpret_cast<const uint2*>(tf + v[q]);
    };
    uint32_t x0[NQ], x1[NQ], v[NQ];
    uint2 p[NQ];
    load_v(0, v);
    load_p(T.tap[0].fix, v, p);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        x0[q] = p[q].x;
        x1[q] = p[q].y;
    }
    load_v(1, v);  // one tap ahead
    // two taps per trip where three tiles per SM leave the registers for it (n=8192, whole run of 16,
    // grid R=5: 2939 us per application against 2972)
    constexpr int UNR = strict_tiles<P, R>() == 4 ? 1 : 2;
#pragma unroll UNR
    for (int t = 1; t < KF; ++t) {
        const uint4 ds = desc[t];
        load_p(T.tap[t].fix, v, p);
        load_v(t + 1, v);
        if (ds.w == 0u) {  // one rounding position for the whole window
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const uint64_t s = ((static_cast<uint64_t>(x1[q]) << 32) | x0[q]) +
                                   ((static_cast<uint64_t>(p[q].y) << 32) | p[q].x) + ds.x;
                x1[q] = static_cast<uint32_t>(s >> 32);
                x0[q] = static_cast<uint32_t>(s);
                x0[q] &= ((x0[q] - 1u) & ds.y) | ds.z;
            }
        } else {  // from each sum's leading bit (bits 52 and up of |sum| lie in the high word)
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                uint64_t s = ((static_cast<uint64_t>(x1[q]) << 32) | x0[q]) +
                             ((static_cast<uint64_t>(p[q].y) << 32) | p[q].x);
                int f;
                asm("bfind.s32 %0, %1;" : "=r"(f) : "r"(static_cast<uint32_t>(s >> 32)));
                const uint32_t bit = 1u << max(f - 20, 0);  // 2^b
                const uint32_t c = bit - 1u, c2 = c << 1;
                s += bit >> 1;
                x1[q] = static_cast<uint32_t>(s >> 32);
                x0[q] = static_cast<uint32_t>(s);
                x0[q] &= ((x0[q] - 1u) & (c2 & ~c)) | ~(c | c2);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        if constexpr (ONE) {
            // One conversion instruction (it runs on the binary64 pipe, which has room at one application
            // per launch), exact for 53 significant bits, then the unit into the exponent.
            const uint64_t b = as_bits(__ll2double_rn(static_cast<long long>((static_cast<uint64_t>(x1[q]) << 32) | x0[q])));
            d[q] = as_dbl(b == 0 ? 0ull : b + (static_cast<uint64_t>(static_cast<int64_t>(unit)) << 52));
        } else {
            d[q] = as_dbl(fx64_to_bits(x0[q], x1[q], unit));
        }
    }
#pragma unroll 1
    for (int t = KF; t < N; ++t) {
        const NarrowTap tp = T.tap[t];
        load_v(t, v);
        load_p(tp.t64, v, p);
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            d[q] = __dadd_rn(d[q], as_dbl((static_cast<uint64_t>(p[q].y ^ tp.sign) << 32) | p[q].x));
    }
}

// True when a positive weight lies among the fixed taps: then the fixed part never sums to -0 (a rounded sum
// is -0 only when every term is -0, and w * v with w > 0 is never -0).
template <int P, int R, bool ONE>
constexpr bool fixed_prefix_has_positive()
{
    constexpr StrictTaps<P, R> t = make_strict_taps<P, R>();
    for (int k = 0; k < fixed_taps<P, R, ONE>(); ++k)
        if (!t.neg[k]) return true;
    return false;
}

// The 96-bit form: out += the chains of columns c and c + 32 of every WARPS-th row from r on, for the rows and
// columns whose bits are set. `point`, `out` and `tbl`: shared-memory addresses of the int32 tile's and the
// out words' (r, c), and of the tables, which cover [base, base + TBL_L). The adds of the first
// fixed_taps<P, R, ONE>() taps run in fixed point (fx::fx96_acc_round), the rest on the binary64 pipe.
// Bound by the integer ALU, so the taps are unrolled, with their offsets and signs in the instructions; as a
// loop over the taps, values about zero, n=4096, us per application: star R=5 in launches of two 450
// against 411, grid R=3 855 against 770, star R=3 on 64-row tiles 293 against 247. A call, because the windows
// that take this form are few and inlined it cost every kernel of the stencil registers and code (the call
// costs star R=3, 4 up to 2% at one application, n=16384, PRK field: 2533 to 2578 us, 2938 to 2999).
template <int P, int R, int SW, int TW, bool ONE>
__device__ __noinline__ void table_rows(uint32_t point, uint32_t out, uint32_t tbl, int base, uint32_t rows, uint32_t cols)
{
    constexpr StrictTaps<P, R> TP = make_strict_taps<P, R>();
    constexpr int N = tap_count(P, R), KF = fixed_taps<P, R, ONE>(), NG = group_count<P, R>();
    constexpr bool POS = fixed_prefix_has_positive<P, R, ONE>();
    const uint64_t* T64 = static_cast<const uint64_t*>(__cvta_shared_to_generic(tbl));
    const uint4* T96 = static_cast<const uint4*>(__cvta_shared_to_generic(tbl + NG * TBL_L * 8));
#pragma unroll 1
    for (; rows; rows >>= 1, point += WARPS * SW * 4, out += WARPS * TW * 8) {
        if (!(rows & 1u)) continue;
        const int32_t* sp = static_cast<const int32_t*>(__cvta_shared_to_generic(point));
        uint32_t x[2][3] = {};
        int anyv[2] = {};
#pragma unroll
        for (int t = 0; t < KF; ++t) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int v = sp[TP.dr[t] * SW + TP.dc[t] + 32 * h];
                if (!POS) anyv[h] |= v;
                const uint4 p = T96[TP.g[t] * TBL_L + (v - base)];
                if (TP.neg[t])
                    fx::fx96_acc_round<true>(x[h][0], x[h][1], x[h][2], p.x, p.y, p.z);
                else
                    fx::fx96_acc_round<false>(x[h][0], x[h][1], x[h][2], p.x, p.y, p.z);
            }
        }
        double d[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) d[h] = as_dbl(fx::fx96_to_bits(x[h][0], x[h][1], x[h][2], !POS && anyv[h] == 0));
#pragma unroll
        for (int t = KF; t < N; ++t) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int v = sp[TP.dr[t] * SW + TP.dc[t] + 32 * h];
                const double p = as_dbl(T64[TP.g[t] * TBL_L + (v - base)]);
                d[h] = TP.neg[t] ? __dsub_rn(d[h], p) : __dadd_rn(d[h], p);
            }
        }
        uint64_t* o = static_cast<uint64_t*>(__cvta_shared_to_generic(out));
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (cols >> h & 1u) o[32 * h] = as_bits(__dadd_rn(as_dbl(o[32 * h]), d[h]));
    }
}

// ---------------------------------------------------------------------------------------------
// FP64, real-valued tiles: fewer binary64 instructions with the same roundings
//
// The binary64 pipe (1/73 of the FP32 rate) bounds a tile that no exact route takes: one rounded product
// and one rounded add per tap. Two identities take most products off it without changing a bit, for
// values that are zero or far from the ends of the exponent range (checked per tile):
//  - Multiplying by +-2^-k is exact, so the product and the add of a power-of-two weight are one fused
//    multiply-add.
//  - fl(v / (2^k d)) = 2^-k fl(v / d), so the weights whose denominators share their odd part share one
//    rounded product per value, and every tap that uses it is again a fused multiply-add by +-2^-k. The
//    products of a family of weights are computed once per value into a plane of the tile in shared
//    memory (over the `out` words, the TMA kernel's barrier, which has ended, and the tables: this path
//    needs none of them by then) instead of once per tap.
// A family that has no plane multiplies per tap. Binary64 instructions per point, before and now: star
// R=2 17 and 10, star R=3 24 and 16, grid R=2 37 and 23. At n=8192, one fused application, us: star R=2
// 2185 to 1293, R=3 3199 to 2019, R=4 4215 to 2493, R=5 5229 to 3907; grid R=2 4850 to 2974, R=3 9926 to
// 8071, R=4 16775 to 13154, R=5 25399 to 22047.

__host__ __device__ constexpr int odd_part(int d)
{
    while (d % 2 == 0) d /= 2;
    return d;
}

// The families of a stencil: plane 0 is the tile itself (family 1, weights that are powers of two) or, in
// place of it, the plane of a family; plane 1 the family with the most taps beside it (0: none).
template <int P, int R, bool INPLACE>
struct RealPlan {
    int fam0 = 1, fam1 = 0;        // odd parts
    int den0 = 1, den1 = 1;        // the planes hold fl(v / den)
    int off_dr[tap_count(P, R)] = {}, off_dc[tap_count(P, R)] = {};
    int plane[tap_count(P, R)] = {};   // 0, 1, or 2: a product of its own
    double c[tap_count(P, R)] = {};    // the factor of the plane's value, or the weight
};

template <int P, int R>
__host__ __device__ constexpr int taps_of_family(int fam)
{
    int k = 0;
    for (int dc = -R; dc <= R; ++dc)
        for (int dr = -R; dr <= R; ++dr) {
            const int d = weight_den(P, R, dc, dr);
            if (d != 0 && odd_part(d) == fam) ++k;
        }
    return k;
}

// The family with the most taps other than 1 and `but`, 0 when there is none.
template <int P, int R>
__host__ __device__ constexpr int largest_family(int but)
{
    int best = 0, most = 0;
    for (int dc = -R; dc <= R; ++dc)
        for (int dr = -R; dr <= R; ++dr) {
            const int d = weight_den(P, R, dc, dr);
            if (d == 0) continue;
            const int f = odd_part(d);
            if (f != 1 && f != but && taps_of_family<P, R>(f) > most) {
                best = f;
                most = taps_of_family<P, R>(f);
            }
        }
    return best;
}

// True when two families cover every tap, so that both planes' values replace the tile's.
template <int P, int R>
__host__ __device__ constexpr bool two_families()
{
    const int a = largest_family<P, R>(0);
    const int b = a ? largest_family<P, R>(a) : 0;
    return b != 0 && taps_of_family<P, R>(a) + taps_of_family<P, R>(b) == tap_count(P, R);
}

template <int P, int R, bool INPLACE>
constexpr RealPlan<P, R, INPLACE> make_real_plan()
{
    RealPlan<P, R, INPLACE> t{};
    const int big = largest_family<P, R>(0);
    if (INPLACE) {
        t.fam0 = big;
        t.fam1 = largest_family<P, R>(big);
    } else {
        t.fam1 = big;
    }
    // a plane's denominator: the first tap's of its family, so that the chain's first product needs no factor
    for (int pass = 0; pass < 2; ++pass) {
        int k = 0;
        bool set0 = false, set1 = false;
        for (int dc = -R; dc <= R; ++dc)
            for (int dr = -R; dr <= R; ++dr) {
                const int d = weight_den(P, R, dc, dr);
                if (d == 0) continue;
                const int f = odd_part(d), s = weight_sign(P, R, dc, dr);
                if (pass == 0) {
                    if (INPLACE && f == t.fam0 && !set0) {
                        t.den0 = d;
                        set0 = true;
                    }
                    if (t.fam1 != 0 && f == t.fam1 && !set1) {
                        t.den1 = d;
                        set1 = true;
                    }
                } else {
                    t.off_dr[k] = dr;
                    t.off_dc[k] = dc;
                    t.plane[k] = f == t.fam0 ? 0 : (f == t.fam1 ? 1 : 2);
                    const int den = t.plane[k] == 0 ? t.den0 : t.den1;
                    t.c[k] = t.plane[k] == 2 ? weight(P, R, dc, dr) : s * (static_cast<double>(den) / d);
                }
                ++k;
            }
    }
    return t;
}

// The planes of the staged tile: plane 1 beside it, and plane 0 in its place (INPLACE).
template <int P, int R, bool INPLACE, int ELEMS>
__device__ __forceinline__ void real_planes(double* s_in, double* p1)
{
    constexpr RealPlan<P, R, INPLACE> T = make_real_plan<P, R, INPLACE>();
    if constexpr (T.fam1 != 0) {
#pragma unroll 4
        for (int idx = threadIdx.x; idx < ELEMS; idx += THREADS) {
            const double v = s_in[idx];
            p1[idx] = __dmul_rn(v, 1.0 / T.den1);
            if (INPLACE) s_in[idx] = __dmul_rn(v, 1.0 / T.den0);
        }
    }
}

// S of CPT adjacent points: the reference's chain, its products from the planes; p0 and p1 point at the
// first point's value in them.
template <int P, int R, bool INPLACE, int LD, int CPT>
__device__ __forceinline__ void real_points(const double* p0, const double* p1, double (&acc)[CPT])
{
    constexpr RealPlan<P, R, INPLACE> T = make_real_plan<P, R, INPLACE>();
#pragma unroll
    for (int t = 0; t < tap_count(P, R); ++t) {
        const double* src = (T.plane[t] == 1 ? p1 : p0) + T.off_dr[t] * LD + T.off_dc[t];
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            if (t == 0)
                acc[k] = T.c[t] == 1.0 && T.plane[t] != 2 ? src[k]
                         : T.c[t] == -1.0 && T.plane[t] != 2
                             ? as_dbl(as_bits(src[k]) ^ fx::SIGN)
                             : __dmul_rn(src[k], T.c[t]);
            else if (T.plane[t] == 2)
                acc[k] = __dadd_rn(acc[k], __dmul_rn(src[k], T.c[t]));
            else
                acc[k] = __fma_rn(src[k], T.c[t], acc[k]);
        }
    }
}

// S of two adjacent points, by real_points (real) or fp64_pair_strict. A call, so that its registers are
// its own: inlined, it spilled the HBM-bound kernels around it (n=16384, one fused application, star R=2
// 1209 us against 1205); bound by the binary64 pipe, it loses nothing by it.
template <int P, int R, bool INPLACE, int LD>
__device__ __noinline__ double2 fp64_pair(const double* p0, const double* p1, bool real)
{
    if (!real) return fp64_pair_strict<P, R, LD>(p0);
    double d[2];
    real_points<P, R, INPLACE, LD, 2>(p0, p1, d);
    return make_double2(d[0], d[1]);
}

// A value the path takes: zero, or normal with every product of it normal.
__device__ __forceinline__ bool real_value(uint64_t b)
{
    return (b << 1) == 0 || ((static_cast<uint32_t>(b >> 52) & 0x7FFu) - 128u) < 1772u;
}

// Bytes of the shared-memory out area the table route needs besides its tables in kernels that keep
// out in HBM (one FP64 tile of out words; the TMA kernel updates its out tile instead).
__host__ __device__ constexpr int table_out_bytes() { return Cfg<FP64>::TW * Cfg<FP64>::TH * 8; }

// dst = src + one over a whole int32 tile, halo included, as 16-byte vectors.
template <int ELEMS>
__device__ __forceinline__ void advance_i32_to(const int32_t* src, int32_t* dst, int one)
{
    constexpr int NV = ELEMS / 4;
#pragma unroll
    for (int q = 0; q < (NV + THREADS - 1) / THREADS; ++q) {
        const int idx = threadIdx.x + q * THREADS;
        if (NV % THREADS == 0 || idx < NV) {
            int4 v = reinterpret_cast<const int4*>(src)[idx];
            v.x += one;
            v.y += one;
            v.z += one;
            v.w += one;
            reinterpret_cast<int4*>(dst)[idx] = v;
        }
    }
}

// Where a whole-number tile's int32 words lie (elements from the stage) and how they hold the values:
// value = (word >> shift) + add.
struct WholeTile {
    int off = 0, shift = 0, add = 0;
};

// The table route for a whole tile whose int32 values (the tile's in, halo included) lie in
// [lo, hi]: `nsteps` applications. The int32 tile takes half of the FP64 stage, so the other half
// holds the next application's in: while application t reads one, in + 1 goes to the other, and
// one barrier per application separates them; *fin says where and how the last application's in is
// left for the stores. Lane l owns columns l and l + 32 of its warp's rows; every application
// adds its S into their out words in o_s, a shared-memory tile of out words (row stride TW). With
// OUT_SMEM, o_s is the TMA kernel's out tile, which the stores then read in their own layout; with
// the other sources o_s is scratch, filled from the out array (out_g points at the tile's (0, 0),
// row stride n) before the first application and written back after the last, each thread its own
// points. Returns false, having done nothing, when the values span TBL_L or more (lo and hi are
// block-uniform). ONE: the launch applies the stencil once (the fixed-point share of one application).
template <int P, int R, int SW, int SH, int TW, int ROWS, int OUT_SRC, bool ONE>
__device__ __forceinline__ bool table_tile(int32_t* si, uint64_t* o_s, uint64_t* out_g, unsigned char* tbl, int lo,
                                           int hi, int nsteps, int64_t i0, int64_t j0, int64_t n, int64_t goff,
                                           int64_t row_end, bool has_out, WholeTile* fin)
{
    constexpr int ELEMS = SW * SH;
    static_assert(TW == 64, "two columns per lane, 32 apart");
    static_assert(ELEMS % 4 == 0, "the advance moves 16-byte vectors");
    if (hi - lo >= TBL_L) return false;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t* T64 = reinterpret_cast<uint64_t*>(tbl);
    uint4* T96 = reinterpret_cast<uint4*>(tbl + group_count<P, R>() * TBL_L * 8);
    // Application t's in is the int32 tile at si + cur: values, or (narrow) byte offsets into the
    // window's tables. The other half of the stage takes in + 1 for application t + 1.
    constexpr int QR = ROWS * WARPS / 4;
    static_assert(QR % WARPS == 0, "a thread's rows in groups of four, QR apart");
    int cur = 0, base = lo, unit = 0;
    bool narrow = false;
    // The tables of the window of values from application t's smallest on, complete on return: the
    // narrow form's (with the tile turned into table offsets) where it holds, else the 96-bit form's. si is
    // at application t.
    auto build = [&](int t) {
        base = lo + t;
        narrow = build_narrow<P, R, SW, ONE>(tbl, base, min(hi + nsteps - 1, base + TBL_L - 1), &unit);
        if (narrow) {
            offsets_tile<ELEMS, true>(si + cur, base);
            __syncthreads();
        }
        if (!narrow) {
            __syncthreads();  // a form that was tried and given up is overwritten
            build_tables<P, R>(T64, T96, base);
            __syncthreads();
        }
    };
    if constexpr (OUT_SRC != OUT_SMEM) {
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp + WARPS * rr;
            const int64_t gi = i0 + r;
            if (!table_row_active(has_out, gi, gi + goff, row_end, n, R)) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                if (j0 + c >= R && j0 + c < n - R) o_s[r * TW + c] = out_g[r * n + c];
            }
        }
    }
    // which of a word row's eight points are updated: bit q of the group's mask (narrow form)
    auto active = [&](int wr) {
        uint32_t m = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int64_t gi = i0 + wr + (q >> 1) * QR, c = j0 + lane + 32 * (q & 1);
            if (table_row_active(has_out, gi, gi + goff, row_end, n, R) && c >= R && c < n - R) m |= 1u << q;
        }
        return m;
    };
    const uint32_t act0 = active(warp);
    build(0);
#pragma unroll 1
    for (int t = 0; t < nsteps; ++t) {
        if (t > 0 && hi + t >= base + TBL_L) {  // the values outgrew the table: rebuild it at the new minimum
            if (narrow) offsets_tile<ELEMS, false>(si + cur, base);
            build(t);
        }
        if (narrow) {
#pragma unroll 1
            for (int wr = warp; wr < QR; wr += WARPS) {
                const uint32_t act = ROWS == 4 ? act0 : active(wr);
                if (__ballot_sync(0xffffffffu, act != 0) == 0) continue;  // no interior point in the warp's rows
                double d[8];
                narrow_chain<P, R, SW, QR, ONE>(si + cur + (wr + R) * SW + (SW - TW) / 2 + lane, tbl, unit, d);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    uint64_t* o = o_s + (wr + (q >> 1) * QR) * TW + lane + 32 * (q & 1);
                    if (act >> q & 1u) *o = as_bits(__dadd_rn(as_dbl(*o), d[q]));
                }
            }
        } else {
            uint32_t rows = 0, cols = 0;  // the warp's rows and columns that hold points to update
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                const int64_t gi = i0 + warp + WARPS * rr;
                if (table_row_active(has_out, gi, gi + goff, row_end, n, R)) rows |= 1u << rr;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (j0 + lane + 32 * h >= R && j0 + lane + 32 * h < n - R) cols |= 1u << h;
            table_rows<P, R, SW, TW, ONE>(smem_addr(si + cur + (warp + R) * SW + (SW - TW) / 2 + lane),
                                          smem_addr(o_s + warp * TW + lane), smem_addr(tbl), base, rows, cols);
        }
        if (t + 1 < nsteps) {  // in += 1
            advance_i32_to<ELEMS>(si + cur, si + (ELEMS - cur), narrow ? 8 : 1);
            cur = ELEMS - cur;
            __syncthreads();  // the next application's in complete, this one's reads done
        }
    }
    // The last application's in, for the stores: value = (word >> shift) + add. The words stay as they
    // are, as other warps may still be reading them.
    fin->off = cur;
    fin->shift = narrow ? 3 : 0;
    fin->add = narrow ? base : 0;
    if constexpr (OUT_SRC != OUT_SMEM) {
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp + WARPS * rr;
            const int64_t gi = i0 + r;
            if (!table_row_active(has_out, gi, gi + goff, row_end, n, R)) continue;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = lane + 32 * h;
                if (j0 + c >= R && j0 + c < n - R) out_g[r * n + c] = o_s[r * TW + c];
            }
        }
    }
    __syncthreads();  // the out tile complete before the stores read it in their layout
    return true;
}

// ---------------------------------------------------------------------------------------------
// The kernel

// True when the tile at (i0, j0) holds interior points, i.e. has an out tile to load and update.
__device__ __forceinline__ bool tile_has_out(int64_t i0, int64_t j0, int64_t n, int R, int tw, int th)
{
    return (i0 + th > R) && (i0 < n - R) && (j0 + tw > R) && (j0 < n - R);
}


// Evaluate one tile whose `in` (with halo) is in shared memory: STEPS applications (`depth` when
// STEPS = 0), then in_next and out to HBM, with out read from OUT_SRC. vec_ok: rows are 16-byte
// aligned and n is a multiple of CPT, so a thread's CPT points move as one vector; otherwise they
// move one by one.
// The arrays hold rows of an n x n grid (row stride n); i0 is the tile's first row in the arrays and
// goff the grid row of the arrays' row 0 (0 for a whole grid; a row slab's first row otherwise).
// Rows from row_end on (in the arrays) are not stored; the interior test uses grid rows.
template <int P, int R, int DT, int STEPS, int OUT_SRC = OUT_SMEM, int TH_ = 32>
__device__ __forceinline__ void process_tile(unsigned char* stage, int* s_red, int64_t i0, int64_t j0, int64_t n,
                                             bool has_out, void* in_next_v, void* out_v,
                                             bool vec_ok, int depth, int64_t goff, int64_t row_end,
                                             unsigned char* tbl, const IntTile& pre = IntTile{})
{
    const int nsteps = STEPS > 0 ? STEPS : (STEPS == OPERATOR ? 1 : depth);
    constexpr bool ROUTE = int_route<P, R, DT, STEPS, OUT_SRC != OUT_SMEM>();
    using G = Geo<DT, R, TH_>;
    using C = Cfg<DT, TH_>;
    using T = typename C::T;
    constexpr int CPT = C::CPT;
    constexpr int ROWS = G::ROWS;
    constexpr bool EXACT = DT == FP64 && pow2_weights(P, R);
    T* s_in = reinterpret_cast<T*>(stage);
    uint64_t* o_tile = reinterpret_cast<uint64_t*>(stage + G::OUT_OFF);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c0 = lane * CPT;
    const int64_t gj = j0 + c0;
    const bool col_ok = gj < n;  // at least the first of the thread's CPT columns is in the grid
    const bool cols_interior = gj >= R && gj + CPT <= n - R;
    // the out word of point (r, c0 + k), from the smem out tile or from HBM
    auto load_out = [&](int r, int k) -> uint64_t {
        if constexpr (OUT_SRC != OUT_SMEM) {
            return gj + k < n ? static_cast<const uint64_t*>(out_v)[(i0 + r) * n + gj + k] : 0ull;
        } else {
            return o_tile[r * C::TW + c0 + k];
        }
    };
    // the CPT out words of row r: from HBM as 16-byte vectors where the row's words start on a 16-byte
    // boundary and lie inside the grid (every other row when n is odd), else one by one
    auto load_out_row = [&](int r, uint64_t (&o)[CPT]) {
        if constexpr (OUT_SRC != OUT_SMEM) {
            const uint64_t* src = static_cast<const uint64_t*>(out_v) + (i0 + r) * n + gj;
            if (gj + CPT <= n && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
#pragma unroll
                for (int k = 0; k < CPT; k += 2) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(src + k);
                    o[k] = w.x;
                    o[k + 1] = w.y;
                }
                return;
            }
        }
#pragma unroll
        for (int k = 0; k < CPT; ++k) o[k] = load_out(r, k);
    };

    // the same words as FP32C pairs
    auto load_pairs = [&](int r, float (&hi)[CPT], float (&lo)[CPT]) {
        const float2* src = OUT_SRC == OUT_SMEM
                                ? reinterpret_cast<const float2*>(o_tile) + r * C::TW + c0
                                : static_cast<const float2*>(static_cast<const void*>(out_v)) + (i0 + r) * n + gj;
        if (OUT_SRC == OUT_SMEM || (gj + CPT <= n && (reinterpret_cast<uintptr_t>(src) & 15u) == 0)) {
#pragma unroll
            for (int k = 0; k < CPT; k += 2) {
                const float4 w = *reinterpret_cast<const float4*>(src + k);
                hi[k] = w.x;
                lo[k] = w.y;
                hi[k + 1] = w.z;
                lo[k + 1] = w.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < CPT; ++k)
                if (gj + k < n) {
                    const float2 w = src[k];
                    hi[k] = w.x;
                    lo[k] = w.y;
                }
        }
    };

    // ---- FP64 power-of-two stencils: certify the tile for an exact route ----
    // First the FP32 route: every value +0 or an integer of magnitude below 2^20 (checked with a few
    // integer ops and one FP32 round trip, no binary64 instruction). Otherwise the general integer
    // route (lowest-set-bit classification, int32/int64 arithmetic), otherwise strict binary64.
    int unit = fx::NOT_FIXED;
    bool narrow = false;
    bool fexact = false;
    if constexpr (EXACT) {
        constexpr int SHIFT = pow2_shift(P, R);
        constexpr long long L1 = pow2_coef_l1(P, R);
        constexpr int PER = (G::ELEMS + THREADS - 1) / THREADS;
        // FP32 route bound: L1 * (2^20 + steps) < 2^24 for L1 <= 15 and steps <= FP32_MAX_STEPS
        static_assert(L1 < 16 && STEPS <= FP32_MAX_STEPS, "FP32 route bound");
        const uint64_t* raw = reinterpret_cast<const uint64_t*>(s_in);
        float fv[PER];
        bool ok = true;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int idx = threadIdx.x + q * THREADS;
            const uint64_t b = idx < G::ELEMS ? raw[idx] : 0ull;
            const uint32_t hi32 = static_cast<uint32_t>(b >> 32), lo32 = static_cast<uint32_t>(b);
            const uint32_t e = (hi32 >> 20) & 0x7FFu;
            const bool small = e >= 1023u && e < 1043u && (lo32 & 0x1FFFFFFFu) == 0u;
            const float f = __uint_as_float((hi32 & 0x80000000u) | (((hi32 & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo32 >> 29));
            const float fr = __fsub_rn(__fadd_rn(f, 12582912.0f), 12582912.0f);  // nearest integer, |f| < 2^22
            ok = ok && (b == 0ull || (small && fr == f));
            fv[q] = b == 0ull ? 0.0f : f;
        }
        if (STEPS == 0 && nsteps > FP32_MAX_STEPS) ok = false;
        ok = __syncthreads_and(ok) != 0;
        if (ok) {
            float* sf = reinterpret_cast<float*>(s_in);
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int idx = threadIdx.x + q * THREADS;
                if (idx < G::ELEMS) sf[idx] = fv[q];
            }
            fexact = true;
        } else {
            int lo = fx::ZERO_LO, hi = fx::ZERO_HI;
            for (int idx = threadIdx.x; idx < G::ELEMS; idx += THREADS) {
                int l, h;
                fx::classify(raw[idx], l, h);
                lo = min(lo, l);
                hi = max(hi, h);
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                s_red[2 * warp] = lo;
                s_red[2 * warp + 1] = hi;
            }
            __syncthreads();
            lo = s_red[0];
            hi = s_red[1];
#pragma unroll
            for (int w = 1; w < WARPS; ++w) {
                lo = min(lo, s_red[2 * w]);
                hi = max(hi, s_red[2 * w + 1]);
            }
            unit = fx::certify(lo, hi, SHIFT, L1, nsteps);
            if (unit != fx::NOT_FIXED) {
                // int32 arithmetic suffices when every partial sum and every updated value stays below 2^31
                const int span = hi == fx::ZERO_HI ? 0 : hi + 1 - unit;
                narrow = span <= 30 && -unit <= 26 &&
                         ((1ll << span) + static_cast<long long>(nsteps) * (1ll << (-unit))) < (1ll << 31) / L1;
                __syncthreads();  // every thread has read its raw words
                int64_t* iv = reinterpret_cast<int64_t*>(s_in);
                for (int idx = threadIdx.x; idx < G::ELEMS; idx += THREADS) iv[idx] = fx::to_fixed(raw[idx], unit);
            }
        }
        __syncthreads();  // every converted word visible
    }
    // Elements no stored point reads (outside the grid, or past the last row's halo) hold zeros. They stay
    // out of a tile's range, so that a tile at the grid's edge has the range of its own values: counted
    // in, they made it too wide for the table and integer routes (at n=1000 on 18% of the tiles).
    const int64_t row_hi = min(row_end + R, n - goff);  // first array row past those that are read
    const bool edge = i0 < R || j0 < G::RA || i0 + C::TH + R > row_hi || j0 + C::TW + G::RA > n;
    auto inside = [&](int idx) {
        const int r = idx / G::SW, c = idx - r * G::SW;
        return static_cast<uint64_t>(i0 - R + r) < static_cast<uint64_t>(row_hi) &&
               static_cast<uint64_t>(j0 - G::RA + c) < static_cast<uint64_t>(n);
    };

    // ---- FP64, other weights: whole-number tiles take their products off the binary64 pipe ----
    // Every value +0 or a whole number below 2^19 (so that up to 2^19 applications of in += 1 stay
    // below 2^20): the tile is held as int32 and fp64_points_whole evaluates it.
    bool iwhole = false;
    if constexpr (DT == FP64 && !EXACT) {
        constexpr int PER = (G::ELEMS + THREADS - 1) / THREADS;
        const uint64_t* raw = reinterpret_cast<const uint64_t*>(s_in);
        int32_t iv[PER];
        bool ok = nsteps <= (1 << 19);
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int idx = threadIdx.x + q * THREADS;
            const uint64_t b = idx < G::ELEMS ? raw[idx] : 0ull;
            // |v| in [1, 2^19) by its exponent; then v as a float (the exponent rebiased, the fraction
            // bits a float cannot hold checked for zero) and as an integer, rounded by the magic number
            // and compared back
            const uint32_t hi32 = static_cast<uint32_t>(b >> 32), lo32 = static_cast<uint32_t>(b);
            const bool in_range = (hi32 & 0x7FFFFFFFu) - 0x3FF00000u < (19u << 20);
            const uint32_t fb = __funnelshift_l(lo32, hi32, 3) - (128u << 23);
            const float f = __uint_as_float((hi32 & 0x80000000u) | (fb & 0x7FFFFFFFu));
            const float t = __fadd_rn(f, 12582912.0f);  // 1.5 * 2^23
            const bool whole = in_range && (lo32 & 0x1FFFFFFFu) == 0u && __fsub_rn(t, 12582912.0f) == f;
            iv[q] = whole ? static_cast<int32_t>(__float_as_uint(t) - 0x4B400000u) : 0;
            ok = ok && (b == 0ull || whole);
        }
        if constexpr (table_route<P, R, DT>()) {
            // the tile's range for the table route, published with the certification's barrier
            int lo = 0x7FFFFFFF, hi = -0x7FFFFFFF;
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int idx = threadIdx.x + q * THREADS;
                if (idx < G::ELEMS && (!edge || inside(idx))) {
                    lo = min(lo, iv[q]);
                    hi = max(hi, iv[q]);
                }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                s_red[2 * warp] = lo;
                s_red[2 * warp + 1] = hi;
            }
        }
        iwhole = __syncthreads_and(ok) != 0;
        if (iwhole) {
            int32_t* si = reinterpret_cast<int32_t*>(s_in);
            int fill = 0;
            if (edge) {
                fill = s_red[0];
#pragma unroll
                for (int w = 1; w < WARPS; ++w) fill = min(fill, s_red[2 * w]);
            }
#pragma unroll
            for (int q = 0; q < PER; ++q) {
                const int idx = threadIdx.x + q * THREADS;
                if (idx < G::ELEMS) si[idx] = !edge || inside(idx) ? iv[q] : fill;
            }
        }
        __syncthreads();
    }

    // ---- FP64, other weights: the table route (table_tile), when the kernel has a table area and
    // the tile's range fits it ----
    bool tbl_done = false;
    WholeTile iw_fin;  // the int32 tile of the last application's in
    if constexpr (table_route<P, R, DT>()) {
        if (iwhole && tbl) {
            int lo = s_red[0], hi = s_red[1];
#pragma unroll
            for (int w = 1; w < WARPS; ++w) {
                lo = min(lo, s_red[2 * w]);
                hi = max(hi, s_red[2 * w + 1]);
            }
            // kernels that keep out in HBM give the route an out area right after the tables
            uint64_t* o_s = OUT_SRC == OUT_SMEM ? o_tile : reinterpret_cast<uint64_t*>(tbl + table_bytes<P, R, DT>());
            tbl_done = table_tile<P, R, G::SW, G::SH, C::TW, ROWS, OUT_SRC, one_application(STEPS)>(
                reinterpret_cast<int32_t*>(s_in), o_s, static_cast<uint64_t*>(out_v) + i0 * n + j0, tbl, lo, hi,
                nsteps, i0, j0, n, goff, row_end, has_out, &iw_fin);
        }
    }

    // The table route with out in HBM has stored out itself; the stores then write in_next only
    const bool out_via_rows = !(tbl_done && OUT_SRC != OUT_SMEM);

    // ---- FP32C: whole-number tiles of small range take the integer route ----
    int sums = 0;  // applications one FP32 sum takes on the route
    float uref = 0.0f;
    if constexpr (ROUTE) {
        if (pre.known) {
            sums = pre.sums;
            uref = pre.ref;
        } else {
            constexpr int NV = G::ELEMS / 4, PER = (NV + THREADS - 1) / THREADS;
            static_assert(G::ELEMS % 4 == 0, "the tile as 16-byte vectors");
            // the value nearest the tile's middle inside the grid
            const int rm = static_cast<int>(min(static_cast<int64_t>(G::SH / 2), row_hi - 1 - (i0 - R)));
            const int cm = static_cast<int>(min(static_cast<int64_t>(G::SW / 2), n - 1 - (j0 - G::RA)));
            uref = s_in[rm * G::SW + cm];
            if (IntCheck::hopeful<P, R>(uref, s_in[R * G::SW + G::RA], s_in[rm * G::SW + G::RA])) {  // block-uniform
                float4 u[PER];
                IntCheck check;
#pragma unroll
                for (int q = 0; q < PER; ++q) {
                    const int v = threadIdx.x + q * THREADS;
                    u[q] = v < NV ? reinterpret_cast<const float4*>(s_in)[v] : make_float4(uref, uref, uref, uref);
                    float* e = reinterpret_cast<float*>(&u[q]);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float x = e[k];
                        e[k] = __fsub_rn(x, uref);
                        if (!edge || inside(4 * v + k)) check.add(x, e[k]);
                    }
                }
                sums = check.sums<P, R>(uref, nsteps);
                if (sums) {
#pragma unroll
                    for (int q = 0; q < PER; ++q) {
                        const int v = threadIdx.x + q * THREADS;
                        if (v < NV) reinterpret_cast<float4*>(s_in)[v] = u[q];
                    }
                    __syncthreads();
                }
            }
        }
    }

    const bool inted = sums != 0;

    // ---- FP64, real-valued tiles: products shared or fused into the adds (real_points) ----
    constexpr bool INPLACE = one_application(STEPS) && two_families<P, R>();
    constexpr bool PLANES = DT == FP64 && !EXACT;  // the power-of-two stencils need no plane beside the tile
    bool real = false;
    // plane 1: from the out words on (read into registers first), over the reduction words, the TMA kernel's
    // barrier (ended by then) and the tables
    double* p1 = nullptr;
    if constexpr (DT == FP64) {
        if ((EXACT ? one_application(STEPS) && !fexact && unit == fx::NOT_FIXED : !iwhole) && (!PLANES || tbl)) {
            bool ok = true;
            for (int idx = threadIdx.x; idx < G::ELEMS; idx += THREADS)
                ok = ok && real_value(reinterpret_cast<const uint64_t*>(s_in)[idx]);
            real = __syncthreads_and(ok) != 0;
            p1 = reinterpret_cast<double*>(OUT_SRC == OUT_SMEM ? stage + G::OUT_OFF : tbl);
            constexpr int AREA = OUT_SRC == OUT_SMEM
                                     ? table_offset<DT, R, TH_>() + table_bytes<P, R, DT>() - G::OUT_OFF
                                     : table_bytes<P, R, DT>() + table_out_bytes();
            static_assert(!PLANES || AREA >= G::IN_BYTES, "plane 1 fits over the out words and the tables");
        }
    }
    // S of the two points of row r by binary64 instructions, into the out words
    auto fp64_row = [&](int r, uint64_t* o) {
        if constexpr (DT == FP64) {
            const int soff = (r + R) * G::SW + G::RA + c0;
            const double2 S =
                fp64_pair<P, R, INPLACE, G::SW>(reinterpret_cast<const double*>(s_in) + soff, p1 + soff, real);
            o[0] = as_bits(__dadd_rn(as_dbl(o[0]), S.x));
            o[1] = as_bits(__dadd_rn(as_dbl(o[1]), S.y));
        }
    };

    // Set by the multi-application FP32 route when the tile's out words are held as integers
    bool oint = false;
    // Offset in floats of the FP32 tile holding the last application's in (double-buffered route)
    int fin_off = 0;

    // S of CPT points of row r (tile coordinates) added into the out words o[] (in place)
    auto apply_row = [&](int r, uint64_t* o) {
        const int soff = (r + R) * G::SW + G::RA + c0;  // in(r, c0) in the tile
        if constexpr (DT == FP64) {
            bool done = false;
            if constexpr (EXACT) {
                constexpr int SHIFT = pow2_shift(P, R);
                const int64_t* v = reinterpret_cast<const int64_t*>(s_in) + soff;
                if (fexact) {
                    float S[CPT];
                    fexact_points<P, R, CPT, G::RA>(reinterpret_cast<const float*>(s_in) + soff, G::SW, S);
                    if (oint) {
#pragma unroll
                        for (int k = 0; k < CPT; ++k) {
                            if constexpr (STEPS == 0)
                                o[k] += static_cast<uint64_t>(static_cast<int64_t>(__float2int_rn(S[k])));
                            else
                                o[k] = static_cast<uint32_t>(static_cast<uint32_t>(o[k]) + static_cast<uint32_t>(__float2int_rn(S[k])));
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < CPT; ++k) o[k] = as_bits(__dadd_rn(as_dbl(o[k]), as_dbl(f2d(S[k], -SHIFT))));
                    }
                    done = true;
                } else if (unit != fx::NOT_FIXED) {
                    if (narrow) {
                        int32_t S[CPT];
                        fx_points<P, R, CPT, G::RA>(v, G::SW, S);
#pragma unroll
                        for (int k = 0; k < CPT; ++k)
                            o[k] = as_bits(__dadd_rn(as_dbl(o[k]), as_dbl(from_fixed32(S[k], unit - SHIFT))));
                    } else {
                        int64_t S[CPT];
                        fx_points<P, R, CPT, G::RA>(v, G::SW, S);
#pragma unroll
                        for (int k = 0; k < CPT; ++k)
                            o[k] = as_bits(__dadd_rn(as_dbl(o[k]), as_dbl(fx::from_fixed(S[k], unit - SHIFT))));
                    }
                    done = true;
                }
            }
            if constexpr (!EXACT) {
                if (iwhole) {
                    double S[CPT];
                    fp64_points_whole<P, R, G::SW, CPT>(reinterpret_cast<const int32_t*>(s_in) + soff, S);
#pragma unroll
                    for (int k = 0; k < CPT; ++k) o[k] = as_bits(__dadd_rn(as_dbl(o[k]), S[k]));
                    done = true;
                }
            }
            if constexpr (EXACT && !one_application(STEPS)) {
                // products and adds apart, inlined: calls here cost the FP32 loop of several applications 2%
                if (!done) {
                    const double* sp = reinterpret_cast<const double*>(s_in) + soff;
#pragma unroll
                    for (int k = 0; k < CPT; ++k)
                        o[k] = as_bits(__dadd_rn(as_dbl(o[k]), fp64_point<P, R>(sp + k, G::SW)));
                }
            } else if (!done) {
                fp64_row(r, o);
            }
        } else {
            const float* sp = reinterpret_cast<const float*>(s_in) + soff;
            float sh[CPT], sl[CPT];
            // the operator form keeps one product per tap: a group's sum would round its differences again
            if constexpr (STEPS == OPERATOR)
                fp32c_taps<P, R, CPT, G::RA>(sp, G::SW, sh, sl);
            else
                fp32c_points<P, R, CPT, G::RA>(sp, G::SW, sh, sl);
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                float oh = __uint_as_float(static_cast<uint32_t>(o[k]));
                float ol = __uint_as_float(static_cast<uint32_t>(o[k] >> 32));
                df_add(oh, ol, sh[k], sl[k]);
                o[k] = static_cast<uint64_t>(__float_as_uint(oh)) | (static_cast<uint64_t>(__float_as_uint(ol)) << 32);
            }
        }
    };

    // in_next (in + 1 after the last application) of row r to HBM
    auto store_next = [&](int r) {
        if constexpr (STEPS != OPERATOR) {
            const int64_t gi = i0 + r;
            const int soff = (r + R) * G::SW + G::RA + c0;
            T nxt[CPT];
            bool done = false;
            if constexpr (EXACT) {
                if (fexact) {
                    const float* v = reinterpret_cast<const float*>(s_in) + fin_off + soff;
#pragma unroll
                    for (int k = 0; k < CPT; ++k) nxt[k] = as_dbl(f2d(__fadd_rn(v[k], 1.0f), 0));
                    done = true;
                } else if (unit != fx::NOT_FIXED) {
                    const int64_t* v = reinterpret_cast<const int64_t*>(s_in) + soff;
                    const int64_t one = 1ll << (-unit);
                    if (narrow) {
#pragma unroll
                        for (int k = 0; k < CPT; ++k) nxt[k] = as_dbl(from_fixed32(static_cast<int32_t>(v[k] + one), unit));
                    } else {
#pragma unroll
                        for (int k = 0; k < CPT; ++k) nxt[k] = as_dbl(fx::from_fixed(v[k] + one, unit));
                    }
                    done = true;
                }
            }
            if constexpr (DT == FP64 && !EXACT) {
                if (iwhole) {
                    const int32_t* v = reinterpret_cast<const int32_t*>(s_in) + iw_fin.off + soff;
#pragma unroll
                    for (int k = 0; k < CPT; ++k) nxt[k] = as_dbl(whole_bits((v[k] >> iw_fin.shift) + iw_fin.add + 1));  // below 2^20
                    done = true;
                }
            }
            if (!done) {
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    if constexpr (DT == FP64)
                        nxt[k] = inc_exact(s_in[soff + k]);
                    else  // the tile holds in - uref on the integer route
                        nxt[k] = __fadd_rn(s_in[soff + k], inted ? __fadd_rn(uref, 1.0f) : 1.0f);
                }
            }
            T* nx = static_cast<T*>(in_next_v) + gi * n + gj;
            // 16-byte stores wherever the row's words start on a 16-byte boundary inside the grid (every
            // row for the TMA tiles; every other row for an odd n)
            if (vec_ok || (gj + CPT <= n && (reinterpret_cast<uintptr_t>(nx) & 15u) == 0)) {
                st_vec(nx, nxt);
            } else {
#pragma unroll
                for (int k = 0; k < CPT; ++k)
                    if (gj + k < n) nx[k] = nxt[k];
            }
        }
    };

    // and out
    auto store_out = [&](int r, const uint64_t* o, bool row_out) {
        const int64_t gi = i0 + r;
        if (row_out) {
            uint64_t* out = static_cast<uint64_t*>(out_v) + gi * n + gj;
            if (cols_interior && (vec_ok || (reinterpret_cast<uintptr_t>(out) & 15u) == 0)) {
#pragma unroll
                for (int k = 0; k < CPT; k += 2) *reinterpret_cast<ulonglong2*>(out + k) = make_ulonglong2(o[k], o[k + 1]);
            } else {
#pragma unroll
                for (int k = 0; k < CPT; ++k)
                    if (gj + k >= R && gj + k < n - R) out[k] = o[k];
            }
        }
    };

    auto store_row = [&](int r, const uint64_t* o, bool row_out) {
        store_next(r);
        store_out(r, o, row_out);
    };

    if constexpr (one_application(STEPS) && PLANES) {
        if (real) {
            // in_next leaves first (the tile may be overwritten by a plane), and out waits in registers
            uint64_t o[ROWS][CPT];
            bool act[ROWS];
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                const int r = warp * ROWS + rr;
                const int64_t gi = i0 + r, gg = gi + goff;
                const bool row = col_ok && gi < row_end;
                act[rr] = row && has_out && gg >= R && gg < n - R;
                if (row) store_next(r);
                if (act[rr]) load_out_row(r, o[rr]);
            }
            __syncthreads();  // every thread has read its values and out words
            real_planes<P, R, INPLACE, G::ELEMS>(reinterpret_cast<double*>(s_in), p1);
            __syncthreads();
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                const int r = warp * ROWS + rr;
                if (!act[rr]) continue;
                fp64_row(r, o[rr]);
                store_out(r, o[rr], true);
            }
            return;
        }
    }
    if constexpr (one_application(STEPS) && EXACT) {
        if (!fexact) {
            // the other routes row by row in a loop of their own, so that the FP32 route's code below keeps
            // its registers
#pragma unroll 1
            for (int rr = 0; rr < ROWS; ++rr) {
                const int r = warp * ROWS + rr;
                const int64_t gi = i0 + r, gg = gi + goff;
                if (!col_ok || gi >= row_end) continue;
                const bool row_out = has_out && gg >= R && gg < n - R;
                uint64_t o[CPT];
                if (row_out) {
                    load_out_row(r, o);
                    apply_row(r, o);
                }
                store_row(r, o, row_out);
            }
            return;
        }
    }
    if constexpr (one_application(STEPS)) {
        // one pass: each row's new out and in_next leave as soon as they are computed. OUT_HBM_AHEAD:
        // every row's out words are requested first, so that their latencies overlap instead of
        // stalling each row in turn.
        constexpr bool PRELOAD = OUT_SRC == OUT_HBM_AHEAD && EXACT;
        uint64_t o_pre[PRELOAD ? ROWS : 1][CPT];
        if constexpr (PRELOAD) {
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                const int r = warp * ROWS + rr;
                const int64_t gi = i0 + r, gg = gi + goff;
                const bool row_out = col_ok && gi < row_end && has_out && gg >= R && gg < n - R;
                if (row_out) {
                    load_out_row(r, o_pre[rr]);
                } else {
#pragma unroll
                    for (int k = 0; k < CPT; ++k) o_pre[rr][k] = 0ull;
                }
            }
        }
        if constexpr (ROUTE) {
            if (inted) {  // a loop of its own, so that neither route's registers burden the other
                float si[ROWS][CPT] = {};  // M * S of the thread's points
                if (has_out)
                    int_rows<P, R, CPT, ROWS, G::RA>(s_in + (warp * ROWS + R) * G::SW + G::RA + c0, G::SW, si);
#pragma unroll
                for (int rr = 0; rr < ROWS; ++rr) {
                    const int r = warp * ROWS + rr;
                    const int64_t gi = i0 + r, gg = gi + goff;
                    if (!col_ok || gi >= row_end) continue;
                    const bool row_out = has_out && gg >= R && gg < n - R;
                    uint64_t o[CPT];
                    if (row_out) {
                        load_out_row(r, o);
#pragma unroll
                        for (int k = 0; k < CPT; ++k) int_add<P, R>(o[k], si[rr][k], 0.0f);
                    }
                    store_row(r, o, row_out);
                }
                return;
            }
        }
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp * ROWS + rr;
            const int64_t gi = i0 + r, gg = gi + goff;
            if (!col_ok || gi >= row_end) continue;
            const bool row_out = out_via_rows && has_out && gg >= R && gg < n - R;
            uint64_t o[CPT];
            if (row_out) {
                if constexpr (PRELOAD) {
#pragma unroll
                    for (int k = 0; k < CPT; ++k) o[k] = o_pre[rr][k];
                } else {
                    load_out_row(r, o);
                }
                if (!tbl_done) apply_row(r, o);
            }
            store_row(r, o, row_out);
        }
    } else if constexpr (DT == FP32C) {
        static_assert(G::ELEMS % 4 == 0, "the in-place advance moves 16-byte vectors");
        if (ROUTE && inted) {
            // The integer route: M * S of every application summed exactly, out read and updated once
            // at the end. `sums` applications fit the FP32 sum; it then goes to an integer.
            // The in += 1 of the thread's own points from the values its sums have just read, the halo beside
            // them; a pass over the whole tile where the extra registers cost more (n=8192, whole runs,
            // us per application: star R=1 47 to 43, R=2 51 to 48; launches of eight, R=5 85 to 88; whole
            // runs of 50 of the star grids of a batch of 256, which are evaluated in calls: 12.98 ms with it,
            // 10.84 without).
            constexpr bool FUSED_ADVANCE = P == STAR && R <= 2 && OUT_SRC != OUT_HBM;
            float a[ROWS][CPT] = {};
            int acc[ROWS][CPT] = {};
            int held = 0;
#pragma unroll 1
            for (int t = 0; t < nsteps; ++t) {
                if (held == sums) {
                    held = 0;
#pragma unroll
                    for (int rr = 0; rr < ROWS; ++rr)
#pragma unroll
                        for (int k = 0; k < CPT; ++k) {
                            acc[rr][k] += __float2int_rn(a[rr][k]);
                            a[rr][k] = 0.0f;
                        }
                }
                ++held;
                float* const mine = s_in + (warp * ROWS + R) * G::SW + G::RA + c0;
                float own[ROWS][CPT];
                if (has_out) int_rows<P, R, CPT, ROWS, G::RA>(mine, G::SW, a, FUSED_ADVANCE ? own : nullptr);
                if (t + 1 < nsteps) {  // in += 1
                    __syncthreads();
                    if (FUSED_ADVANCE && has_out) {
#pragma unroll
                        for (int rr = 0; rr < ROWS; ++rr) {
#pragma unroll
                            for (int k = 0; k < CPT; ++k) own[rr][k] = __fadd_rn(own[rr][k], 1.0f);
                            st_vec(mine + rr * G::SW, own[rr]);
                        }
                        advance_halo_f32<G::SW, G::SH, R, G::RA>(s_in, s_in);
                    } else {
                        advance_f32<G::ELEMS>(s_in);
                    }
                    __syncthreads();
                }
            }
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr)
#pragma unroll
                for (int k = 0; k < CPT; ++k) acc[rr][k] += __float2int_rn(a[rr][k]);
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                const int r = warp * ROWS + rr;
                const int64_t gi = i0 + r, gg = gi + goff;
                if (!col_ok || gi >= row_end) continue;
                const bool row_out = has_out && gg >= R && gg < n - R;
                uint64_t o[CPT];
                if (row_out) {
                    load_out_row(r, o);
#pragma unroll
                    for (int k = 0; k < CPT; ++k) {
                        const int t = acc[rr][k];
                        const float th = __int2float_rn(t);
                        int_add<P, R>(o[k], th, __int2float_rn(t - __float2int_rn(th)));
                    }
                }
                store_row(r, o, row_out);
            }
            return;
        }
        // The group sums: out stays in registers, accumulated without renormalising. As floats, not in the
        // loop of FP64 words below: there the two routes together spilled (n=8192, real values, eight
        // applications, us per application: star R=4 151 to 141, grid R=4 377 to 330; on the loop of
        // words without the integer route 144 and 353).
        float oh[ROWS][CPT], ol[ROWS][CPT];
        bool ract[ROWS];  // the row holds interior points
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp * ROWS + rr;
            const int64_t gi = i0 + r, gg = gi + goff;
            ract[rr] = col_ok && gi < row_end && has_out && gg >= R && gg < n - R;
#pragma unroll
            for (int k = 0; k < CPT; ++k) oh[rr][k] = ol[rr][k] = 0.0f;
            if (ract[rr]) load_pairs(r, oh[rr], ol[rr]);
        }
#pragma unroll 1
        for (int t = 0; t < nsteps; ++t) {
            if (t > 0) {  // in += 1 over the whole tile, halo included
                __syncthreads();
                advance_f32<G::ELEMS>(s_in);
                __syncthreads();
            }
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr) {
                if (!ract[rr]) continue;
                float sh[CPT], sl[CPT];
                fp32c_points<P, R, CPT, G::RA>(s_in + (warp * ROWS + rr + R) * G::SW + G::RA + c0, G::SW, sh, sl);
#pragma unroll
                for (int k = 0; k < CPT; ++k) df_add_lazy(oh[rr][k], ol[rr][k], sh[k], sl[k]);
            }
        }
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp * ROWS + rr;
            if (!col_ok || i0 + r >= row_end) continue;
            uint64_t o[CPT];
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                float h, l;
                fast_two_sum(oh[rr][k], ol[rr][k], h, l);
                o[k] = static_cast<uint64_t>(__float_as_uint(h)) | (static_cast<uint64_t>(__float_as_uint(l)) << 32);
            }
            store_row(r, o, ract[rr]);
        }
    } else {
        static_assert(G::ELEMS % 4 == 0, "the in-place advance moves 16-byte vectors");
        // out of the thread's points stays in registers across the applications
        uint64_t o[ROWS][CPT];
        bool ract[ROWS];  // the row holds interior points
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp * ROWS + rr;
            const int64_t gi = i0 + r, gg = gi + goff;
            ract[rr] = out_via_rows && col_ok && gi < row_end && has_out && gg >= R && gg < n - R;
            if (ract[rr]) {
                load_out_row(r, o[rr]);
            } else {
#pragma unroll
                for (int k = 0; k < CPT; ++k) o[rr][k] = 0ull;
            }
        }
        if constexpr (EXACT) {
            // FP32 route: when every out word the tile stores is an integer V of 2^-SHIFT units with
            // |V| < 2^21, out is held as V. Every S is an integer below 2^24 units, so each binary64
            // add of the reference chain (out + S) is exact (the running V stays below 2^28 for 8
            // applications, int32, and below 2^41 for FP32_MAX_STEPS, int64) and its conversion at
            // the end gives the same bits; a zero comes out +0 both ways (S is never -0). The
            // applications then add integers instead of issuing binary64 adds.
            if (fexact) {
                constexpr int SHIFT = pow2_shift(P, R);
                int32_t V[ROWS][CPT];
                bool ok = true;
#pragma unroll
                for (int rr = 0; rr < ROWS; ++rr) {
#pragma unroll
                    for (int k = 0; k < CPT; ++k) {
                        const bool fits = out_units(o[rr][k], SHIFT, V[rr][k]);
                        const bool stored = ract[rr] && gj + k >= R && gj + k < n - R;
                        ok = ok && (!stored || fits);
                    }
                }
                oint = __syncthreads_and(ok) != 0;
                if (oint) {
#pragma unroll
                    for (int rr = 0; rr < ROWS; ++rr)
#pragma unroll
                        for (int k = 0; k < CPT; ++k) {
                            if constexpr (STEPS == 0)
                                o[rr][k] = static_cast<uint64_t>(static_cast<int64_t>(V[rr][k]));
                            else  // V in the low word, high word zero
                                o[rr][k] = static_cast<uint32_t>(V[rr][k]);
                        }
                }
            }
        }
        bool fast = false;  // the FP32 route with integer-held out (block-uniform)
        if constexpr (EXACT) fast = fexact && oint;
        if (fast) {
            // The same applications in their tightest form: the route is fixed for the launch, and
            // a thread's S for all its rows comes from one pass over its column strip. The FP32
            // tile takes half of the binary64 stage, so the other half holds the next
            // application's in: while application t reads one, in + 1 is written to the other (each
            // thread its own points, from the values it has just read, and the threads together
            // the halo), and one barrier per application separates them.
            if constexpr (EXACT) {
                float* const buf = reinterpret_cast<float*>(s_in);
                const int own = (warp * ROWS + R) * G::SW + G::RA + c0;
#pragma unroll 1
                for (int t = 0; t < nsteps; ++t) {
                    const int cur = (t & 1) * G::ELEMS;
                    float S[ROWS][CPT], v[ROWS][CPT];
                    fexact_rows<P, R, CPT, ROWS, G::RA>(buf + cur + own, G::SW, S, v);
                    if (t + 1 < nsteps) {
                        float* nx = buf + (G::ELEMS - cur);
#pragma unroll
                        for (int rr = 0; rr < ROWS; ++rr) {
                            static_assert(CPT == 2, "own points move as one 8-byte pair");
                            *reinterpret_cast<float2*>(nx + own + rr * G::SW) =
                                make_float2(__fadd_rn(v[rr][0], 1.0f), __fadd_rn(v[rr][1], 1.0f));
                        }
                        advance_halo_f32<G::SW, G::SH, R, G::RA>(buf + cur, nx);
                        __syncthreads();
                    }
#pragma unroll
                    for (int rr = 0; rr < ROWS; ++rr)
#pragma unroll
                        for (int k = 0; k < CPT; ++k) {
                            if constexpr (STEPS == 0)
                                o[rr][k] += static_cast<uint64_t>(static_cast<int64_t>(__float2int_rn(S[rr][k])));
                            else
                                o[rr][k] = static_cast<uint32_t>(static_cast<uint32_t>(o[rr][k]) +
                                                                 static_cast<uint32_t>(__float2int_rn(S[rr][k])));
                        }
                }
                fin_off = ((nsteps - 1) & 1) * G::ELEMS;
            }
        } else if (!tbl_done) {
#pragma unroll 1
        for (int t = 0; t < nsteps; ++t) {
            if (t > 0) {  // advance the whole tile, halo included: in_{k+1} = in_k + 1
                __syncthreads();
                bool adv = false;
                if constexpr (EXACT) {
                    if (fexact) {
                        advance_f32<G::ELEMS>(reinterpret_cast<float*>(s_in));
                        adv = true;
                    } else if (unit != fx::NOT_FIXED) {
                        advance_i64<G::ELEMS>(reinterpret_cast<int64_t*>(s_in), 1ll << (-unit));
                        adv = true;
                    }
                }
                if constexpr (!EXACT) {
                    if (iwhole) {
                        advance_i32<G::ELEMS>(reinterpret_cast<int32_t*>(s_in));
                        adv = true;
                    }
                }
                if (!adv) advance_f64<G::ELEMS>(s_in);
                __syncthreads();
            }
            if constexpr (PLANES) {
                if (real) {
                    if (t == 0) __syncthreads();  // every thread has its out words in registers
                    real_planes<P, R, INPLACE, G::ELEMS>(reinterpret_cast<double*>(s_in), p1);
                    __syncthreads();
#pragma unroll
                    for (int rr = 0; rr < ROWS; ++rr)
                        if (ract[rr]) fp64_row(warp * ROWS + rr, o[rr]);
                    continue;
                }
            }
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr)
                if (ract[rr]) apply_row(warp * ROWS + rr, o[rr]);
        }
        }
        if (oint) {
#pragma unroll
            for (int rr = 0; rr < ROWS; ++rr)
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    if constexpr (STEPS == 0)
                        o[rr][k] = fx::from_fixed(static_cast<int64_t>(o[rr][k]), -pow2_shift(P, R));
                    else
                        o[rr][k] = from_fixed32(static_cast<int32_t>(static_cast<uint32_t>(o[rr][k])), -pow2_shift(P, R));
                }
        }
#pragma unroll
        for (int rr = 0; rr < ROWS; ++rr) {
            const int r = warp * ROWS + rr;
            const int64_t gi = i0 + r, gg = gi + goff;
            if (!col_ok || gi >= row_end) continue;
            store_row(r, o[rr], out_via_rows && has_out && gg >= R && gg < n - R);
        }
    }
}

// Register budget: the single-application kernels keep as many tiles resident as shared memory
// allows, so that every SM has enough loads in flight; the multi-application kernels hold `out` in
// registers and run at most four tiles per SM.
template <int P, int R, int DT, int STEPS, int TH_>
constexpr int min_blocks()
{
    // the table route: as many 32-row tiles as strict_tiles says (n=8192, four against three: star R=3 686
    // us per application against 765, its whole runs 430 against 463; grid R=2 865 against 937); tiles
    // whose shared memory admits at most two per SM get the registers of two (the 64-row tiles of grid
    // R=3..5)
    if (DT == FP64 && !pow2_weights(P, R)) {
        constexpr int fit = SMEM_PER_SM / (tile_smem<P, R, DT, TH_>() + 1024);
        return fit < 3 ? 2 : (fit < strict_tiles<P, R>() ? fit : strict_tiles<P, R>());
    }
    // FP32C grid R >= 3: three tiles per SM (80 registers). n=8192, us per application against two tiles, one
    // application: grid R=3 257 against 303 on whole numbers and 286 against 369 on reals, R=5 376 against
    // 432 and 560 against 596; whole runs: R=4 150 against 155 and 332 against 337. The group sums of grid
    // R=5 hold 72 values per thread and want the registers of two tiles in several applications (whole
    // runs: 502 against 550 on reals, 227 against 219 on whole numbers; launches of two do not, 531 and 523
    // on reals, 305 and 335).
    if (DT == FP32C && P == GRID && R >= 3) {
        constexpr int most = R == 5 && !one_application(STEPS) && STEPS != 2 ? 2 : 3;
        return Geo<DT, R, TH_>::CTAS < most ? Geo<DT, R, TH_>::CTAS : most;
    }
    const int b = Geo<DT, R, TH_>::CTAS;
    if (one_application(STEPS)) return b;
    const int cap = DT == FP64 ? 4 : 3;  // FP64 power-of-two: the FP32 route is shared-memory bound
    return b < cap ? b : cap;
}

// One CTA per tile: blockIdx = (tile column, tile row). The elected thread issues the tile's two TMA
// loads; every thread waits on the mbarrier with a bounded spin, and on a timeout the CTA flags
// `status`, waits (again bounded) for the copies to land and returns. The arrays hold rows of the
// n x n grid from grid row goff (the tensor maps cover exactly the rows they hold, so the hardware
// zero-fills anything beyond); rows from row_end on are read as halo but not stored.
template <int P, int R, int DT, int STEPS, int TH_>
__global__ void __launch_bounds__(THREADS, min_blocks<P, R, DT, STEPS, TH_>())
    k_stencil_tile(const __grid_constant__ CUtensorMap tm_in, const __grid_constant__ CUtensorMap tm_out,
                   const int64_t n, void* in_next_v, void* out_v, unsigned* status,
                   const int depth, const int64_t row0, const int64_t goff, const int64_t row_end)
{
    using G = Geo<DT, R, TH_>;
    using C = Cfg<DT, TH_>;
    extern __shared__ __align__(128) unsigned char smem[];
    int* s_red = reinterpret_cast<int*>(smem + G::RED_OFF);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + G::BAR_OFF);
    const int64_t i0 = row0 + static_cast<int64_t>(blockIdx.y) * C::TH;
    const int64_t j0 = static_cast<int64_t>(blockIdx.x) * C::TW;
    const bool has_out = tile_has_out(i0 + goff, j0, n, R, C::TW, C::TH);

    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    chain_wait();
    if (threadIdx.x == 0) {
        mbar_arrive_expect_tx(bar, G::IN_BYTES + (has_out ? G::OUT_BYTES : 0));
        tma_load_2d(smem, &tm_in, static_cast<int32_t>(j0 - G::RA), static_cast<int32_t>(i0 - R), bar);
        if (has_out) tma_load_2d(smem + G::OUT_OFF, &tm_out, static_cast<int32_t>(j0), static_cast<int32_t>(i0), bar);
    }
    __syncthreads();
    // One decision for the whole CTA: process_tile's barriers need every thread, so the tile is
    // evaluated only when every thread saw the loads land.
    if (!__syncthreads_and(mbar_wait_bounded(bar, 0))) {
        if (threadIdx.x == 0) atomicOr(status, 1u);
        mbar_wait_bounded(bar, 0);  // let the copies land before the CTA's shared memory is released
        return;
    }
    // process_tile may put a plane of products over the barrier, several block barriers further on
    if (table_route<P, R, DT>() && threadIdx.x == 0) mbar_inval(bar);
    process_tile<P, R, DT, STEPS, OUT_SMEM, TH_>(smem, s_red, i0, j0, n, has_out, in_next_v, out_v, true, depth, goff,
                                                 row_end,
                                                 table_route<P, R, DT>() ? smem + table_offset<DT, R, TH_>() : nullptr);
}

template <int P, int R, int DT, int STEPS, int TH_>
cudaError_t launch(const Launch& L)
{
    using C = Cfg<DT, TH_>;
    constexpr int SMEM = tile_smem<P, R, DT, TH_>();
    static_assert(SMEM <= SMEM_PER_CTA_MAX, "the tile and its tables must fit in shared memory");
    if constexpr (SMEM > SMEM_DEFAULT_MAX)
        if (cudaError_t e = cudaFuncSetAttribute(k_stencil_tile<P, R, DT, STEPS, TH_>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM))
            return e;
    const int64_t nr = L.nr > 0 ? L.nr : L.n;
    if (L.row0 < 0 || L.row0 >= nr || L.rows < 0 || (STEPS == 0 && L.depth < 1) || L.goff < 0 || L.goff + nr > L.n)
        return cudaErrorInvalidValue;
    const int64_t rows = L.rows > 0 && L.rows < nr - L.row0 ? L.rows : nr - L.row0;
    const int64_t tx = (L.n + C::TW - 1) / C::TW, ty = (rows + C::TH - 1) / C::TH;
    if (ty > 65535) return cudaErrorInvalidValue;
    const dim3 grid(static_cast<unsigned>(tx), static_cast<unsigned>(ty));
    return launch_chained(k_stencil_tile<P, R, DT, STEPS, TH_>, grid, THREADS, SMEM, L.stream, L.tm_in, L.tm_out, L.n,
                          L.in_next, L.out, L.status, L.depth, L.row0, L.goff, L.row0 + rows);
}

// Supported temporal depths; a run of any length is split into launches of these, or runs in one
// launch of the run-time-depth kernel (steps = 0, TH = 32 only).
constexpr int MAX_STEPS = 8;

template <int P, int DT, int TH_>
cudaError_t launch_pattern(int R, int steps, const Launch& L)
{
#define PRK_TILE_CASE(RR)                                        \
    case RR:                                                     \
        switch (steps) {                                         \
        case 1: return launch<P, RR, DT, 1, TH_>(L);             \
        case 2: return launch<P, RR, DT, 2, TH_>(L);             \
        case 4: return launch<P, RR, DT, 4, TH_>(L);             \
        case 8: return launch<P, RR, DT, 8, TH_>(L);             \
        case 0:                                                  \
            if constexpr (TH_ == TH_DEFAULT)                     \
                return launch<P, RR, DT, 0, TH_>(L);             \
            else                                                 \
                return cudaErrorInvalidValue;                    \
        case OPERATOR:                                           \
            if constexpr (TH_ == TH_DEFAULT)                     \
                return launch<P, RR, DT, OPERATOR, TH_>(L);      \
            else                                                 \
                return cudaErrorInvalidValue;                    \
        default: return cudaErrorInvalidValue;                   \
        }
    switch (R) {
        PRK_TILE_CASE(1)
        PRK_TILE_CASE(2)
        PRK_TILE_CASE(3)
        PRK_TILE_CASE(4)
        PRK_TILE_CASE(5)
    }
#undef PRK_TILE_CASE
    return cudaErrorInvalidValue;
}

// Tile geometry for the host: box sizes of the two tensor maps for tile height th.
inline void boxes(int dtype, int R, int th, int* in_x, int* in_y, int* out_x, int* out_y)
{
    const int vec = dtype == FP64 ? 2 : 4;
    const int ra = ((R + vec - 1) / vec) * vec;
    const int tw = dtype == FP64 ? Cfg<FP64>::TW : Cfg<FP32C>::TW;
    *in_x = tw + 2 * ra;
    *in_y = th + 2 * R;
    *out_x = tw;
    *out_y = th;
}

// Per-translation-unit entry points (tile_*.cu), one per storage form, pattern and tile height.
cudaError_t launch_fp64_star(int R, int steps, const Launch& L);
cudaError_t launch_fp64_grid(int R, int steps, const Launch& L);
cudaError_t launch_fp32c_star(int R, int steps, const Launch& L);
cudaError_t launch_fp32c_grid(int R, int steps, const Launch& L);
cudaError_t launch_fp64_star_tall(int R, int steps, const Launch& L);
cudaError_t launch_fp64_grid_tall(int R, int steps, const Launch& L);
cudaError_t launch_fp32c_star_tall(int R, int steps, const Launch& L);
cudaError_t launch_fp32c_grid_tall(int R, int steps, const Launch& L);

}  // namespace tile
}  // namespace prk
