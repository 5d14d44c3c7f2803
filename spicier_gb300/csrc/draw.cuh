// Per-sample parameter draws (sp_draw_kind) on the device.
#pragma once
#include <math_constants.h>

#include "circuit_dev.cuh"
#include "rng.cuh"

namespace sp {

// One drawn value.  gaussian_scaled = mean + z * sigma (rng.rs:148-150), two
// roundings; no product is fused into a sum in any translation unit.
__device__ inline double draw_one(const sp_param& p, uint64_t seed, uint32_t sweep, const double* row, unsigned* hard) {
    switch (p.kind) {
        case SP_DRAW_FIXED: return p.a;
        case SP_DRAW_GAUSS: return __dadd_rn(p.a, __dmul_rn(rng_gaussian(seed, sweep, p.rng_index, hard), p.b));
        case SP_DRAW_UNIFORM:
            return __dadd_rn(p.a, __dmul_rn(rng_uniform(seed, sweep, p.rng_index), __dsub_rn(p.b, p.a)));
        case SP_DRAW_LOGUNIFORM:
            return __dmul_rn(p.a, cr_exp(__dmul_rn(rng_uniform(seed, sweep, p.rng_index), cr_log(p.b / p.a, hard)), hard));
        case SP_DRAW_TABLE: return row ? row[p.rng_index] : CUDART_NAN;
    }
    return CUDART_NAN;
}

// The FP32 rounding of a Gaussian draw without the draw's 53 bits.
//
// Its consumer (the double-float Newton kernel) rounds every drawn parameter to
// FP32, so the correctly rounded FP64 ln and cos are needed only where that
// rounding is in doubt.  Here G = mean + sqrt(-2 ln u1) cos(2 pi u2) sigma is
// formed as an FP32 pair from 32-bit integer series on the same tables:
//
//   -ln u1  2^-56 fixed point, error below 2^-45 (r to 2^-40 in the series'
//           second-order term, which r^5 ends: the next one is 2^-50)
//   cos     2^-61 fixed point, error below 2^-38.5 (d = a - j/512 to 2^-41);
//           the FP64 path's rounded 2 pi u2 moves it by less than 2^-50
//   then the square root, both products and the sum on FP32 pairs, 2^-44
//
// so that |G - the FP64 draw| < eps = sigma (s 2^-37 + 2^-42 / s) + (|mean| + |G|) 2^-45
// with s the square root: about three times the sum of those bounds.  When G - eps
// and G + eps round to the same FP32 number, that is the rounding of the FP64
// draw; otherwise (about 3 draws in 10^5 of the op-amp's), within 2^-14 of
// u1 = 1, below u1 = 1.2e-10 (where the draw clamps) and for means or sigmas
// far from 1, false: the caller draws in full.
//
// About 256 instructions where the full draw takes 880; 65,536 x 17 draws:
// 44 -> 18 us under ncu.  ms: mean and sigma as FP32 pairs (NaN sigma: never decided).
template <class Probe = void>
__device__ __forceinline__ bool gauss_f32(uint64_t base, uint64_t pk1, uint64_t pk2, float4 ms, float* out, Probe* probe = nullptr) {
    const uint64_t D = splitmix64(base ^ pk1) >> 11;
    const uint64_t H = splitmix64(base ^ pk2) & ~0x7ffULL;
    // -ln u1, u1 = m 2^-ae with m in [1, 2)
    const int lz = __clzll((long long)D);
    const uint64_t mant = D << (lz - 11);
    const int ae = lz - 10;
    const ulonglong2 row =
        __ldg(reinterpret_cast<const ulonglong2*>(&cr::kLnRowsDev[(uint32_t)(mant >> 44) & 0xffu]));  // c, -ln c 2^56
    const uint64_t r0 = mant * row.x;                      // r 2^68
    const uint32_t R = (uint32_t)(r0 >> 28);                 // r 2^40
    uint32_t h = 0x33333333u;                                // 1/5 - in Q0.32
    h = 0x40000000u - (__umulhi(R, h) >> 8);
    h = 0x55555555u - (__umulhi(R, h) >> 8);
    h = 0x80000000u - (__umulhi(R, h) >> 8);                 // 1/2 - r/3 + r^2/4 - r^3/5
    const uint32_t q2 = __umulhi(__umulhi(R, R), h);         // r^2 (...) 2^48
    const uint64_t lnm = row.y + (r0 >> 12) - ((uint64_t)q2 << 8);
    const uint64_t ln2w[2] = {SP_CR_LN2};
    const uint64_t L = ln2w[0] * (uint64_t)(uint32_t)ae - lnm;  // 2^-56 units
    // s = sqrt(2 L) as an FP32 pair
    const float lh = __fmul_rn((float)(uint32_t)(L >> 37), 0x1p-18f), ll = __fmul_rn((float)(uint32_t)(L >> 5), 0x1p-50f);
    const float lf = __fadd_rn(lh, ll), le = __fsub_rn(ll, __fsub_rn(lf, lh));
    float y0;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(lf));
    const float s0 = __fmul_rn(lf, y0);
    const float s1 = __fmul_rn(__fmul_rn(0.5f, y0), __fadd_rn(__fmaf_rn(-s0, s0, lf), le));
    // cos(2 pi u2): quadrant, fold to a in [0, pi/4], a = j/512 + d
    const uint32_t quad = (uint32_t)(H >> 62);
    const uint64_t f = H << 2;
    const bool fold = (long long)f < 0;
    const uint64_t a63 = __umul64hi(fold ? 0 - f : f, 0xC90FDAA22168C234ULL);  // pi/2 2^63 times f
    const uint32_t d = (uint32_t)(a63 >> 22);                // d 2^41
    const uint32_t d2 = __umulhi(d, d);                      // d^2 2^50
    const uint32_t cm = (d2 >> 1) - (__umulhi(__umulhi(d2, d2), 178956971u) >> 18);  // 1 - cos d, 2^50
    const uint32_t sd = d - (__umulhi(__umulhi(d, d2), 715827883u) >> 18);           // sin d, 2^41
    const uint64_t* crow = reinterpret_cast<const uint64_t*>(&cr::kCosRowsDev[(uint32_t)(a63 >> 54)]);
    const uint64_t ch = __ldg(crow), sh = __ldg(crow + 2);   // cos and sin of j/512, 2^61
    const bool use_sin = ((quad & 1u) != 0) != fold;
    const uint64_t X = use_sin ? sh : ch, Y = use_sin ? ch : sh;
    const uint64_t xcm = ((uint64_t)(uint32_t)(X >> 30) * cm) >> 20, ysd = ((uint64_t)(uint32_t)(Y >> 30) * sd) >> 11;
    const uint64_t V = use_sin ? X - xcm + ysd : X - xcm - ysd;
    const float vh = __fmul_rn((float)(uint32_t)(V >> 37), 0x1p-24f), vl = __fmul_rn((float)(uint32_t)(V >> 5), 0x1p-56f);
    // z sigma + mean
    const float sg = __uint_as_float((quad == 1u || quad == 2u) ? 0xbf800000u : 0x3f800000u);
    const float ph = __fmul_rn(s0, vh);
    const float pe = __fmaf_rn(s1, vh, __fmaf_rn(s0, vl, __fmaf_rn(s0, vh, -ph)));
    const float sh32 = __fmul_rn(sg, ms.z), sl32 = __fmul_rn(sg, ms.w);
    const float gh = __fmul_rn(ph, sh32);
    const float ge = __fmaf_rn(pe, sh32, __fmaf_rn(ph, sl32, __fmaf_rn(ph, sh32, -gh)));
    const float S = __fadd_rn(ms.x, gh), bb = __fsub_rn(S, ms.x);
    const float err = __fadd_rn(__fsub_rn(ms.x, __fsub_rn(S, bb)), __fsub_rn(gh, bb));
    const float lo = __fadd_rn(err, __fadd_rn(ms.y, ge));
    const float hi = __fadd_rn(S, lo), rest = __fsub_rn(lo, __fsub_rn(hi, S));
    const float eps = __fmaf_rn(fabsf(ms.z), __fmaf_rn(s0, 0x1p-37f, __fmul_rn(y0, 0x1p-42f)),
                                __fmul_rn(__fadd_rn(fabsf(ms.x), fabsf(hi)), 0x1p-45f));
    const float up = __fadd_rn(hi, __fadd_rn(rest, eps)), down = __fadd_rn(hi, __fsub_rn(rest, eps));
    if constexpr (!std::is_void<Probe>::value) probe->set(hi, rest, eps);
    *out = up;
    return up == down && D >= (1ull << 20) && L - (1ull << 42) < (1ull << 61);  // (L may round below 0 at u1 = 1)
}

// What a sample's draws need beyond the circuit, and where its constants go.
struct RedrawArgs {
    uint64_t seed = 0, first_index = 0;
    const double* table = nullptr;
    uint32_t table_cols = 0;
    double* derived = nullptr;  // [num_derived][stride], or nullptr: the constants are there already
};

// The derived constants of one sample (derive_element's, of the elements that
// sweeps with FP32 draws have: R, C, L, V, I and Level-1 MOSFETs) from its
// draws in FP64: the fallback's, for the samples it takes over.
__device__ __noinline__ static void redraw_sample(const DevCircuit& c, const RedrawArgs& a, size_t stride, size_t s) {
    const double* row = a.table ? a.table + s * a.table_cols : nullptr;
    const uint32_t sweep = (uint32_t)(a.first_index + s);
    for (int e = 0; e < c.num_elements; ++e) {
        const sp_element& el = c.el[e];
        double* out = a.derived + (size_t)c.doff[e] * stride + s;
        const bool mos = el.kind == SP_EL_NMOS || el.kind == SP_EL_PMOS;
        double v[6];
        for (int f = 0; f < (mos ? 6 : 1); ++f) v[f] = draw_one(c.par[el.field[f]], a.seed, sweep, row, nullptr);
        out[0] = mos ? fabs(v[0]) : el.kind == SP_EL_R ? ieee_div(1.0, v[0]) : v[0];
        if (mos) {
            out[stride] = ieee_div(ieee_mul(ieee_mul(v[1], v[5]), v[3]), v[4]);  // ((kp nf) w) / l
            out[2 * stride] = v[2];
        }
    }
}

}  // namespace sp
