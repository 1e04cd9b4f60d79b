// w^(1/gamma) / w as a pair of floats, and a channel times it rounded as the FP64
// product rounds. The reference evaluates the factor in FP64 (assets/kernels/
// tonemap.cu:67-104), which this part runs at 1/64 of the FP32 rate. In pairs of FP32
// numbers it is within kPowPairError of the exact value: where no float boundary lies
// within that of the product, the FP64 product rounds to the same float, and the few
// channels left (1 in 350) are for FP64 itself.
//   w = 2^e m, m in [sqrt(1/2), sqrt(2)): ln m = 2 atanh(s), s = (m - 1) / (m + 1),
//   by its power series; y = (1/gamma - 1) log2 w = n + j / 32 + f; 2^y = 2^n
//   2^(j / 32) e^(f ln 2) with the table's 2^(j / 32) and a quartic in f ln 2.
// Products that an addition follows are pp_mul, which is not contracted. Plain C++
// where there is no CUDA compiler (compiled with -ffp-contract=off), so that the
// error can be measured without a GPU.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define RFK_PP_FN __device__ __forceinline__
#else
#include <cstring>
#define RFK_PP_FN inline
struct float2 {
    float x, y;
};
#endif

namespace rfk_tm {

#ifdef __CUDACC__
RFK_PP_FN unsigned pp_bits(float v) { return __float_as_uint(v); }
RFK_PP_FN float pp_float(unsigned u) { return __uint_as_float(u); }
RFK_PP_FN float pp_mul(float a, float b) { return __fmul_rn(a, b); }
RFK_PP_FN float pp_div(float a, float b) { return __fdividef(a, b); }  // 2 ulp
RFK_PP_FN int pp_int(float v) { return __float2int_rn(v); }
#else
using std::fmaf;
RFK_PP_FN unsigned pp_bits(float v) {
    unsigned u;
    std::memcpy(&u, &v, 4);
    return u;
}
RFK_PP_FN float pp_float(unsigned u) {
    float v;
    std::memcpy(&v, &u, 4);
    return v;
}
RFK_PP_FN float pp_mul(float a, float b) { return a * b; }
float pp_div(float a, float b);  // any quotient within 2 ulp
RFK_PP_FN int pp_int(float v) { return (int)std::nearbyint(v); }
#endif

// Relative error of the pair for gamma >= 1/2 (the logarithm's error enters times
// 1/gamma - 1): 2^-34.4 at most over every significand at 60 exponents and 8 gammas from
// 1/2 to 1000, with quotients up to 2 ulp off.
constexpr float kPowPairError = 1.1641532182693481e-10f;  // 2^-33
constexpr float kPowPairGamma = 0.5f;                     // the least gamma

struct pow_table {
    float2 t[32];  // 2^(j / 32) as a pair
    float2 q;      // 1 / gamma - 1 as a pair
};

RFK_PP_FN bool pow_pair(float w, const float2* table, float2 q, float& hi, float& lo) {
    const unsigned u = pp_bits(w);
    if (u - 0x00800000u >= 0x7f800000u - 0x00800000u) return false;  // negative, zero, subnormal, infinite, NaN
    const int e = (int)(u - 0x3f3504f3u) >> 23;
    const float m = pp_float(u - ((unsigned)e << 23));
    const float num = m - 1.0f, dh = m + 1.0f, dl = m - (dh - 1.0f);
    const float sh = pp_div(num, dh);
    const float sl = pp_div(fmaf(-sh, dl, fmaf(-sh, dh, num)), dh);
    const float s2h = pp_mul(sh, sh), s2l = fmaf(2.0f * sh, sl, fmaf(sh, sh, -s2h));
    float p = fmaf(1.0f / 15, s2h, 1.0f / 13);
    p = fmaf(p, s2h, 1.0f / 11);
    p = fmaf(p, s2h, 1.0f / 9);
    p = fmaf(p, s2h, 1.0f / 7);
    p = fmaf(p, s2h, 0.2f);
    const float third = (float)(1.0 / 3), third_l = (float)(1.0 / 3 - (double)third);
    const float c = pp_mul(s2h, p), ch = third + c, cl = (c - (ch - third)) + third_l;
    const float uh = pp_mul(s2h, ch), ul = fmaf(s2l, ch, fmaf(s2h, cl, fmaf(s2h, ch, -uh)));
    const float vh = 1.0f + uh, vl = (uh - (vh - 1.0f)) + ul;
    const float lh = pp_mul(sh, vh), ll = fmaf(sl, vh, fmaf(sh, vl, fmaf(sh, vh, -lh)));
    constexpr double k2 = 2.8853900817779268147;  // 2 / ln 2
    const float kh = (float)k2, kl = (float)(k2 - (double)kh);
    const float gh = pp_mul(lh, kh), gl = fmaf(ll, kh, fmaf(lh, kl, fmaf(lh, kh, -gh)));
    const float ef = (float)e, th = ef + gh, tl = (gh - (th - ef)) + gl;
    const float yh = pp_mul(th, q.x), yl = fmaf(tl, q.x, fmaf(th, q.y, fmaf(th, q.x, -yh)));
    if (!(fabsf(yh) < 120.0f)) return false;
    const int n = pp_int(yh * 32.0f);
    const float f = fmaf((float)n, -1.0f / 32, yh), g = f + yl, fl = yl - (g - f);
    constexpr double l2 = 0.69314718055994530942;
    const float l2h = (float)l2, l2l = (float)(l2 - (double)l2h);
    const float rh = pp_mul(g, l2h), rl = fmaf(fl, l2h, fmaf(g, l2l, fmaf(g, l2h, -rh)));
    const float r2 = fmaf(pp_mul(rh, rh), fmaf(rh, fmaf(rh, 1.0f / 24, 1.0f / 6), 0.5f), rl);
    const float2 t = table[n & 31];
    const float ph = pp_mul(t.x, rh), pl = fmaf(t.x, r2, fmaf(t.x, rh, -ph)) + fmaf(t.y, rh, t.y);
    const float z = t.x + ph, zl = (ph - (z - t.x)) + pl;
    const float scale = pp_float((unsigned)(127 + (n >> 5)) << 23);
    hi = z * scale;
    lo = zl * scale;
    return true;
}

// (float)(col * factor) for the factor in 64 bits that hi + lo stands for; false where
// the pair's error leaves two floats, or the product is not a normal number.
RFK_PP_FN bool scale_pair(float col, float hi, float lo, float& out) {
    const float p = pp_mul(col, hi), size = fabsf(p);
    const float r = fmaf(col, lo, fmaf(col, hi, -p)), d = size * kPowPairError;
    out = p + (r - d);
    if (col == 0.0f) out = p;
    return col == 0.0f || (out == p + (r + d) && size >= 1e-30f && size <= 1e30f);
}

inline pow_table make_pow_table(float gamma) {
    static const pow_table powers = [] {
        pow_table p{};
        for (int j = 0; j < 32; j++) {
            const double v = std::exp2(j / 32.0);
            p.t[j].x = (float)v;
            p.t[j].y = (float)(v - (double)p.t[j].x);
        }
        return p;
    }();
    pow_table p = powers;
    const double q = 1.0 / (double)gamma - 1.0;
    p.q.x = (float)q;
    p.q.y = (float)(q - (double)p.q.x);
    return p;
}

}  // namespace rfk_tm
