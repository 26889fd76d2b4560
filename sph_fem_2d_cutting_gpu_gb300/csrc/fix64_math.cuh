// fix64_math.cuh -- log2, exp2, pow and log of doubles, and the angle functions of the
// artificial stress, on the integer pipes.
//
// CUDA's double pow() is a chain of some hundred operations for the FP64 pipe, and
// a return mapping evaluates ten to twenty of them one after another: on a small
// system those chains are what the step waits for.  Here the same functions run in
// 64-bit fixed point (fix64.cuh): table-driven argument reduction and a short
// series, after P. T. P. Tang, "Table-driven implementation of the logarithm
// function in IEEE floating-point arithmetic" (ACM TOMS 16, 1990) and "... of the
// exponential function ..." (ACM TOMS 15, 1989), with series and tables of this
// file's own: log2 within 2 units of 2^-64, exp2 within 40 units of 2^-63
// (tests/test_fix64.py), so pow() is within 0.6 units in the last place on its range.
#pragma once

#include "fix64.cuh"

namespace sphfem {

// log2: the mantissa m in [1, 2) of interval i = floor(128 (m - 1)) times c_i =
// kLog2K[i] / 512, the smallest multiple of 1/512 with m c_i >= 1 there;
// kLog2T[i] = -log2(c_i) 2^64.  exp2: kExp2T[i] = 2^(i / 64) 2^63.
__device__ const uint16_t kLog2K[128] = {
    512, 509, 505, 501, 497, 493, 490, 486, 482, 479, 475, 472, 469, 465, 462, 459,
    456, 452, 449, 446, 443, 440, 437, 435, 432, 429, 426, 423, 421, 418, 415, 413,
    410, 408, 405, 403, 400, 398, 395, 393, 391, 388, 386, 384, 382, 379, 377, 375,
    373, 371, 369, 367, 365, 363, 361, 359, 357, 355, 353, 351, 349, 347, 345, 344,
    342, 340, 338, 337, 335, 333, 331, 330, 328, 327, 325, 323, 322, 320, 319, 317,
    316, 314, 313, 311, 310, 308, 307, 305, 304, 303, 301, 300, 298, 297, 296, 294,
    293, 292, 290, 289, 288, 287, 285, 284, 283, 282, 281, 279, 278, 277, 276, 275,
    274, 272, 271, 270, 269, 268, 267, 266, 265, 264, 263, 262, 261, 260, 259, 258,
};
__device__ const uint64_t kLog2T[128] = {
    0x0000000000000000ull, 0x022b9fd1d5d90603ull, 0x05159298864a0d18ull, 0x080573fa8160e1ceull,
    0x0afb5c508e1e308eull, 0x0df7648a8d561729ull, 0x10387efbca869da1ull, 0x133f7cde14cf59e2ull,
    0x164ce26c067156b4ull, 0x189b33091d6fe815ull, 0x1bb4102f925393c6ull, 0x1e0b1ae8f2fd5665ull,
    0x2065f775dcdaca19ull, 0x238fcefbbc67b716ull, 0x25f3c65ab7fba134ull, 0x285bba57436952a4ull,
    0x2ac7b853ff596419ull, 0x2e08c0638f3f097cull, 0x307e6099b8b54d72ull, 0x32f8396278fd810bull,
    0x35765953d8e8e4c6ull, 0x37f8cf4fffe9980eull, 0x3a7faa87495ab8f5ull, 0x3c31601c26247a0dull,
    0x3ebfb1520c7c6921ull, 0x415291d2fc3addfeull, 0x43ea120112cd4422ull, 0x4686429759d281a3ull,
    0x48465ba1d1cf42ccull, 0x4aea830d2f87afc0ull, 0x4d9389447320833cull, 0x4f5c4afe7277bb32ull,
    0x520d979a575e5aa9ull, 0x53dbeecb3b1661e4ull, 0x5695b5e8dc37b588ull, 0x5869c5f2b0660c45ull,
    0x5b2c3da19723a80eull, 0x5d062b3aefc63ad9ull, 0x5fd18b96385a20a1ull, 0x61b17cdb7a8f6eeaull,
    0x6393e0fe8517b6bfull, 0x666c1caa5b1ac9bdull, 0x6854bc50a606cf5full, 0x6a3fe5c604297860ull,
    0x6c2d9fd3d1a03fd4ull, 0x6f17152249532e75ull, 0x710b57131a22cf3cull, 0x7302423866def475ull,
    0x74fbdddb50ffcfc4ull, 0x76f831630f3fc696ull, 0x78f74455941f7763ull, 0x7af91e5838f02200ull,
    0x7cfdc7306d8a6e0bull, 0x7f0546c46cd9006eull, 0x810fa51bf65fd771ull, 0x831cea610ceafcbcull,
    0x852d1ee0ba90c6b0ull, 0x87404b0bda359fc8ull, 0x89567777e6c11bfbull, 0x8b6facdfd0360ab8ull,
    0x8d8bf424d6e130b2ull, 0x8fab564f6cd468ffull, 0x91cddc901de619a3ull, 0x92e050231df57d70ull,
    0x95079e1a0382dc79ull, 0x973227d6027ebd8aull, 0x995ff71b8773432dull, 0x9a781beb62fd91ccull,
    0x9caae63128f23953ull, 0x9ee10f309e79c8e1ull, 0xa11aa14eb954eea2ull, 0xa238b5160413106eull,
    0xa47778c98bcc86a2ull, 0xa5982b6dccad1e5dull, 0xa7dc392f5add49a4ull, 0xaa23db93321cd53cull,
    0xab49080ecda53209ull, 0xad961ed0cb91d407ull, 0xaebe0c048ac0f1adull, 0xb110b17d788c15aaull,
    0xb23b6cc56cc84c9aull, 0xb493bc0ec9954244ull, 0xb5c153293365f274ull, 0xb81f68249dc7b350ull,
    0xb94fe935b83e3eb6ull, 0xbbb3e094b3d228d4ull, 0xbce75a2aaf55c56cull, 0xbf515176cbe67114ull,
    0xc087d28dfb2febb9ull, 0xc1bf598dbee1b171ull, 0xc43180389d6fe23dull, 0xc56c23679b4d206eull,
    0xc7e492644d64237eull, 0xc92261d140d42d28ull, 0xca6143a49626d820ull, 0xcce245f1031e41faull,
    0xce246a2f95a92894ull, 0xcf67a85fa1f89a04ull, 0xd1f17a5621fb01acull, 0xd338120a6dd9d306ull,
    0xd47fcb8c0852f0c1ull, 0xd5c8a8df0b46eb6full, 0xd85dd724caeb3820ull, 0xd9aa2c3b0ea3cbc1ull,
    0xdaf7ad69f0b380e5ull, 0xdc465cd155a90943ull, 0xdd963c96edf3a402ull, 0xe03995f0f4ff5b70ull,
    0xe18d13ee805a4de3ull, 0xe2e1cb1ca47d25b3ull, 0xe437bdbf5254459cull, 0xe58eee20cb7b6c15ull,
    0xe6e75e91b9cca552ull, 0xe99c090536ece983ull, 0xeaf847c9fcc4492bull, 0xec55d022d80e3d28ull,
    0xedb4a481eca5c376ull, 0xef14c7605d60654cull, 0xf0763b3e66d6302full, 0xf1d902a37aaa5086ull,
    0xf33d201e5b5735d0ull, 0xf4a2964538813c67ull, 0xf60967b5cbd2ecf0ull, 0xf77197157665f689ull,
    0xf8db27115ebc1e66ull, 0xfa461a5e8f4b759dull, 0xfbb273ba15a13cedull, 0xfd2035e9221ef5d0ull,
};
__device__ const uint64_t kExp2T[64] = {
    0x8000000000000000ull, 0x8164d1f3bc030773ull, 0x82cd8698ac2ba1d7ull, 0x843a28c3acde4046ull,
    0x85aac367cc487b15ull, 0x871f61969e8d1010ull, 0x88980e8092da8527ull, 0x8a14d575496efd9aull,
    0x8b95c1e3ea8bd6e7ull, 0x8d1adf5b7e5ba9e6ull, 0x8ea4398b45cd53c0ull, 0x9031dc431466b1dcull,
    0x91c3d373ab11c336ull, 0x935a2b2f13e6e92cull, 0x94f4efa8fef70961ull, 0x96942d3720185a00ull,
    0x9837f0518db8a96full, 0x99e0459320b7fa65ull, 0x9b8d39b9d54e5539ull, 0x9d3ed9a72cffb751ull,
    0x9ef5326091a111aeull, 0xa0b0510fb9714fc2ull, 0xa27043030c496819ull, 0xa43515ae09e6809eull,
    0xa5fed6a9b15138eaull, 0xa7cd93b4e965356aull, 0xa9a15ab4ea7c0ef8ull, 0xab7a39b5a93ed337ull,
    0xad583eea42a14ac6ull, 0xaf3b78ad690a4375ull, 0xb123f581d2ac2590ull, 0xb311c412a9112489ull,
    0xb504f333f9de6484ull, 0xb6fd91e328d17791ull, 0xb8fbaf4762fb9ee9ull, 0xbaff5ab2133e45fbull,
    0xbd08a39f580c36bfull, 0xbf1799b67a731083ull, 0xc12c4cca66709456ull, 0xc346ccda24976407ull,
    0xc5672a115506daddull, 0xc78d74c8abb9b15dull, 0xc9b9bd866e2f27a3ull, 0xcbec14fef2727c5dull,
    0xce248c151f8480e4ull, 0xd06333daef2b2595ull, 0xd2a81d91f12ae45aull, 0xd4f35aabcfedfa1full,
    0xd744fccad69d6af4ull, 0xd99d15c278afd7b6ull, 0xdbfbb797daf23755ull, 0xde60f4825e0e9124ull,
    0xe0ccdeec2a94e111ull, 0xe33f8972be8a5a51ull, 0xe5b906e77c8348a8ull, 0xe8396a503c4bdc68ull,
    0xeac0c6e7dd24392full, 0xed4f301ed9942b84ull, 0xefe4b99bdcdaf5cbull, 0xf281773c59ffb13aull,
    0xf5257d152486cc2cull, 0xf7d0df730ad13bb9ull, 0xfa83b2db722a033aull, 0xfd3e0c0cf486c175ull,
};

// log2(m / 2^63) 2^64 for m in [2^63, 2^64) with 53 significant bits; 2^64 (log2 of
// nearly 2) cannot come out.
__device__ __forceinline__ uint64_t log2_frac(uint64_t m) {
    const int i = (int)(m >> 56) & 0x7f;
    const uint64_t S = ((m >> 9) * (uint64_t)__ldg(kLog2K + i) - (1ull << 63)) << 7;   // (64 r) 2^64, m c = 1 + r
    const uint32_t s = (uint32_t)(S >> 32);
    // ln(1 + r) / r = 1 - r (1/2 - r (1/3 - ... - r / 10)), the tail in 32 bits
    uint32_t h = 0x1c71c71cu - (__umulhi(s, 0x1999999au) >> 6);
    h = 0x20000000u - (__umulhi(s, h) >> 6);
    h = 0x24924925u - (__umulhi(s, h) >> 6);
    h = 0x2aaaaaabu - (__umulhi(s, h) >> 6);
    uint64_t H = 0x3333333333333333ull - (mul_hi(S, (uint64_t)h << 32) >> 6);
    H = 0x4000000000000000ull - (mul_hi(S, H) >> 6);
    H = 0x5555555555555555ull - (mul_hi(S, H) >> 6);
    H = 0x8000000000000000ull - (mul_hi(S, H) >> 6);
    H = ~0ull - (mul_hi(S, H) >> 6);
    return __ldg(kLog2T + i) + (mul_hi(mul_hi(S, H), 0xb8aa3b295c17f0bcull) >> 5);   // log2(e) 2^63
}

// 2^(F / 2^64) 2^63.
__device__ __forceinline__ uint64_t exp2_frac(uint64_t F) {
    const uint64_t T = __ldg(kExp2T + (int)(F >> 58));
    const uint64_t w = mul_hi(F << 6, 0xb17217f7d1cf79acull);   // (64 w) 2^64, w = ln 2 times the rest
    const uint32_t v = (uint32_t)(w >> 32);
    // (e^w - 1) / w = 1 + w (1/2 + w (1/6 + ... + w / 5040))
    uint32_t h = 0x5b05b0u + (__umulhi(v, 0xd00d0u) >> 6);
    h = 0x2222222u + (__umulhi(v, h) >> 6);
    h = 0xaaaaaabu + (__umulhi(v, h) >> 6);
    uint64_t H = 0x2aaaaaaaaaaaaaabull + (mul_hi(w, (uint64_t)h << 32) >> 6);
    H = 0x8000000000000000ull + (mul_hi(w, H) >> 6);
    return T + (mul_hi(T, w + mul_hi(w, mul_hi(w, H) >> 6)) >> 6);
}

// |log2(x)| of a positive normal x, its top bit set (or 0); negative: log2(x) < 0.
__device__ __forceinline__ Fix64 fix_log2(double x, bool &negative) {
    const Fix64 a = fix_of(x);
    int E = a.e + 63;
    uint64_t f = log2_frac(a.m);
    negative = E < 0;
    if (negative) {   // -(E + f) = (-E - 1) + (1 - f)
        E = -E - (f ? 1 : 0);
        f = 0ull - f;
    }
    const int b = 32 - __clz(E);   // bits of the integer part
    return fix_norm({b ? ((uint64_t)(uint32_t)E << (64 - b)) | (f >> b) : f, b - 64});
}

// 2^(+-y) for y < 2^11 with its top bit set (or 0).
__device__ __forceinline__ Fix64 fix_exp2(Fix64 y, bool negative) {
    int n = 0;
    uint64_t F;
    if (y.e > -64) {
        n = (int)(y.m >> -y.e);
        F = y.m << (64 + y.e);
    } else {
        F = y.e <= -128 ? 0ull : y.m >> (-64 - y.e);
    }
    if (negative) {
        n = -n - (F ? 1 : 0);
        F = 0ull - F;
    }
    return {exp2_frac(F), n - 63};
}

// a / b, correctly rounded: the 53-bit quotient of the mantissas from the reciprocal is
// within one unit, and the sign of its exact remainder settles it, as in fix_recip_rn;
// arguments beyond 2^+-64 (b) and 2^+-511 (a) divide on the FP64 pipe.
static __device__ __noinline__ double div_general(double a, double b) { return a / b; }
__device__ __forceinline__ double fix_div(double a, double b) {
    const uint64_t ab = (uint64_t)__double_as_longlong(a), bb = (uint64_t)__double_as_longlong(b);
    const uint32_t ah = (uint32_t)(ab >> 32) & 0x7fffffffu, bh = (uint32_t)(bb >> 32) & 0x7fffffffu;
    if (bh - 0x3bf00000u >= 0x08000000u || (ah - 0x20000000u >= 0x40000000u && flag_nonzero(a)))
        return div_general(a, b);
    const uint64_t A = (ab & 0xfffffffffffffull) | 0x10000000000000ull;
    const uint64_t B = (bb & 0xfffffffffffffull) | 0x10000000000000ull;
    const bool less = A < B;                             // a quotient in [1/2, 1), else in [1, 2)
    uint64_t q = (mul_hi(recip_mant(B) << (less ? 2 : 1), A << 11) + 512) >> 10;   // [2^52, 2^53]
    const long long rem = (long long)((A << (less ? 53 : 52)) - q * B);
    q += 2 * rem > (long long)B ? 1 : 2 * rem < -(long long)B ? -1 : 0;
    const uint64_t sign = (ab ^ bb) & 0x8000000000000000ull;
    const int e = (int)(ah >> 20) - (int)(bh >> 20) + (less ? 1022 : 1023);
    return __longlong_as_double((long long)(flag_nonzero(a) ? sign + ((uint64_t)(uint32_t)(e - 1) << 52) + q : sign));
}

// pow(x, n) for x > 0 and n in [2^-9, 2), within 0.6 units in the last place; other
// arguments, and results beyond 2^+-32, go to the library's pow(): n log2(x) has 64 bits, and
// nine of them before the point would cost the result 0.4 units.
static __device__ __noinline__ double pow_general(double x, double n) { return pow(x, n); }
__device__ __forceinline__ double fix_pow(double x, double n) {
    const uint32_t xh = (uint32_t)__double2hiint(x), nh = (uint32_t)__double2hiint(n);
    bool neg;
    const Fix64 l = fix_log2(x, neg);
    const Fix64 y = fix_norm(l * fix_abs(n));
    if (nh - 0x3f600000u >= 0x00a00000u || xh - 0x00100000u >= 0x7fe00000u || y.e + 63 >= 5) {
        if (nh - 0x3f600000u < 0x00a00000u && (xh | (uint32_t)__double2loint(x)) == 0u) return 0.;
        return pow_general(x, n);
    }
    return fix_double(fix_exp2(y, neg));
}

// log(x) for x > 1; infinities and NaN to the library's log().
static __device__ __noinline__ double log_general(double x) { return log(x); }
__device__ __forceinline__ double fix_log_above_1(double x) {
    bool neg;
    const Fix64 l = fix_log2(x, neg);
    if ((uint32_t)__double2hiint(x) >= 0x7ff00000u) return log_general(x);
    return fix_double(l * Fix64{0xb17217f7d1cf79acull, -64});
}

// pow(x, n), or for lanes with `lg` log(x) of x > 1: fix_pow and fix_log_above_1 with their
// common part formed once, for lanes that need either to stay together.
__device__ __forceinline__ double fix_pow_or_log(double x, double n, bool lg) {
    const uint32_t xh = (uint32_t)__double2hiint(x), nh = (uint32_t)__double2hiint(n);
    bool neg;
    const Fix64 l = fix_log2(x, neg);
    if (lg) return xh >= 0x7ff00000u ? log_general(x) : fix_double(l * Fix64{0xb17217f7d1cf79acull, -64});
    const Fix64 y = fix_norm(l * fix_abs(n));
    if (nh - 0x3f600000u >= 0x00a00000u || xh - 0x00100000u >= 0x7fe00000u || y.e + 63 >= 5) {
        if (nh - 0x3f600000u < 0x00a00000u && (xh | (uint32_t)__double2loint(x)) == 0u) return 0.;
        return pow_general(x, n);
    }
    return fix_double(fix_exp2(y, neg));
}

// ---- atan2, sin and cos of floats ------------------------------------------------------------
// The reference's atan2f, sinf and cosf, formed to 2^-57 and rounded once to float (the
// CPU restatement rounds its double functions once, too).  atan by one step to the
// nearest table angle below, tan(a - b) = (tan a - tan b) / (1 + tan a tan b), and
// five terms of its series; sin and cos by their series on [0, pi/4].
// kAtanT[i] = atan(i / 64) 2^63
__device__ const uint64_t kAtanT[64] = {
    0x0000000000000000ull, 0x01fff555bbb729abull, 0x03ffaab7752ec495ull, 0x05fee0610c368a7eull,
    0x07fd56edcb3f7a72ull, 0x09facf873e2aceb6ull, 0x0bf70c1301788746ull, 0x0df1cf5f3783e1bfull,
    0x0feadd4d5617b6e3ull, 0x11e1fafb043726e5ull, 0x13d6eee8c6626c58ull, 0x15c9811e3ec269dfull,
    0x17b97b4bce5b0227ull, 0x19a6a8e96c86261dull, 0x1b90d7529260a204ull, 0x1d77d5df20573672ull,
    0x1f5b75f92c80dd63ull, 0x213b8b2fb0c6c4b1ull, 0x2317eb4617e2f04cull, 0x24f06e40afde8b7cull,
    0x26c4ee6e0fd7979aull, 0x2895486d855e1351ull, 0x2a615b32a39a93b7ull, 0x2c290806139fc32cull,
    0x2dec3283c9bde11dull, 0x2faac096c767eeb5ull, 0x31649a7294364adbull, 0x3319aa8a9ad630cfull,
    0x34c9dd879847f96eull, 0x3675223b4cb8d8d7ull, 0x381b69929d93df1aull, 0x39bca6865826a12full,
    0x3b58ce0ac3769ed1ull, 0x3cefd6fe2eb46887ull, 0x3e81ba16a8282f97ull, 0x400e71cf06902e4dull,
    0x4195fa536cc33f15ull, 0x4318516d6d0f6833ull, 0x4495766fef4aa3dbull, 0x460d6a22f9f04dc6ull,
    0x47802eaf7bfacfceull, 0x48edc78b3279a871ull, 0x4a563964c238c37bull, 0x4bb98a101b2f29c6ull,
    0x4d17c07338deed10ull, 0x4e70e473505c66ddull, 0x4fc4fee27a5bd0f6ull, 0x5114196de56d5704ull,
    0x525e3e8c9a7b8492ull, 0x53a3796edbb0114aull, 0x54e3d5ee24187ae4ull, 0x561f607dccbeeb51ull,
    0x5756261c5a6c6040ull, 0x5888344575ee37b5ull, 0x59b598e48f821b49ull, 0x5ade62482cf66258ull,
    0x5c029f15e118cf3aull, 0x5d225e3eea383c18ull, 0x5e3daef574c57940ull, 0x5f54a0a27e824d56ull,
    0x606742dc56293320ull, 0x6175a55db30b145bull, 0x627fd7fd5fc7deaaull, 0x6385eaa67301770aull};

// The float nearest to m * 2^e (a normal float or 0).
__device__ __forceinline__ float fix_float(Fix64 a) {
    a = fix_norm(a);
    const uint32_t r = (uint32_t)(a.m >> 40) + ((uint32_t)(a.m >> 39) & 1u);
    return (long long)a.m >= 0 ? 0.f : __int_as_float((int)(((uint32_t)(a.e + 189) << 23) + r));
}
// The double of a positive normal float.
__device__ __forceinline__ double double_of_normal(float x) {
    const uint32_t b = (uint32_t)__float_as_int(x);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

static __device__ __noinline__ float atan2_general(float y, float x) { return (float)atan2((double)y, (double)x); }
__device__ __forceinline__ float fix_atan2f(float y, float x) {
    const uint32_t ab = (uint32_t)__float_as_int(y) & 0x7fffffffu, bb = (uint32_t)__float_as_int(x) & 0x7fffffffu;
    const uint32_t lb = min(ab, bb), hb = max(ab, bb);
    const int s = (int)(hb >> 23) - (int)(lb >> 23);
    // not both normal and of like size, or so large that the quotient's 1 / hi would flush to zero
    if (lb < 0x00800000u || hb > 0x7e800000u || s > 60) {
        if (ab == 0 && bb <= 0x7f800000u) return copysignf(__float_as_int(x) < 0 ? 3.14159274f : 0.f, y);
        if (bb == 0 && ab <= 0x7f800000u) return copysignf(1.57079637f, y);
        return atan2_general(y, x);
    }
    const float lo = __int_as_float((int)lb), hi = __int_as_float((int)hb);
    const uint64_t ml = (lb & 0x7fffffu) | 0x800000u, mh = (hb & 0x7fffffu) | 0x800000u;
    const bool swap = ab > bb;
    // i / 64 <= lo / hi, at most 1 / 64 below it
    const int i = (int)(lo * __fdividef(1.f, hi) * 63.9999f);
    const uint64_t den = i ? mh << s : mh;
    const uint64_t N = i ? 64ull * ml - (uint64_t)i * den : ml, Dn = i ? 64ull * den + (uint64_t)i * ml : mh;
    const int z = __clzll((long long)Dn);
    const uint64_t Y = recip_mant((Dn << z) >> 11);   // 1 / Dn = Y 2^(z - 125)
    const Fix64 n = fix_norm({N, i ? 0 : -s});
    const Fix64 q = fix_norm({mul_hi(n.m, Y << 1), n.e + z - 62});
    const uint64_t z2 = mul_hi(q.m, q.m) >> min(-(2 * q.e + 128), 63);   // q^2 2^64
    const uint32_t h = 0x24924925u - __umulhi((uint32_t)(z2 >> 32), 0x1c71c71cu);
    uint64_t H = 0x3333333333333333ull - mul_hi(z2, (uint64_t)h << 32);
    H = 0x5555555555555555ull - mul_hi(z2, H);
    const Fix64 at = fix_norm({mul_hi(q.m, ~0ull - mul_hi(z2, H)), q.e});
    if (i == 0 && !swap && x > 0.f) return copysignf(fix_float(at), y);
    const int sh = -61 - at.e;
    uint64_t r = (sh < 64 ? at.m >> sh : 0ull) + (__ldg(kAtanT + i) >> 2);   // 2^61
    if (swap) r = 0x3243f6a8885a308dull - r;
    if (x < 0.f) r = 0x6487ed5110b4611aull - r;
    return copysignf(fix_float({r, -61}), y);
}

// |x| <= pi/2 and a little; NaN for all others.
__device__ __forceinline__ void fix_sincosf(float x, float &sn, float &cs) {
    const uint32_t b = (uint32_t)__float_as_int(x) & 0x7fffffffu;
    // below 2^-13 the nearest floats are x and 1
    const bool tiny = b < 0x39000000u;
    const uint64_t T = (uint64_t)((b & 0x7fffffu) | 0x800000u) << ((int)(tiny ? 0x72u : b >> 23) - 87);   // |x| 2^63
    const uint64_t kHi = 0xc90fdaa22168c234ull, kLo = 0xc4c6628b80dc1cd1ull;                              // pi/2 2^63
    const bool big = T > (kHi >> 1), neg = T > kHi;
    // big: pi/2 - |x| in 128 bits, so that its leading 64 are exact beside pi/2
    const uint64_t hi = neg ? T - kHi - 1 : kHi - T, lo = neg ? 0ull - kLo : kLo;
    const int z = min(__clzll((long long)(hi | 1ull)), 63);
    const Fix64 dl = big ? Fix64{z ? (hi << z) | (lo >> (64 - z)) : hi, -63 - z} : fix_norm({T, -63});
    const int sh = -64 - dl.e;
    const uint64_t dq = dl.m >> min(sh, 63);   // 2^64
    const uint64_t d2 = mul_hi(dq, dq);
    const uint32_t d = (uint32_t)(d2 >> 32);
    uint32_t h = 0xd73f9fu - __umulhi(d, 0xca96u);
    h = 0xb092309du - __umulhi(d, h);
    uint64_t S = 0x6b99159fd5ull - mul_hi(d2, h);
    S = 0x2e3bc74aad8eull - mul_hi(d2, S);
    S = 0xd00d00d00d00dull - mul_hi(d2, S);
    S = 0x222222222222222ull - mul_hi(d2, S);
    S = 0x2aaaaaaaaaaaaaabull - mul_hi(d2, S);
    h = 0xd73fau - __umulhi(d, 0xb41u);
    h = 0xc9cba54u - __umulhi(d, h);
    uint64_t Cc = 0x8f76c77fcull - mul_hi(d2, h);
    Cc = 0x49f93edde28ull - mul_hi(d2, Cc);
    Cc = 0x1a01a01a01a02ull - mul_hi(d2, Cc);
    Cc = 0x5b05b05b05b05bull - mul_hi(d2, Cc);
    Cc = 0xaaaaaaaaaaaaaabull - mul_hi(d2, Cc);
    Cc = 0x8000000000000000ull - mul_hi(d2, Cc);
    const float sd = fix_float({mul_hi(dl.m, ~0ull - mul_hi(d2, S)), dl.e});
    const float cd = fix_float({~0ull - mul_hi(d2, Cc), -64});
    sn = tiny ? x : copysignf(big ? cd : sd, x);
    cs = tiny ? 1.f : big ? (neg ? -sd : sd) : cd;
    if (b >= 0x3fcccccdu) sn = cs = __int_as_float(0x7fffffff);
}

}  // namespace sphfem
