// x^y in double precision for the entropy K = P rho^-gamma of the face states
// (two a face, three directions, every sub-step).
//
// Table-driven logarithm and exponential after P. T. P. Tang (ACM Trans. Math.
// Softw. 16 (1990) 378-400 and 15 (1989) 144-157), base 2, the logarithm
// carried in two doubles so that the product with y loses nothing:
//   x = 2^e m, 1 <= m < 2; the leading 7 bits of m pick c ~ 1/m with 9
//   fractional bits; r = m c - 1 (one fma, |r| < 2^-7.7, error < 2^-60);
//   log2 x = e - log2 c + log2(1 + r), -log2 c tabulated as hi + lo with hi a
//   multiple of 2^-40 (e + hi is exact), log2(1 + r) by its series, the first
//   term with its error;
//   z = y log2 x as hi + lo; 2^z = 2^n 2^(j/32) 2^f with |f| <= 1/64, 2^(j/32)
//   tabulated as hi + lo, 2^f by its series.
// Error below 0.56 ulp (tests/test_pow.py, against extended precision), for
// positive normal x and results well inside the normal range; pow() takes the
// rest. About 36 FP64 operations and no branch but the one for the rest.
#pragma once
#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define HAMR_HD __host__ __device__ __forceinline__
#define HAMR_TABLE static __device__ const
#else
#define HAMR_HD static inline
#define HAMR_TABLE static const
#endif

namespace hamr {

// -log2 c (hi, lo), c, padding: one 32-byte row per leading 7 bits of m
HAMR_TABLE double pow_log2[128][4] = {
    {0x1.720d9c0700000p-8, -0x1.5f28564439c1ap-42, 0x1.fe00000000000p-1, 0.},
    {0x1.16a21e20c0000p-6, -0x1.f5baf436cbec7p-42, 0x1.fa00000000000p-1, 0.},
    {0x1.d23afc4900000p-6, 0x1.39f89bcdae7bdp-42, 0x1.f600000000000p-1, 0.},
    {0x1.47aa073580000p-5, -0x1.1f61a96b8ce77p-42, 0x1.f200000000000p-1, 0.},
    {0x1.8f135b8100000p-5, 0x1.e44675020ccd7p-43, 0x1.ef00000000000p-1, 0.},
    {0x1.eef7925080000p-5, 0x1.6d3ac26e64b73p-42, 0x1.eb00000000000p-1, 0.},
    {0x1.27d24bae80000p-4, 0x1.26d610050fdb5p-43, 0x1.e700000000000p-1, 0.},
    {0x1.4c560fe690000p-4, -0x1.41dfc7d7c3321p-42, 0x1.e400000000000p-1, 0.},
    {0x1.7d60496d00000p-4, -0x1.12ce6312ebb82p-42, 0x1.e000000000000p-1, 0.},
    {0x1.a26ccd9980000p-4, 0x1.852899427dd61p-44, 0x1.dd00000000000p-1, 0.},
    {0x1.d4300a2520000p-4, 0x1.3505dacd2ed72p-42, 0x1.d900000000000p-1, 0.},
    {0x1.f9c95dc1d0000p-4, 0x1.164e932b2d51cp-44, 0x1.d600000000000p-1, 0.},
    {0x1.1625931870000p-3, -0x1.2c81df0fdbc29p-42, 0x1.d200000000000p-1, 0.},
    {0x1.293ac3dc18000p-3, 0x1.33432f2c33fc6p-42, 0x1.cf00000000000p-1, 0.},
    {0x1.3c6fb650d0000p-3, -0x1.0d7af4dda9c36p-42, 0x1.cc00000000000p-1, 0.},
    {0x1.4fc4d4d9b8000p-3, 0x1.989af85862e57p-42, 0x1.c900000000000p-1, 0.},
    {0x1.633a8bf438000p-3, -0x1.8f7aac147fdc1p-46, 0x1.c600000000000p-1, 0.},
    {0x1.7d60496cf8000p-3, 0x1.da6339da288fcp-42, 0x1.c200000000000p-1, 0.},
    {0x1.9123c15290000p-3, -0x1.c9908593990cfp-42, 0x1.bf00000000000p-1, 0.},
    {0x1.a5094b54d0000p-3, 0x1.41420276dd59dp-42, 0x1.bc00000000000p-1, 0.},
    {0x1.b9115db838000p-3, 0x1.1ee969a95f529p-42, 0x1.b900000000000p-1, 0.},
    {0x1.cd3c712d30000p-3, 0x1.109325dd5e814p-43, 0x1.b600000000000p-1, 0.},
    {0x1.e18b00e130000p-3, 0x1.23d066fdd7c23p-43, 0x1.b300000000000p-1, 0.},
    {0x1.ef28aacd70000p-3, 0x1.118906313e79dp-42, 0x1.b100000000000p-1, 0.},
    {0x1.01d9bbcfa8000p-2, -0x1.e2ba25d9aeffdp-42, 0x1.ae00000000000p-1, 0.},
    {0x1.0c318aee00000p-2, -0x1.87f13324f6d23p-43, 0x1.ab00000000000p-1, 0.},
    {0x1.169c053640000p-2, -0x1.d4f1b95e0ff45p-43, 0x1.a800000000000p-1, 0.},
    {0x1.21196e8748000p-2, -0x1.85e9a1fc3cc8ep-43, 0x1.a500000000000p-1, 0.},
    {0x1.28225bb5e8000p-2, -0x1.b5c17154f4086p-42, 0x1.a300000000000p-1, 0.},
    {0x1.32bfee3710000p-2, -0x1.1979a5db68722p-42, 0x1.a000000000000p-1, 0.},
    {0x1.3d712bf9c8000p-2, 0x1.deecc62372284p-42, 0x1.9d00000000000p-1, 0.},
    {0x1.449d115ef8000p-2, -0x1.3c49c247ab6afp-45, 0x1.9b00000000000p-1, 0.},
    {0x1.4f6fbb2cec000p-2, 0x1.661e393a16b95p-44, 0x1.9800000000000p-1, 0.},
    {0x1.56b22e6b58000p-2, -0x1.c6d8d86531d56p-44, 0x1.9600000000000p-1, 0.},
    {0x1.61a717cac0000p-2, 0x1.983115f01e8fep-42, 0x1.9300000000000p-1, 0.},
    {0x1.6900a8836c000p-2, 0x1.0d5074f35e53cp-42, 0x1.9100000000000p-1, 0.},
    {0x1.7418acebc0000p-2, -0x1.ce2935fff809ap-43, 0x1.8e00000000000p-1, 0.},
    {0x1.7b89f02cf4000p-2, -0x1.552ce0ec3a295p-42, 0x1.8c00000000000p-1, 0.},
    {0x1.8304d90c10000p-2, 0x1.fd32a3ab0a4b5p-42, 0x1.8a00000000000p-1, 0.},
    {0x1.8e4f83fa14000p-2, 0x1.7b6bf20f1e8c4p-44, 0x1.8700000000000p-1, 0.},
    {0x1.95e2f9b520000p-2, -0x1.f63a1b3264f72p-43, 0x1.8500000000000p-1, 0.},
    {0x1.9d806ebc98000p-2, 0x1.21b8c1b8b7dfdp-42, 0x1.8300000000000p-1, 0.},
    {0x1.a8ff971810000p-2, 0x1.4bc302ffa76fbp-43, 0x1.8000000000000p-1, 0.},
    {0x1.b0b67f4f48000p-2, -0x1.7f00af09dc1c7p-42, 0x1.7e00000000000p-1, 0.},
    {0x1.b877c57b1c000p-2, -0x1.f20203b3186a6p-43, 0x1.7c00000000000p-1, 0.},
    {0x1.c043859e30000p-2, -0x1.2642415d47384p-45, 0x1.7a00000000000p-1, 0.},
    {0x1.c819dc2d44000p-2, 0x1.fe43895d8ac46p-42, 0x1.7800000000000p-1, 0.},
    {0x1.d3ef776d44000p-2, -0x1.81e2b378ff59dp-51, 0x1.7500000000000p-1, 0.},
    {0x1.dbe0c58c3c000p-2, 0x1.fe34ad4ba7ee9p-43, 0x1.7300000000000p-1, 0.},
    {0x1.e3dd115650000p-2, 0x1.f77628aa1aed8p-44, 0x1.7100000000000p-1, 0.},
    {0x1.ebe47960e4000p-2, -0x1.fbc00d8d6cbcfp-45, 0x1.6f00000000000p-1, 0.},
    {0x1.f3f71cc1b8000p-2, -0x1.d647d323e3e73p-42, 0x1.6d00000000000p-1, 0.},
    {0x1.fc151b11b4000p-2, -0x1.37fc8cafdef46p-43, 0x1.6b00000000000p-1, 0.},
    {0x1.021f4a37ec000p-1, 0x1.7f5dc57266758p-42, 0x1.6900000000000p-1, 0.},
    {0x1.0639d4c21a000p-1, -0x1.50343f8df4b43p-44, 0x1.6700000000000p-1, 0.},
    {0x1.0a5a3dc176000p-1, -0x1.bce53e5c9e604p-42, 0x1.6500000000000p-1, 0.},
    {0x1.0e809617b4000p-1, 0x1.acfe41bb5518cp-43, 0x1.6300000000000p-1, 0.},
    {0x1.12aceeefce000p-1, -0x1.f72024e94ae2bp-43, 0x1.6100000000000p-1, 0.},
    {0x1.16df59bfa0000p-1, 0x1.b055bd48256adp-43, 0x1.5f00000000000p-1, 0.},
    {0x1.18fadb6e2e000p-1, -0x1.87cc95d0a2ee8p-42, 0x1.5e00000000000p-1, 0.},
    {0x1.1d368296b6000p-1, -0x1.b567e7ee54aefp-42, 0x1.5c00000000000p-1, 0.},
    {0x1.217868b0c4000p-1, -0x1.030ab442ce320p-42, 0x1.5a00000000000p-1, 0.},
    {0x1.25c0a0463c000p-1, -0x1.50520a377c7ecp-45, 0x1.5800000000000p-1, 0.},
    {0x1.2a0f3c3408000p-1, -0x1.f48e1a4725559p-42, 0x1.5600000000000p-1, 0.},
    {0x1.2e644fac04000p-1, 0x1.faf6283bf2868p-42, 0x1.5400000000000p-1, 0.},
    {0x1.30914c5326000p-1, 0x1.a207724e30639p-42, 0x1.5300000000000p-1, 0.},
    {0x1.34f037d6c6000p-1, -0x1.3719eb3af5b8dp-47, 0x1.5100000000000p-1, 0.},
    {0x1.3955cc6252000p-1, -0x1.b8d59e8492d6ep-45, 0x1.4f00000000000p-1, 0.},
    {0x1.3b8b1c68fa000p-1, 0x1.bb4b69336b66ep-43, 0x1.4e00000000000p-1, 0.},
    {0x1.3ffad4e750000p-1, -0x1.c5432aeb609f5p-42, 0x1.4c00000000000p-1, 0.},
    {0x1.44716a2c08000p-1, 0x1.3106e404cabb7p-44, 0x1.4a00000000000p-1, 0.},
    {0x1.46af4e41a2000p-1, -0x1.829434d994a2ap-46, 0x1.4900000000000p-1, 0.},
    {0x1.4b3056db9a000p-1, -0x1.4b868c5485435p-42, 0x1.4700000000000p-1, 0.},
    {0x1.4fb8725eb6000p-1, -0x1.15b2de01cea41p-43, 0x1.4500000000000p-1, 0.},
    {0x1.51ff2e3022000p-1, -0x1.6879fa00b120ap-42, 0x1.4400000000000p-1, 0.},
    {0x1.5692101d9c000p-1, -0x1.6b37dcf60e620p-42, 0x1.4200000000000p-1, 0.},
    {0x1.5b2c3da198000p-1, -0x1.b8afe492bf6ffp-42, 0x1.4000000000000p-1, 0.},
    {0x1.5d7c180916000p-1, -0x1.f8729ab413ffap-43, 0x1.3f00000000000p-1, 0.},
    {0x1.622162faf2000p-1, -0x1.cfa95830dd0dap-42, 0x1.3d00000000000p-1, 0.},
    {0x1.6476d98ada000p-1, -0x1.bd9b32266d92cp-43, 0x1.3c00000000000p-1, 0.},
    {0x1.6927781d94000p-1, -0x1.aaf6f137a3d8cp-42, 0x1.3a00000000000p-1, 0.},
    {0x1.6b82a65266000p-1, 0x1.97c9cfc5e95bep-42, 0x1.3900000000000p-1, 0.},
    {0x1.703ed0493c000p-1, -0x1.c2657d0d1a7f0p-43, 0x1.3700000000000p-1, 0.},
    {0x1.729fd26b70000p-1, 0x1.f1f5ae718f241p-43, 0x1.3600000000000p-1, 0.},
    {0x1.7767c12968000p-1, -0x1.6eb9612e0b4f3p-43, 0x1.3400000000000p-1, 0.},
    {0x1.79ceb4555e000p-1, 0x1.5715b04e05be8p-42, 0x1.3300000000000p-1, 0.},
    {0x1.7c37a9227e000p-1, 0x1.fed21f9cb2cc5p-43, 0x1.3200000000000p-1, 0.},
    {0x1.810fa51bf6000p-1, 0x1.7f5dc57266758p-43, 0x1.3000000000000p-1, 0.},
    {0x1.837eb31b7e000p-1, -0x1.e4e8eea54ce63p-44, 0x1.2f00000000000p-1, 0.},
    {0x1.886300713a000p-1, 0x1.bf88f20dec619p-42, 0x1.2d00000000000p-1, 0.},
    {0x1.8ad846cf36000p-1, 0x1.3481b85a54d7fp-42, 0x1.2c00000000000p-1, 0.},
    {0x1.8d4fa70e24000p-1, -0x1.b912d8994b162p-44, 0x1.2b00000000000p-1, 0.},
    {0x1.9244c3a282000p-1, -0x1.5e96bed8cce30p-43, 0x1.2900000000000p-1, 0.},
    {0x1.94c287492c000p-1, 0x1.36c101ee13440p-43, 0x1.2800000000000p-1, 0.},
    {0x1.974273737e000p-1, -0x1.c35651c429393p-42, 0x1.2700000000000p-1, 0.},
    {0x1.9c48d45f2c000p-1, -0x1.5b5dae6a10ccap-42, 0x1.2500000000000p-1, 0.},
    {0x1.9ecf50bf44000p-1, -0x1.d97ee9124773bp-46, 0x1.2400000000000p-1, 0.},
    {0x1.a15804e0be000p-1, 0x1.1108740d92f89p-42, 0x1.2300000000000p-1, 0.},
    {0x1.a6702414dc000p-1, -0x1.3167ccc538261p-43, 0x1.2100000000000p-1, 0.},
    {0x1.a8ff971810000p-1, 0x1.4bc302ffa76fbp-42, 0x1.2000000000000p-1, 0.},
    {0x1.ab9151be16000p-1, 0x1.1badba7fbb3d2p-42, 0x1.1f00000000000p-1, 0.},
    {0x1.ae255819f0000p-1, 0x1.1659d8e2d7d38p-44, 0x1.1e00000000000p-1, 0.},
    {0x1.b35458761e000p-1, -0x1.70d0fa8f9603bp-42, 0x1.1c00000000000p-1, 0.},
    {0x1.b5ef5ad3e2000p-1, -0x1.31fc6bb455652p-42, 0x1.1b00000000000p-1, 0.},
    {0x1.b88cb9a2ac000p-1, -0x1.5bdaf522a183cp-42, 0x1.1a00000000000p-1, 0.},
    {0x1.bb2c792ddc000p-1, -0x1.8b7fcd690403ep-45, 0x1.1900000000000p-1, 0.},
    {0x1.c0732be1ea000p-1, -0x1.49209a68c72a1p-49, 0x1.1700000000000p-1, 0.},
    {0x1.c31a27dd00000p-1, 0x1.69378d0928989p-42, 0x1.1600000000000p-1, 0.},
    {0x1.c5c3963948000p-1, 0x1.f496cbd31c337p-42, 0x1.1500000000000p-1, 0.},
    {0x1.c86f7b7ea4000p-1, 0x1.51167134e9647p-42, 0x1.1400000000000p-1, 0.},
    {0x1.cb1ddc4196000p-1, 0x1.edb052ee9f871p-42, 0x1.1300000000000p-1, 0.},
    {0x1.cdcebd2374000p-1, -0x1.9ad57391924a7p-43, 0x1.1200000000000p-1, 0.},
    {0x1.d338120a6e000p-1, -0x1.3167ccc538261p-44, 0x1.1000000000000p-1, 0.},
    {0x1.d5f08f93fa000p-1, -0x1.ddb6a7969bdb5p-43, 0x1.0f00000000000p-1, 0.},
    {0x1.d8aba045b0000p-1, 0x1.c7a4ff65ddbc9p-45, 0x1.0e00000000000p-1, 0.},
    {0x1.db694903da000p-1, -0x1.68f2268b3cd45p-42, 0x1.0d00000000000p-1, 0.},
    {0x1.de298ec0ba000p-1, 0x1.819530c22d152p-42, 0x1.0c00000000000p-1, 0.},
    {0x1.e0ec767cce000p-1, -0x1.4e7e87341aeeep-43, 0x1.0b00000000000p-1, 0.},
    {0x1.e3b20546f6000p-1, -0x1.56bde9f1f0d3dp-42, 0x1.0a00000000000p-1, 0.},
    {0x1.e67a403cb6000p-1, 0x1.5cd73ebe3895ep-42, 0x1.0900000000000p-1, 0.},
    {0x1.e9452c8a72000p-1, -0x1.fb0e626c0de13p-42, 0x1.0800000000000p-1, 0.},
    {0x1.ec12cf6b98000p-1, -0x1.6898809d2dc10p-43, 0x1.0700000000000p-1, 0.},
    {0x1.eee32e2aec000p-1, 0x1.97da24fd75f61p-42, 0x1.0600000000000p-1, 0.},
    {0x1.f1b64e22be000p-1, -0x1.0f86666e80f71p-42, 0x1.0500000000000p-1, 0.},
    {0x1.f48c34bd1e000p-1, 0x1.2dd67591d81dfp-42, 0x1.0400000000000p-1, 0.},
    {0x1.f764e7742c000p-1, -0x1.7b0c4bb41a6c9p-42, 0x1.0300000000000p-1, 0.},
    {0x1.fa406bd244000p-1, 0x1.ef5d00e390a00p-44, 0x1.0200000000000p-1, 0.},
    {0x1.fd1ec77250000p-1, 0x1.54e22d4990b6ep-42, 0x1.0100000000000p-1, 0.},
};

// 2^(j/32) (hi, lo)
HAMR_TABLE double pow_exp2[32][2] = {
    {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54},
};

#ifdef __CUDA_ARCH__
__device__ __forceinline__ int pow_hi(double x) { return __double2hiint(x); }
__device__ __forceinline__ int pow_lo(double x) { return __double2loint(x); }
__device__ __forceinline__ double pow_bits(int hi, int lo) { return __hiloint2double(hi, lo); }
__device__ __noinline__ double pow_rest(double x, double y) { return pow(x, y); }
#else
static inline int pow_hi(double x) { long long b; memcpy(&b, &x, 8); return (int)(b >> 32); }
static inline int pow_lo(double x) { long long b; memcpy(&b, &x, 8); return (int)b; }
static inline double pow_bits(int hi, int lo) {
    long long b = ((long long)hi << 32) | (unsigned)lo;
    double x;
    memcpy(&x, &b, 8);
    return x;
}
static inline double pow_rest(double x, double y) { return pow(x, y); }
#endif

HAMR_HD double pow_tab(double x, double y) {
    const int hx = pow_hi(x);
    if ((unsigned)hx - 0x00100000u >= 0x7fe00000u) return pow_rest(x, y);   // not a positive normal number
    const int e = (hx >> 20) - 1023, i = (hx >> 13) & 127;
    const double m = pow_bits((hx & 0x000fffff) | 0x3ff00000, pow_lo(x));
    const double *row = pow_log2[i];
    const double lhi = row[0], llo = row[1], c = row[2];
    // e as a double: 2^52 + 2^31 + e from its bits
    const double ed = pow_bits(0x43300000, (int)(0x80000000u ^ (unsigned)e)) - 4503601774854144.0;
    const double r = fma(m, c, -1.0);
    const double p1 = r * 0x1.71547652b82fep+0;
    const double e1 = fma(r, 0x1.777d0ffda0d24p-56, fma(r, 0x1.71547652b82fep+0, -p1));
    double q = 0x1.a61762a7aded9p-3;
    q = fma(q, r, -0x1.ec709dc3a03fdp-3);
    q = fma(q, r, 0x1.2776c50ef9bfep-2);
    q = fma(q, r, -0x1.71547652b82fep-2);
    q = fma(q, r, 0x1.ec709dc3a03fdp-2);
    q = fma(q, r, -0x1.71547652b82fep-1);
    const double t = ed + lhi;
    // t + p1 = s + es exactly: t is 0 or exceeds |p1| in magnitude, or both
    // are small multiples of 2^-61
    const double s = t + p1;
    const double bb = s - t;
    const double es = (t - (s - bb)) + (p1 - bb);
    const double lo = es + fma(q, r * r, e1 + llo);
    const double z = y * s;
    const double zl = fma(y, lo, fma(y, s, -z));
    if (!(fabs(z) < 1000.)) return pow_rest(x, y);
    const double k = fma(z, 32., 6755399441055744.0);   // 1.5 2^52: the integer nearest 32 z in its low bits
    const int n = pow_lo(k);
    const double f = fma(k - 6755399441055744.0, -0.03125, z) + zl;
    double p = 0x1.430912f86c787p-13;
    p = fma(p, f, 0x1.5d87fe78a6731p-10);
    p = fma(p, f, 0x1.3b2ab6fba4e77p-7);
    p = fma(p, f, 0x1.c6b08d704a0c0p-5);
    p = fma(p, f, 0x1.ebfbdff82c58fp-3);
    p = fma(p, f, 0x1.62e42fefa39efp-1);
    const double th = pow_exp2[n & 31][0], tl = pow_exp2[n & 31][1];
    const double w = th + fma(th, p * f, tl);
    return pow_bits(pow_hi(w) + ((n >> 5) << 20), pow_lo(w));
}

}  // namespace hamr
