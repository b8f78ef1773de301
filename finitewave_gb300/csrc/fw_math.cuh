// fw_math.cuh -- exponentials, logarithms and reciprocals of the detailed
// models' updates, in both precisions behind one set of names (namespace
// fw::dm), so that an update is written once.
//
// float64: GB300 executes two float64 instructions a clock and SM, so a step
// of a detailed model takes as long as the float64 instructions it issues
// (86 % of the pipe's time measured on the TP06 step with CUDA's functions).
// These forms spend few of them and leave the rest to the integer and
// special-function units:
//   * exp: the table-driven method of P. T. P. Tang (ACM TOMS 15, 1989) with
//     2^(j/256): x = n ln2/256 + r (n rounded in float32 from the high
//     word, so |r| < 1.5e-3 for |x| < 60, < 2.1e-3 up to 700), e^r by its
//     series to r^4 / 24 (remainder below 7e-17, 3.5e-16), the power of two
//     added to the exponent field: 8 float64 instructions;
//   * log: P. T. P. Tang (ACM TOMS 16, 1990) with 128 intervals: x = 2^e m,
//     r = c_j m - 1, |r| < 4.0e-3, log1p by its series to r^6 / 6: 10;
//   * reciprocal: rcp.approx.ftz.f64 (PTX: relative error at most 2^-20) and
//     one step of third order, y (1 + e + e^2), e = 1 - d y: 3;
//   * reciprocal square root: rsqrt.approx.ftz.f64 and the third-order step
//     y (1 + e / 2 + 3 e^2 / 8), e = 1 - d y^2: 5.
// Errors against extended precision: exp within 1.5 ulp for |x| < 60 and 2.5
// up to 700 (half an ulp each for the table and the last sum, the rest the
// series' remainder), the reciprocals within 1.5 ulp, log within 1.5 ulp of
// max(1, |log x|).  Arguments are those of the models'
// in-range updates: finite, exponents of at most a few hundred, positive
// normal numbers under log, 1 / x and 1 / sqrt(x) (log hands anything else
// to CUDA's).
//
// float32: ex2.approx / lg2.approx / rcp.approx / rsqrt.approx, one
// special-function instruction each.  A division costs one of them and a
// product here (a / b compiles to about eight instructions even with
// --prec-div=false).
#pragma once

#include <stdint.h>

namespace fw {
namespace dm {
namespace {

// 2^(j/256), j = 0..255, correctly rounded
__device__ const double kExp2Tab[256] = {
    0x1.0000000000000p+0, 0x1.00b1afa5abcbfp+0, 0x1.0163da9fb3335p+0, 0x1.02168143b0281p+0,
    0x1.02c9a3e778061p+0, 0x1.037d42e11bbccp+0, 0x1.04315e86e7f85p+0, 0x1.04e5f72f654b1p+0,
    0x1.059b0d3158574p+0, 0x1.0650a0e3c1f89p+0, 0x1.0706b29ddf6dep+0, 0x1.07bd42b72a836p+0,
    0x1.0874518759bc8p+0, 0x1.092bdf66607e0p+0, 0x1.09e3ecac6f383p+0, 0x1.0a9c79b1f3919p+0,
    0x1.0b5586cf9890fp+0, 0x1.0c0f145e46c85p+0, 0x1.0cc922b7247f7p+0, 0x1.0d83b23395decp+0,
    0x1.0e3ec32d3d1a2p+0, 0x1.0efa55fdfa9c5p+0, 0x1.0fb66affed31bp+0, 0x1.1073028d7233ep+0,
    0x1.11301d0125b51p+0, 0x1.11edbab5e2ab6p+0, 0x1.12abdc06c31ccp+0, 0x1.136a814f204abp+0,
    0x1.1429aaea92de0p+0, 0x1.14e95934f312ep+0, 0x1.15a98c8a58e51p+0, 0x1.166a45471c3c2p+0,
    0x1.172b83c7d517bp+0, 0x1.17ed48695bbc0p+0, 0x1.18af9388c8deap+0, 0x1.1972658375d2fp+0,
    0x1.1a35beb6fcb75p+0, 0x1.1af99f8138a1cp+0, 0x1.1bbe084045cd4p+0, 0x1.1c82f95281c6bp+0,
    0x1.1d4873168b9aap+0, 0x1.1e0e75eb44027p+0, 0x1.1ed5022fcd91dp+0, 0x1.1f9c18438ce4dp+0,
    0x1.2063b88628cd6p+0, 0x1.212be3578a819p+0, 0x1.21f49917ddc96p+0, 0x1.22bdda27912d1p+0,
    0x1.2387a6e756238p+0, 0x1.2451ffb82140ap+0, 0x1.251ce4fb2a63fp+0, 0x1.25e85711ece75p+0,
    0x1.26b4565e27cddp+0, 0x1.2780e341ddf29p+0, 0x1.284dfe1f56381p+0, 0x1.291ba7591bb70p+0,
    0x1.29e9df51fdee1p+0, 0x1.2ab8a66d10f13p+0, 0x1.2b87fd0dad990p+0, 0x1.2c57e39771b2fp+0,
    0x1.2d285a6e4030bp+0, 0x1.2df961f641589p+0, 0x1.2ecafa93e2f56p+0, 0x1.2f9d24abd886bp+0,
    0x1.306fe0a31b715p+0, 0x1.31432edeeb2fdp+0, 0x1.32170fc4cd831p+0, 0x1.32eb83ba8ea32p+0,
    0x1.33c08b26416ffp+0, 0x1.3496266e3fa2dp+0, 0x1.356c55f929ff1p+0, 0x1.36431a2de883bp+0,
    0x1.371a7373aa9cbp+0, 0x1.37f26231e754ap+0, 0x1.38cae6d05d866p+0, 0x1.39a401b7140efp+0,
    0x1.3a7db34e59ff7p+0, 0x1.3b57fbfec6cf4p+0, 0x1.3c32dc313a8e5p+0, 0x1.3d0e544ede173p+0,
    0x1.3dea64c123422p+0, 0x1.3ec70df1c5175p+0, 0x1.3fa4504ac801cp+0, 0x1.40822c367a024p+0,
    0x1.4160a21f72e2ap+0, 0x1.423fb2709468ap+0, 0x1.431f5d950a897p+0, 0x1.43ffa3f84b9d4p+0,
    0x1.44e086061892dp+0, 0x1.45c2042a7d232p+0, 0x1.46a41ed1d0057p+0, 0x1.4786d668b3237p+0,
    0x1.486a2b5c13cd0p+0, 0x1.494e1e192aed2p+0, 0x1.4a32af0d7d3dep+0, 0x1.4b17dea6db7d7p+0,
    0x1.4bfdad5362a27p+0, 0x1.4ce41b817c114p+0, 0x1.4dcb299fddd0dp+0, 0x1.4eb2d81d8abffp+0,
    0x1.4f9b2769d2ca7p+0, 0x1.508417f4531eep+0, 0x1.516daa2cf6642p+0, 0x1.5257de83f4eefp+0,
    0x1.5342b569d4f82p+0, 0x1.542e2f4f6ad27p+0, 0x1.551a4ca5d920fp+0, 0x1.56070dde910d2p+0,
    0x1.56f4736b527dap+0, 0x1.57e27dbe2c4cfp+0, 0x1.58d12d497c7fdp+0, 0x1.59c0827ff07ccp+0,
    0x1.5ab07dd485429p+0, 0x1.5ba11fba87a03p+0, 0x1.5c9268a5946b7p+0, 0x1.5d84590998b93p+0,
    0x1.5e76f15ad2148p+0, 0x1.5f6a320dceb71p+0, 0x1.605e1b976dc09p+0, 0x1.6152ae6cdf6f4p+0,
    0x1.6247eb03a5585p+0, 0x1.633dd1d1929fdp+0, 0x1.6434634ccc320p+0, 0x1.652b9febc8fb7p+0,
    0x1.6623882552225p+0, 0x1.671c1c70833f6p+0, 0x1.68155d44ca973p+0, 0x1.690f4b19e9538p+0,
    0x1.6a09e667f3bcdp+0, 0x1.6b052fa75173ep+0, 0x1.6c012750bdabfp+0, 0x1.6cfdcddd47645p+0,
    0x1.6dfb23c651a2fp+0, 0x1.6ef9298593ae5p+0, 0x1.6ff7df9519484p+0, 0x1.70f7466f42e87p+0,
    0x1.71f75e8ec5f74p+0, 0x1.72f8286ead08ap+0, 0x1.73f9a48a58174p+0, 0x1.74fbd35d7cbfdp+0,
    0x1.75feb564267c9p+0, 0x1.77024b1ab6e09p+0, 0x1.780694fde5d3fp+0, 0x1.790b938ac1cf6p+0,
    0x1.7a11473eb0187p+0, 0x1.7b17b0976cfdbp+0, 0x1.7c1ed0130c132p+0, 0x1.7d26a62ff86f0p+0,
    0x1.7e2f336cf4e62p+0, 0x1.7f3878491c491p+0, 0x1.80427543e1a12p+0, 0x1.814d2add106d9p+0,
    0x1.82589994cce13p+0, 0x1.8364c1eb941f7p+0, 0x1.8471a4623c7adp+0, 0x1.857f4179f5b21p+0,
    0x1.868d99b4492edp+0, 0x1.879cad931a436p+0, 0x1.88ac7d98a6699p+0, 0x1.89bd0a478580fp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8be05bad61778p+0, 0x1.8cf3216b5448cp+0, 0x1.8e06a5e0866d9p+0,
    0x1.8f1ae99157736p+0, 0x1.902fed0282c8ap+0, 0x1.9145b0b91ffc6p+0, 0x1.925c353aa2fe2p+0,
    0x1.93737b0cdc5e5p+0, 0x1.948b82b5f98e5p+0, 0x1.95a44cbc8520fp+0, 0x1.96bdd9a7670b3p+0,
    0x1.97d829fde4e50p+0, 0x1.98f33e47a22a2p+0, 0x1.9a0f170ca07bap+0, 0x1.9b2bb4d53fe0dp+0,
    0x1.9c49182a3f090p+0, 0x1.9d674194bb8d5p+0, 0x1.9e86319e32323p+0, 0x1.9fa5e8d07f29ep+0,
    0x1.a0c667b5de565p+0, 0x1.a1e7aed8eb8bbp+0, 0x1.a309bec4a2d33p+0, 0x1.a42c980460ad8p+0,
    0x1.a5503b23e255dp+0, 0x1.a674a8af46052p+0, 0x1.a799e1330b358p+0, 0x1.a8bfe53c12e59p+0,
    0x1.a9e6b5579fdbfp+0, 0x1.ab0e521356ebap+0, 0x1.ac36bbfd3f37ap+0, 0x1.ad5ff3a3c2774p+0,
    0x1.ae89f995ad3adp+0, 0x1.afb4ce622f2ffp+0, 0x1.b0e07298db666p+0, 0x1.b20ce6c9a8952p+0,
    0x1.b33a2b84f15fbp+0, 0x1.b468415b749b1p+0, 0x1.b59728de5593ap+0, 0x1.b6c6e29f1c52ap+0,
    0x1.b7f76f2fb5e47p+0, 0x1.b928cf22749e4p+0, 0x1.ba5b030a1064ap+0, 0x1.bb8e0b79a6f1fp+0,
    0x1.bcc1e904bc1d2p+0, 0x1.bdf69c3f3a207p+0, 0x1.bf2c25bd71e09p+0, 0x1.c06286141b33dp+0,
    0x1.c199bdd85529cp+0, 0x1.c2d1cd9fa652cp+0, 0x1.c40ab5fffd07ap+0, 0x1.c544778fafb22p+0,
    0x1.c67f12e57d14bp+0, 0x1.c7ba88988c933p+0, 0x1.c8f6d9406e7b5p+0, 0x1.ca3405751c4dbp+0,
    0x1.cb720dcef9069p+0, 0x1.ccb0f2e6d1675p+0, 0x1.cdf0b555dc3fap+0, 0x1.cf3155b5bab74p+0,
    0x1.d072d4a07897cp+0, 0x1.d1b532b08c968p+0, 0x1.d2f87080d89f2p+0, 0x1.d43c8eacaa1d6p+0,
    0x1.d5818dcfba487p+0, 0x1.d6c76e862e6d3p+0, 0x1.d80e316c98398p+0, 0x1.d955d71ff6075p+0,
    0x1.da9e603db3285p+0, 0x1.dbe7cd63a8315p+0, 0x1.dd321f301b460p+0, 0x1.de7d5641c0658p+0,
    0x1.dfc97337b9b5fp+0, 0x1.e11676b197d17p+0, 0x1.e264614f5a129p+0, 0x1.e3b333b16ee12p+0,
    0x1.e502ee78b3ff6p+0, 0x1.e653924676d76p+0, 0x1.e7a51fbc74c83p+0, 0x1.e8f7977cdb740p+0,
    0x1.ea4afa2a490dap+0, 0x1.eb9f4867cca6ep+0, 0x1.ecf482d8e67f1p+0, 0x1.ee4aaa2188510p+0,
    0x1.efa1bee615a27p+0, 0x1.f0f9c1cb6412ap+0, 0x1.f252b376bba97p+0, 0x1.f3ac948dd7274p+0,
    0x1.f50765b6e4540p+0, 0x1.f6632798844f8p+0, 0x1.f7bfdad9cbe14p+0, 0x1.f91d802243c89p+0,
    0x1.fa7c1819e90d8p+0, 0x1.fbdba3692d514p+0, 0x1.fd3c22b8f71f1p+0, 0x1.fe9d96b2a23d9p+0,
};
// (c_j, -log c_j): c_j is 1 / (1 + (j + 1/2) / 128) rounded to 12 bits
__device__ const double2 kLogTab[128] = {
    {0x1.fe00000000000p-1, 0x1.0080559588b35p-8}, {0x1.fa20000000000p-1, 0x1.7a2c82e212c65p-7},
    {0x1.f640000000000p-1, 0x1.3b024b78c5669p-6}, {0x1.f260000000000p-1, 0x1.b9e8027e1918ep-6},
    {0x1.eea0000000000p-1, 0x1.1ad398c6cd588p-5}, {0x1.eae0000000000p-1, 0x1.592bbc15215c9p-5},
    {0x1.e740000000000p-1, 0x1.95e430f8ce45ep-5}, {0x1.e3a0000000000p-1, 0x1.d310ba20455a1p-5},
    {0x1.e020000000000p-1, 0x1.074883629640bp-4}, {0x1.dca0000000000p-1, 0x1.254062f0a9417p-4},
    {0x1.d920000000000p-1, 0x1.4370ce02b7de8p-4}, {0x1.d5c0000000000p-1, 0x1.60c38ba79945dp-4},
    {0x1.d280000000000p-1, 0x1.7d33687c293c9p-4}, {0x1.cf20000000000p-1, 0x1.9af124d64c626p-4},
    {0x1.cbe0000000000p-1, 0x1.b7c9832f5801ap-4}, {0x1.c8c0000000000p-1, 0x1.d3b73f37e1f9bp-4},
    {0x1.c580000000000p-1, 0x1.f0f70cdd992e3p-4}, {0x1.c260000000000p-1, 0x1.06a4d1d26c5e6p-3},
    {0x1.bf60000000000p-1, 0x1.1454d8953741cp-3}, {0x1.bc40000000000p-1, 0x1.22aff2ddbd971p-3},
    {0x1.b960000000000p-1, 0x1.2ffbf29a6645cp-3}, {0x1.b660000000000p-1, 0x1.3df3ab13505f7p-3},
    {0x1.b380000000000p-1, 0x1.4b6d6fefe22a4p-3}, {0x1.b0a0000000000p-1, 0x1.58fe0e4c62eaep-3},
    {0x1.adc0000000000p-1, 0x1.66a5d42a3ad34p-3}, {0x1.ab00000000000p-1, 0x1.73cb9074fd14dp-3},
    {0x1.a820000000000p-1, 0x1.81a18b4220535p-3}, {0x1.a580000000000p-1, 0x1.8e588ebac2dbfp-3},
    {0x1.a2c0000000000p-1, 0x1.9bc062f26fc3ap-3}, {0x1.a020000000000p-1, 0x1.a8a14ffee66bdp-3},
    {0x1.9d80000000000p-1, 0x1.b5971a213acdbp-3}, {0x1.9ae0000000000p-1, 0x1.c2a205610593fp-3},
    {0x1.9860000000000p-1, 0x1.cf21d5ecbaa65p-3}, {0x1.95c0000000000p-1, 0x1.dc56cae452f5ap-3},
    {0x1.9340000000000p-1, 0x1.e8ff2622babc7p-3}, {0x1.90e0000000000p-1, 0x1.f518262c38082p-3},
    {0x1.8e60000000000p-1, 0x1.00f40470c7324p-2}, {0x1.8c00000000000p-1, 0x1.07138604d5862p-2},
    {0x1.89a0000000000p-1, 0x1.0d3c7586cd5e4p-2}, {0x1.8740000000000p-1, 0x1.136ef02e8290cp-2},
    {0x1.8500000000000p-1, 0x1.1956d3b9bc2fap-2}, {0x1.82a0000000000p-1, 0x1.1f9c39f74c557p-2},
    {0x1.8060000000000p-1, 0x1.2596410df963ap-2}, {0x1.7e20000000000p-1, 0x1.2b9943b06bd76p-2},
    {0x1.7be0000000000p-1, 0x1.31a55d07a8591p-2}, {0x1.79c0000000000p-1, 0x1.3763e64645463p-2},
    {0x1.77a0000000000p-1, 0x1.3d2abb3b3b4dfp-2}, {0x1.7560000000000p-1, 0x1.4351b33743eb9p-2},
    {0x1.7340000000000p-1, 0x1.4929e8db4e6e4p-2}, {0x1.7140000000000p-1, 0x1.4eb1f36b07184p-2},
    {0x1.6f20000000000p-1, 0x1.549aec5def881p-2}, {0x1.6d20000000000p-1, 0x1.5a32eb2e4eacbp-2},
    {0x1.6b20000000000p-1, 0x1.5fd2c78c78828p-2}, {0x1.6920000000000p-1, 0x1.657a97b64d437p-2},
    {0x1.6720000000000p-1, 0x1.6b2a72488ad8fp-2}, {0x1.6520000000000p-1, 0x1.70e26e40eb5fap-2},
    {0x1.6340000000000p-1, 0x1.76466197e36dep-2}, {0x1.6140000000000p-1, 0x1.7c0e612785c73p-2},
    {0x1.5f60000000000p-1, 0x1.81818203afc80p-2}, {0x1.5d80000000000p-1, 0x1.86fc19d05148ep-2},
    {0x1.5ba0000000000p-1, 0x1.8c7e3d1c80b30p-2}, {0x1.59e0000000000p-1, 0x1.91a93f1f4a7a8p-2},
    {0x1.5800000000000p-1, 0x1.973a3431356aep-2}, {0x1.5640000000000p-1, 0x1.9c73305d47ebbp-2},
    {0x1.5480000000000p-1, 0x1.a1b3071f75fdap-2}, {0x1.52a0000000000p-1, 0x1.a75a8a89c8c32p-2},
    {0x1.5100000000000p-1, 0x1.ac478d020506fp-2}, {0x1.4f40000000000p-1, 0x1.b19c6125a6f6bp-2},
    {0x1.4d80000000000p-1, 0x1.b6f859e8ef63ap-2}, {0x1.4be0000000000p-1, 0x1.bbf8c95e489bfp-2},
    {0x1.4a20000000000p-1, 0x1.c162bf5df23e5p-2}, {0x1.4880000000000p-1, 0x1.c6704e4016ff8p-2},
    {0x1.46e0000000000p-1, 0x1.cb844750b9995p-2}, {0x1.4540000000000p-1, 0x1.d09ebaee29dd8p-2},
    {0x1.43a0000000000p-1, 0x1.d5bfb9b5ae71fp-2}, {0x1.4200000000000p-1, 0x1.dae75484c9616p-2},
    {0x1.4080000000000p-1, 0x1.dfaf59de8c15dp-2}, {0x1.3ee0000000000p-1, 0x1.e4e3daeddb5f6p-2},
    {0x1.3d60000000000p-1, 0x1.e9b7e6610815ap-2}, {0x1.3be0000000000p-1, 0x1.ee91cce60d249p-2},
    {0x1.3a60000000000p-1, 0x1.f3719cc25c9b0p-2}, {0x1.38e0000000000p-1, 0x1.f857646fd4622p-2},
    {0x1.3760000000000p-1, 0x1.fd43329dc0365p-2}, {0x1.35e0000000000p-1, 0x1.011a8b18f0ed7p-1},
    {0x1.3460000000000p-1, 0x1.03968f24bfdb7p-1}, {0x1.3300000000000p-1, 0x1.05e04c1aa2c06p-1},
    {0x1.3180000000000p-1, 0x1.086248abc4f3bp-1}, {0x1.3020000000000p-1, 0x1.0ab18bf5823c3p-1},
    {0x1.2ec0000000000p-1, 0x1.0d037d237f464p-1}, {0x1.2d60000000000p-1, 0x1.0f5822744fca3p-1},
    {0x1.2be0000000000p-1, 0x1.11e62229bbf4ap-1}, {0x1.2aa0000000000p-1, 0x1.1409a2e6c81dap-1},
    {0x1.2940000000000p-1, 0x1.16668af4dd396p-1}, {0x1.27e0000000000p-1, 0x1.18c640ff75f06p-1},
    {0x1.2680000000000p-1, 0x1.1b28cbb6ec93fp-1}, {0x1.2540000000000p-1, 0x1.1d5650035a98bp-1},
    {0x1.23e0000000000p-1, 0x1.1fbe551db43c1p-1}, {0x1.22a0000000000p-1, 0x1.21f0dfc65ceecp-1},
    {0x1.2160000000000p-1, 0x1.2425d72bd3810p-1}, {0x1.2020000000000p-1, 0x1.265d40adef0b8p-1},
    {0x1.1ec0000000000p-1, 0x1.28d041990b0ebp-1}, {0x1.1d80000000000p-1, 0x1.2b0cdfbf7ad03p-1},
    {0x1.1c60000000000p-1, 0x1.2d1260ad99c76p-1}, {0x1.1b20000000000p-1, 0x1.2f53c9cc59422p-1},
    {0x1.19e0000000000p-1, 0x1.3197c0fa80e6ap-1}, {0x1.18a0000000000p-1, 0x1.33de4c086c40ap-1},
    {0x1.1780000000000p-1, 0x1.35eccf0ac61d0p-1}, {0x1.1640000000000p-1, 0x1.383850278cfd9p-1},
    {0x1.1520000000000p-1, 0x1.3a4b53f86cb2ep-1}, {0x1.1400000000000p-1, 0x1.3c6080c36bfb5p-1},
    {0x1.12c0000000000p-1, 0x1.3eb37978b85b5p-1}, {0x1.11a0000000000p-1, 0x1.40cd448ff6dd6p-1},
    {0x1.1080000000000p-1, 0x1.42e946de080bfp-1}, {0x1.0f60000000000p-1, 0x1.450785145cafep-1},
    {0x1.0e40000000000p-1, 0x1.472803f35eaaep-1}, {0x1.0d20000000000p-1, 0x1.494ac84ab0ed3p-1},
    {0x1.0c00000000000p-1, 0x1.4b6fd6f970c1fp-1}, {0x1.0b00000000000p-1, 0x1.4d59d43fdaba2p-1},
    {0x1.09e0000000000p-1, 0x1.4f8343f9cb679p-1}, {0x1.08c0000000000p-1, 0x1.51af0c774a2d0p-1},
    {0x1.07c0000000000p-1, 0x1.539f107e1d30ap-1}, {0x1.06a0000000000p-1, 0x1.55cf55c5a5438p-1},
    {0x1.05a0000000000p-1, 0x1.57c35f3490184p-1}, {0x1.04a0000000000p-1, 0x1.59b952dcd3e28p-1},
    {0x1.0380000000000p-1, 0x1.5bf053a48690ep-1}, {0x1.0280000000000p-1, 0x1.5dea65985a350p-1},
    {0x1.0180000000000p-1, 0x1.5fe66db228992p-1}, {0x1.0080000000000p-1, 0x1.61e46fda56467p-1},
};

}  // namespace

constexpr double kLog2e = 1.4426950408889634074;

// ---- float64 -----------------------------------------------------------------

// The high word of x as a float: 20 mantissa bits, 0 below 2^-126.
__device__ __forceinline__ float head(double x)
{
    const int hi = __double2hiint(x);
    return __int_as_float((hi & 0x80000000) | (max((hi & 0x7fffffff) - (896 << 20), 0) << 3));
}

// 2^(n/256) and, in p, e^r - 1 for |r| < 2.1e-3
__device__ __forceinline__ double ex_parts(int n, double r, double &p)
{
    double q = fma(r, 1.0 / 24, 1.0 / 6);
    q = fma(q, r, 0.5);
    p = fma(r * r, q, r);
    const double t = __ldg(&kExp2Tab[n & 255]);
    return __hiloint2double(__double2hiint(t) + ((n >> 8) << 20), __double2loint(t));
}

// e^(d s) for |d s| < 700 with the product unrounded: n ln2/256 is
// subtracted from it inside one fma, ln2/256 split so that n times its head
// (35 bits) is exact.  n comes from float32 (sf = 256 log2(e) s): off by at
// most 1/4 more than its rounding, so |r| < 2.1e-3, and < 1.5e-3 for
// |d s| < 60.
constexpr double kLn2_256Hi = 0x1.62e42fef80000p-9, kLn2_256Lo = 0x1.1cf79abc9e3b4p-44;
constexpr float kMagicF = 12582912.f;          // 1.5 * 2^23
constexpr double kMagicD = 4503601774854144.0; // 2^52 + 2^31
__device__ __forceinline__ double ex_scaled(double d, double s, float sf, double &p)
{
    const int n = __float_as_int(fmaf(head(d), sf, kMagicF)) - 0x4b400000;
    const double nd = __hiloint2double(0x43300000, n ^ 0x80000000) - kMagicD;
    double r = fma(d, s, -(nd * kLn2_256Hi));
    r = fma(nd, -kLn2_256Lo, r);
    return ex_parts(n, r, p);
}
__device__ __forceinline__ double ex_scaled(double d, double s, float sf)
{
    double p;
    const double t = ex_scaled(d, s, sf, p);
    return fma(t, p, t);
}
__device__ __forceinline__ double ex(double x)
{
    return ex_scaled(x, 1.0, (float)(256 * kLog2e));
}

// Whether all are finite; whether all are positive, normal and finite.  On
// the bits, beside the float64 pipe.
template <class... A>
__device__ __forceinline__ bool all_finite(A... a)
{
    int m = 0;
    ((m = max(m, __double2hiint(a) & 0x7fffffff)), ...);
    return m < 0x7ff00000;
}
template <class... A>
__device__ __forceinline__ bool all_normal(A... a)
{
    return (((unsigned)(__double2hiint(a) - 0x00100000) < 0x7fe00000u) && ...);
}

// x limited to [-690, 690], on the bits; a NaN (quiet, as arithmetic makes
// them: its high word is above infinity's) stays one
__device__ __forceinline__ double limited(double x)
{
    const int hi = __double2hiint(x), a = hi & 0x7fffffff;
    if (a > 0x40859000 && a <= 0x7ff00000)
        x = __hiloint2double((hi & 0x80000000) | 0x40859000, 0);
    return x;
}
__device__ __forceinline__ double ex_limited(double x) { return ex(limited(x)); }

__device__ static __noinline__ double log_any(double x) { return log(x); }

__device__ __forceinline__ double lg(double x)
{
    const int hi = __double2hiint(x);
    if ((unsigned)(hi - 0x00100000) >= 0x7fe00000u) return log_any(x);
    const int e = (hi >> 20) - 1023;
    const double2 cl = __ldg(&kLogTab[(hi >> 13) & 127]);
    const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
    const double r = fma(m, cl.x, -1.0);
    double q = fma(r, -1.0 / 6, 1.0 / 5);
    q = fma(q, r, -1.0 / 4);
    q = fma(q, r, 1.0 / 3);
    q = fma(q, r, -1.0 / 2);
    const double p = fma(r * r, q, r);
    const double ed = __hiloint2double(0x43300000, e ^ 0x80000000) - kMagicD;
    return fma(ed, 0x1.62e42fefa39efp-1, cl.y) + p;
}

__device__ __forceinline__ double rcp(double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// 1 / d and n / d to about half an ulp, for what a result is proportional to:
// one more residual.
__device__ __forceinline__ double rcp_near(double d)
{
    const double y = rcp(d);
    return fma(y, fma(-d, y, 1.0), y);
}
__device__ __forceinline__ double div_near(double n, double d)
{
    const double y = rcp(d), q = n * y;
    return fma(y, fma(-d, q, n), q);
}

__device__ __forceinline__ double rsq(double d)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d * y, y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// ---- float32 -----------------------------------------------------------------

__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ex(float x) { return ex2(x * (float)kLog2e); }
__device__ __forceinline__ float lg(float x) { return __logf(x); }
__device__ __forceinline__ float rcp(float d)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return y;
}
__device__ __forceinline__ float rcp_near(float d) { return rcp(d); }
__device__ __forceinline__ float div_near(float n, float d)
{
    const float y = rcp(d), q = n * y;
    return fmaf(y, fmaf(-d, q, n), q);
}
__device__ __forceinline__ float rsq(float d)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return y;
}

// n / d under a logarithm: within a few ulp in float64, half of one in
// float32 (whose logarithm is scaled by 27 mV and cancels against u)
__device__ __forceinline__ double quotient(double n, double d) { return n * rcp(d); }
__device__ __forceinline__ float quotient(float n, float d) { return div_near(n, d); }

// ---- both --------------------------------------------------------------------

// e^((u - u0) / d).  float64 takes it from b = e^(u / d), shared by every
// rate with this slope, as b k, k = e^(-u0 / d): one product.  float32 forms
// each from its own difference, whose exponential is accurate where the rate
// bends.
template <class T>
struct Slope {
    T b;   // float64: e^(u / d); float32: u
};
__device__ __forceinline__ double slope_at(const Slope<double> &g, double k, float, float)
{
    return g.b * k;
}
__device__ __forceinline__ float slope_at(const Slope<float> &g, double, float u0, float c)
{
    return ex2((g.b - u0) * c);
}
#define FW_AT(G, U0, D, K) \
    fw::dm::slope_at(G, K, (float)(U0), (float)(fw::dm::kLog2e / (D)))
__device__ __forceinline__ Slope<float> slope(float u, double, float) { return {u}; }
__device__ __forceinline__ Slope<double> slope(double u, double s, float sf)
{
    return {ex_scaled(u, s, sf)};
}
#define FW_SLOPE(U, D) \
    fw::dm::slope(U, 1.0 / (D), (float)(256 * fw::dm::kLog2e / (D)))
__device__ __forceinline__ Slope<float> squared(const Slope<float> &g) { return g; }
__device__ __forceinline__ Slope<double> squared(const Slope<double> &g)
{
    return {g.b * g.b};
}

// e^(x s), s a compile-time constant
__device__ __forceinline__ double ex_by(double x, double s, float sf, float)
{
    return ex_scaled(x, s, sf);
}
__device__ __forceinline__ float ex_by(float x, double, float, float c) { return ex2(x * c); }
#define FW_EX(X, S)                                                 \
    fw::dm::ex_by(X, (double)(S), (float)(256 * fw::dm::kLog2e * (S)), \
                  (float)(fw::dm::kLog2e * (S)))

// The same, float32 rounding x s before it is scaled for ex2, which has no
// rounding of log2(e) s for an error of every argument: one product more.
__device__ __forceinline__ double ex_of(double x, double s, float sf, float)
{
    return ex_scaled(x, s, sf);
}
__device__ __forceinline__ float ex_of(float x, double, float, float s) { return ex(x * s); }
#define FW_EX_OF(X, S) \
    fw::dm::ex_of(X, (double)(S), (float)(256 * fw::dm::kLog2e * (S)), (float)(S))

// What a step of dt does to a gate of the given rate, and the gate's next
// value inf - (inf - x) e^(-dt rate).  ndt is -dt in float64, where the
// exponential less one is formed without rounding the exponential first and
// added to x (most gates are slow: it is 1e-3 or less); -dt log2(e) in
// float32, where it is the exponential.
__device__ __forceinline__ double decay(double ndt, double rate)
{
    double p;
    const double t = ex_scaled(limited(ndt * rate), 1.0, (float)(256 * kLog2e), p);
    return fma(t, p, t - 1.0);
}
__device__ __forceinline__ double gate_to(double x, double inf, double decay)
{
    return fma(x - inf, decay, x);
}
// A gate faster than the step (most of the way to inf): the exponential as
// it is keeps inf's digits.
__device__ __forceinline__ double gate_fast(double x, double inf, double ndt, double rate)
{
    return fma(x - inf, ex_limited(ndt * rate), inf);
}
__device__ __forceinline__ float gate_fast(float x, float inf, float ndt, float rate)
{
    return inf - (inf - x) * ex2(ndt * rate);
}
__device__ __forceinline__ float decay(float ndt, float rate) { return ex2(ndt * rate); }
__device__ __forceinline__ float gate_to(float x, float inf, float decay)
{
    return inf - (inf - x) * decay;
}

// x / (e^x - 1), given e = e^x.  float64: as it stands, like the models'
// expressions, and like theirs NaN at x = 0 and infinite where e rounds to 1
// (Courtemanche's beta_xr at the potential next above 3.3328 mV).  float32:
// the series of the Bernoulli numbers up to |x| = 1/2 (next term
// x^10 / 47900160), where the difference would lose digits.
__device__ __forceinline__ double x_over_expm1(double x, double e)
{
    const double d = e - 1.0;
    double y = rcp(d);   // NaN for d = 0
    if ((__double2hiint(d) | __double2loint(d)) == 0)
        y = __hiloint2double(0x7ff00000, 0);
    return x * y;
}
__device__ __forceinline__ float x_over_expm1(float x, float e)
{
    const float x2 = x * x;
    float s = fmaf(x2, (float)(-1.0 / 1209600), (float)(1.0 / 30240));
    s = fmaf(s, x2, (float)(-1.0 / 720));
    s = fmaf(s, x2, (float)(1.0 / 12));
    s = fmaf(s, x2, fmaf(x, -0.5f, 1.f));
    return fabsf(x) < 0.5f ? s : x * rcp(e - 1.f);
}

}  // namespace dm
}  // namespace fw
