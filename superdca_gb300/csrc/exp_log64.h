// exp_log64.h -- FP64 exp, log and reciprocal over the ranges a node belief
// needs: exp(x) for x <= 0, log(z) and 1 / z for 1 <= z <= 4.
//
// GB300 does some two FP64 operations per clock and SM, so the count of them
// is the time of a belief.  Both functions are table driven (P. T. P. Tang,
// ACM TOMS 15(2), 1989 and 16(4), 1990): a table value at the nearest of 128
// points per octave leaves a remainder so short that the Taylor polynomial
// ends at the fifth (exp) and eighth (log) power, 11 operations each; the
// reciprocal takes three from a single-precision start.  The tables keep the
// rounding error of their values beside them, so the results are within 0.53
// (exp), 0.85 (log) and 0.53 (reciprocal) units in the last place.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define SDCA_EL_HD __host__ __device__ __forceinline__
#define SDCA_EL_TAB __device__ const
#else
#define SDCA_EL_HD inline
#define SDCA_EL_TAB const
#endif

namespace sdca {

struct ExpTab {
    double t, rel;   // 2^(j / 128) rounded, its rounding error relative to t
};
struct LogTab {
    double rc, hi, lo;   // near 1 / c of the interval's middle c, in eleven bits (z rc - 1 is
                         // then all but exact); -log(rc) in two parts
};

constexpr int EXP_N = 128, LOG_N = 257;

// 2^(j / 128)
SDCA_EL_TAB ExpTab kExpTab[EXP_N] = {
    {0x1p+0, 0}, {0x1.0163da9fb3335p+0, 0x1.b3b4f2p-54},
    {0x1.02c9a3e778061p+0, -0x1.16013ap-56}, {0x1.04315e86e7f85p+0, -0x1.05e7a2p-54},
    {0x1.059b0d3158574p+0, 0x1.cd2524p-55}, {0x1.0706b29ddf6dep+0, -0x1.bce802p-55},
    {0x1.0874518759bc8p+0, 0x1.0f74e6p-57}, {0x1.09e3ecac6f383p+0, 0x1.0a3e46p-54},
    {0x1.0b5586cf9890fp+0, 0x1.79aa66p-54}, {0x1.0cc922b7247f7p+0, 0x1.eb51aap-55},
    {0x1.0e3ec32d3d1a2p+0, 0x1.ebe3d8p-60}, {0x1.0fb66affed31bp+0, -0x1.a03348p-57},
    {0x1.11301d0125b51p+0, -0x1.556522p-54}, {0x1.12abdc06c31ccp+0, -0x1.080ef8p-58},
    {0x1.1429aaea92dep+0, -0x1.1c923cp-54}, {0x1.15a98c8a58e51p+0, 0x1.0d3e3ep-55},
    {0x1.172b83c7d517bp+0, -0x1.01b15ep-55}, {0x1.18af9388c8deap+0, -0x1.f1ff06p-55},
    {0x1.1a35beb6fcb75p+0, 0x1.b898c4p-55}, {0x1.1bbe084045cd4p+0, -0x1.6d99c8p-54},
    {0x1.1d4873168b9aap+0, 0x1.aecf74p-54}, {0x1.1ed5022fcd91dp+0, -0x1.fe782cp-55},
    {0x1.2063b88628cd6p+0, 0x1.a6f414p-55}, {0x1.21f49917ddc96p+0, 0x1.07a05cp-55},
    {0x1.2387a6e756238p+0, 0x1.68efdep-54}, {0x1.251ce4fb2a63fp+0, 0x1.75e19p-55},
    {0x1.26b4565e27cddp+0, 0x1.0472bap-55}, {0x1.284dfe1f56381p+0, -0x1.6b87b4p-54},
    {0x1.29e9df51fdee1p+0, 0x1.2f7e16p-55}, {0x1.2b87fd0dad99p+0, -0x1.d219b2p-60},
    {0x1.2d285a6e4030bp+0, 0x1.b37828p-55}, {0x1.2ecafa93e2f56p+0, 0x1.e14928p-57},
    {0x1.306fe0a31b715p+0, 0x1.34d754p-55}, {0x1.32170fc4cd831p+0, 0x1.64201ep-55},
    {0x1.33c08b26416ffp+0, 0x1.fdd396p-55}, {0x1.356c55f929ff1p+0, -0x1.6a3804p-55},
    {0x1.371a7373aa9cbp+0, -0x1.24aedcp-54}, {0x1.38cae6d05d866p+0, -0x1.907f82p-54},
    {0x1.3a7db34e59ff7p+0, -0x1.1d1e84p-56}, {0x1.3c32dc313a8e5p+0, -0x1.91919cp-54},
    {0x1.3dea64c123422p+0, 0x1.59f48ap-55}, {0x1.3fa4504ac801cp+0, -0x1.312608p-54},
    {0x1.4160a21f72e2ap+0, -0x1.8a78f4p-58}, {0x1.431f5d950a897p+0, -0x1.c2c9b6p-56},
    {0x1.44e086061892dp+0, 0x1.363ed6p-59}, {0x1.46a41ed1d0057p+0, 0x1.666094p-54},
    {0x1.486a2b5c13cdp+0, 0x1.ecce1ep-57}, {0x1.4a32af0d7d3dep+0, 0x1.3ff8e4p-54},
    {0x1.4bfdad5362a27p+0, 0x1.690cecp-56}, {0x1.4dcb299fddd0dp+0, 0x1.31dbdep-54},
    {0x1.4f9b2769d2ca7p+0, -0x1.f9434p-55}, {0x1.516daa2cf6642p+0, -0x1.7deccep-55},
    {0x1.5342b569d4f82p+0, -0x1.8dec6cp-56}, {0x1.551a4ca5d920fp+0, -0x1.61246ep-55},
    {0x1.56f4736b527dap+0, 0x1.335052p-54}, {0x1.58d12d497c7fdp+0, 0x1.b98b72p-56},
    {0x1.5ab07dd485429p+0, 0x1.063e1ep-54}, {0x1.5c9268a5946b7p+0, 0x1.4c7856p-60},
    {0x1.5e76f15ad2148p+0, 0x1.432e62p-54}, {0x1.605e1b976dc09p+0, -0x1.ce44a6p-55},
    {0x1.6247eb03a5585p+0, -0x1.c33c54p-55}, {0x1.6434634ccc32p+0, -0x1.453788p-55},
    {0x1.6623882552225p+0, -0x1.3cedd8p-54}, {0x1.68155d44ca973p+0, 0x1.710aa8p-58},
    {0x1.6a09e667f3bcdp+0, -0x1.3b3efcp-54}, {0x1.6c012750bdabfp+0, -0x1.a12ad8p-57},
    {0x1.6dfb23c651a2fp+0, -0x1.367efcp-57}, {0x1.6ff7df9519484p+0, -0x1.0dc3d6p-55},
    {0x1.71f75e8ec5f74p+0, -0x1.81f648p-56}, {0x1.73f9a48a58174p+0, -0x1.6ee4acp-55},
    {0x1.75feb564267c9p+0, -0x1.619322p-55}, {0x1.780694fde5d3fp+0, 0x1.09ccb6p-54},
    {0x1.7a11473eb0187p+0, -0x1.b32dccp-56}, {0x1.7c1ed0130c132p+0, 0x1.4ecfd6p-54},
    {0x1.7e2f336cf4e62p+0, 0x1.5ebe1ap-57}, {0x1.80427543e1a12p+0, -0x1.8a1c52p-55},
    {0x1.82589994cce13p+0, -0x1.369b7p-54}, {0x1.8471a4623c7adp+0, -0x1.05e844p-55},
    {0x1.868d99b4492edp+0, -0x1.4d450ep-54}, {0x1.88ac7d98a6699p+0, 0x1.0ad676p-54},
    {0x1.8ace5422aa0dbp+0, 0x1.db72fcp-55}, {0x1.8cf3216b5448cp+0, -0x1.5b660ap-57},
    {0x1.8f1ae99157736p+0, 0x1.bf6836p-56}, {0x1.9145b0b91ffc6p+0, -0x1.3091fap-54},
    {0x1.93737b0cdc5e5p+0, -0x1.da9b88p-58}, {0x1.95a44cbc8520fp+0, -0x1.c23f98p-57},
    {0x1.97d829fde4e5p+0, -0x1.243432p-54}, {0x1.9a0f170ca07bap+0, -0x1.5ca6cep-55},
    {0x1.9c49182a3f09p+0, 0x1.1affc2p-56}, {0x1.9e86319e32323p+0, 0x1.dd235ep-57},
    {0x1.a0c667b5de565p+0, -0x1.7c5042p-55}, {0x1.a309bec4a2d33p+0, 0x1.b1c86ep-55},
    {0x1.a5503b23e255dp+0, -0x1.1bbd1ep-54}, {0x1.a799e1330b358p+0, 0x1.0cc31ap-54},
    {0x1.a9e6b5579fdbfp+0, 0x1.469846p-55}, {0x1.ac36bbfd3f37ap+0, -0x1.2dfcdap-55},
    {0x1.ae89f995ad3adp+0, 0x1.c1a77ap-55}, {0x1.b0e07298db666p+0, -0x1.07b8f4p-54},
    {0x1.b33a2b84f15fbp+0, -0x1.5c3d96p-58}, {0x1.b59728de5593ap+0, -0x1.0a40e4p-54},
    {0x1.b7f76f2fb5e47p+0, -0x1.8d6f44p-57}, {0x1.ba5b030a1064ap+0, -0x1.1eee26p-54},
    {0x1.bcc1e904bc1d2p+0, 0x1.4ffd7p-56}, {0x1.bf2c25bd71e09p+0, -0x1.1bdfcp-54},
    {0x1.c199bdd85529cp+0, 0x1.36eae4p-56}, {0x1.c40ab5fffd07ap+0, 0x1.ee3326p-55},
    {0x1.c67f12e57d14bp+0, 0x1.4e08fep-55}, {0x1.c8f6d9406e7b5p+0, 0x1.3cdaf4p-57},
    {0x1.cb720dcef9069p+0, 0x1.76b2c6p-57}, {0x1.cdf0b555dc3fap+0, -0x1.08a188p-55},
    {0x1.d072d4a07897cp+0, -0x1.fad5d4p-55}, {0x1.d2f87080d89f2p+0, -0x1.00dae4p-54},
    {0x1.d5818dcfba487p+0, 0x1.4a385ap-56}, {0x1.d80e316c98398p+0, -0x1.2919e2p-55},
    {0x1.da9e603db3285p+0, 0x1.e5a50ep-55}, {0x1.dd321f301b46p+0, 0x1.43a59ap-55},
    {0x1.dfc97337b9b5fp+0, -0x1.2d521p-55}, {0x1.e264614f5a129p+0, -0x1.92ab94p-55},
    {0x1.e502ee78b3ff6p+0, 0x1.4b6046p-56}, {0x1.e7a51fbc74c83p+0, 0x1.3c5ec6p-55},
    {0x1.ea4afa2a490dap+0, -0x1.ff7128p-55}, {0x1.ecf482d8e67f1p+0, -0x1.dae98ep-55},
    {0x1.efa1bee615a27p+0, 0x1.ec3bc4p-55}, {0x1.f252b376bba97p+0, 0x1.42b94cp-55},
    {0x1.f50765b6e454p+0, 0x1.a64a94p-55}, {0x1.f7bfdad9cbe14p+0, -0x1.e37baep-55},
    {0x1.fa7c1819e90d8p+0, 0x1.7893b4p-56}, {0x1.fd3c22b8f71f1p+0, 0x1.305c14p-58},
};

// the interval [1 + i / 128, 1 + (i + 1) / 128) for i < 128, twice that
// beyond, and z = 4; the first has c = 1, so that log keeps its relative
// precision near 1
SDCA_EL_TAB LogTab kLogTab[LOG_N] = {
    {0x1p+0, 0, 0}, {0x1.fap-1, 0x1.82448a388a2aap-7, 0x1.04b162p-62},
    {0x1.f64p-1, 0x1.3b024b78c5669p-6, 0x1.e23a02p-60}, {0x1.f24p-1, 0x1.be0422fcd68f6p-6, 0x1.0a1fccp-61},
    {0x1.ee8p-1, 0x1.1ce5a62bc353ap-5, -0x1.c3939p-59}, {0x1.ebp-1, 0x1.5715c4c03ceefp-5, -0x1.bbf88ep-61},
    {0x1.e74p-1, 0x1.95e430f8ce45ep-5, -0x1.67bb44p-60}, {0x1.e3cp-1, 0x1.d0f2c1dda671cp-5, -0x1.c7de3ep-62},
    {0x1.ep-1, 0x1.08598b59e3a07p-4, -0x1.dd700ap-58}, {0x1.dccp-1, 0x1.242d6c1a58a5cp-4, 0x1.c56324p-60},
    {0x1.d94p-1, 0x1.425bce84749b3p-4, -0x1.4eb798p-59}, {0x1.d5cp-1, 0x1.60c38ba79945dp-4, -0x1.3bc514p-58},
    {0x1.d28p-1, 0x1.7d33687c293c9p-4, -0x1.cf063ep-58}, {0x1.cf4p-1, 0x1.99d62a65eb96fp-4, -0x1.d04f98p-58},
    {0x1.ccp-1, 0x1.b6ac88dad5b1cp-4, -0x1.0057eep-59}, {0x1.c8cp-1, 0x1.d3b73f37e1f9bp-4, -0x1.fd984cp-58},
    {0x1.c58p-1, 0x1.f0f70cdd992e3p-4, 0x1.f6c272p-60}, {0x1.c28p-1, 0x1.06135354d4b18p-3, 0x1.18a0dp-58},
    {0x1.bf4p-1, 0x1.14e75b489fffp-3, -0x1.ee648p-58}, {0x1.bc4p-1, 0x1.22aff2ddbd971p-3, -0x1.535834p-60},
    {0x1.b94p-1, 0x1.3090733ce39fap-3, -0x1.b90764p-57}, {0x1.b64p-1, 0x1.3e892fe9956dbp-3, -0x1.526eb2p-57},
    {0x1.b38p-1, 0x1.4b6d6fefe22a4p-3, 0x1.767ab8p-57}, {0x1.b08p-1, 0x1.59958ff1d52f1p-3, 0x1.f4d12cp-57},
    {0x1.adcp-1, 0x1.66a5d42a3ad34p-3, 0x1.26754p-57}, {0x1.abp-1, 0x1.73cb9074fd14dp-3, -0x1.521ap-57},
    {0x1.a84p-1, 0x1.81070bd7b9008p-3, -0x1.7f5998p-61}, {0x1.a58p-1, 0x1.8e588ebac2dbfp-3, -0x1.46a9a6p-57},
    {0x1.a2cp-1, 0x1.9bc062f26fc3ap-3, 0x1.b03014p-57}, {0x1.ap-1, 0x1.a93ed3c8ad9e3p-3, 0x1.bcafaap-57},
    {0x1.9d8p-1, 0x1.b5971a213acdbp-3, -0x1.e2f8aap-57}, {0x1.9bp-1, 0x1.c2028ab17f9b4p-3, 0x1.f11aa4p-57},
    {0x1.984p-1, 0x1.cfc25714bdcfep-3, -0x1.6658fep-59}, {0x1.95cp-1, 0x1.dc56cae452f5ap-3, -0x1.0abb64p-57},
    {0x1.934p-1, 0x1.e8ff2622babc7p-3, 0x1.3d3398p-60}, {0x1.90cp-1, 0x1.f5bba83060a0ep-3, -0x1.b56b78p-57},
    {0x1.8e8p-1, 0x1.00a1c6adda473p-2, 0x1.8d688cp-56}, {0x1.8cp-1, 0x1.07138604d5862p-2, 0x1.cdb16ep-56},
    {0x1.898p-1, 0x1.0d8fb813eb1efp-2, -0x1.cdde2cp-56}, {0x1.874p-1, 0x1.136ef02e8290cp-2, -0x1.60c396p-58},
    {0x1.85p-1, 0x1.1956d3b9bc2fap-2, 0x1.7b9d68p-56}, {0x1.82cp-1, 0x1.1f477c75732dbp-2, -0x1.2bfef2p-57},
    {0x1.808p-1, 0x1.25410494e56c7p-2, 0x1.7ac0fp-56}, {0x1.7e4p-1, 0x1.2b4386c168f0cp-2, 0x1.39d1a2p-58},
    {0x1.7cp-1, 0x1.314f1e1d35ce4p-2, -0x1.3d699p-56}, {0x1.79cp-1, 0x1.3763e64645463p-2, -0x1.c1adc4p-57},
    {0x1.778p-1, 0x1.3d81fb5946dbap-2, 0x1.c1eab2p-56}, {0x1.758p-1, 0x1.42f9f3ff62642p-2, -0x1.bbf082p-56},
    {0x1.734p-1, 0x1.4929e8db4e6e4p-2, 0x1.5955b2p-58}, {0x1.714p-1, 0x1.4eb1f36b07184p-2, 0x1.1d1b96p-60},
    {0x1.6f4p-1, 0x1.5441aecbc624bp-2, 0x1.ccc012p-58}, {0x1.6dp-1, 0x1.5a8cadbbedfa1p-2, -0x1.e6c2bep-58},
    {0x1.6bp-1, 0x1.602d08af091ecp-2, -0x1.6e892p-58}, {0x1.69p-1, 0x1.65d558d4ce00bp-2, -0x1.7605a4p-56},
    {0x1.67p-1, 0x1.6b85b4cffa3fdp-2, -0x1.8af2c8p-57}, {0x1.654p-1, 0x1.7086b1162b43fp-2, -0x1.d310aap-57},
    {0x1.634p-1, 0x1.76466197e36dep-2, 0x1.375c5ep-59}, {0x1.614p-1, 0x1.7c0e612785c73p-2, 0x1.8f7138p-56},
    {0x1.5f8p-1, 0x1.812444990af63p-2, -0x1.f4a666p-58}, {0x1.5d8p-1, 0x1.86fc19d05148ep-2, 0x1.fc8edcp-56},
    {0x1.5bcp-1, 0x1.8c1ffe400225p-2, -0x1.e89afap-56}, {0x1.59cp-1, 0x1.920800ccb9636p-2, -0x1.d11a16p-56},
    {0x1.58p-1, 0x1.973a3431356aep-2, -0x1.89d282p-57}, {0x1.564p-1, 0x1.9c73305d47ebbp-2, 0x1.eec9c8p-58},
    {0x1.548p-1, 0x1.a1b3071f75fdap-2, 0x1.ac97bap-56}, {0x1.52cp-1, 0x1.a6f9ca8cbc563p-2, 0x1.4a8c5p-56},
    {0x1.51p-1, 0x1.ac478d020506fp-2, 0x1.d19914p-61}, {0x1.4f4p-1, 0x1.b19c6125a6f6bp-2, -0x1.6b77a4p-57},
    {0x1.4d8p-1, 0x1.b6f859e8ef63ap-2, -0x1.9a1efp-60}, {0x1.4bcp-1, 0x1.bc5b8a89b5bf8p-2, 0x1.ea98eap-60},
    {0x1.4a4p-1, 0x1.c0ff81c7055ddp-2, -0x1.4b43a2p-57}, {0x1.488p-1, 0x1.c6704e4016ff8p-2, 0x1.e960f2p-57},
    {0x1.46cp-1, 0x1.cbe88b44dc02bp-2, -0x1.e97fdap-56}, {0x1.454p-1, 0x1.d09ebaee29dd8p-2, -0x1.e7829p-56},
    {0x1.43cp-1, 0x1.d55a7df2b1e7ap-2, -0x1.104cdep-57}, {0x1.42p-1, 0x1.dae75484c9616p-2, -0x1.0b5838p-56},
    {0x1.408p-1, 0x1.dfaf59de8c15dp-2, 0x1.29fcb2p-56}, {0x1.3fp-1, 0x1.e47d1d32e677ep-2, 0x1.96e556p-58},
    {0x1.3d4p-1, 0x1.ea1f2acdd505dp-2, -0x1.33cd58p-56}, {0x1.3bcp-1, 0x1.eef98ee3339ffp-2, 0x1.8e479ep-58},
    {0x1.3a4p-1, 0x1.f3d9dd82ab0afp-2, -0x1.24d154p-56}, {0x1.38cp-1, 0x1.f8c0252a83115p-2, 0x1.62df36p-58},
    {0x1.374p-1, 0x1.fdac748e8717dp-2, -0x1.4961fep-56}, {0x1.35cp-1, 0x1.014f6d4c876bep-1, -0x1.0280b6p-55},
    {0x1.348p-1, 0x1.03617096e0952p-1, 0x1.06614p-55}, {0x1.33p-1, 0x1.05e04c1aa2c06p-1, 0x1.862e54p-60},
    {0x1.318p-1, 0x1.086248abc4f3bp-1, -0x1.263d54p-55}, {0x1.3p-1, 0x1.0ae76e2d054fap-1, 0x1.0d711p-55},
    {0x1.2ecp-1, 0x1.0d037d237f464p-1, -0x1.f0e4a4p-56}, {0x1.2d4p-1, 0x1.0f8e82913feefp-1, -0x1.ea25e2p-55},
    {0x1.2cp-1, 0x1.11af823c75aa8p-1, -0x1.91eee8p-55}, {0x1.2a8p-1, 0x1.1440833add112p-1, -0x1.210abap-55},
    {0x1.294p-1, 0x1.16668af4dd396p-1, -0x1.6061a6p-55}, {0x1.27cp-1, 0x1.18fda3ecf6611p-1, -0x1.4374ap-55},
    {0x1.268p-1, 0x1.1b28cbb6ec93fp-1, -0x1.d68922p-55}, {0x1.254p-1, 0x1.1d5650035a98bp-1, -0x1.0bc702p-55},
    {0x1.24p-1, 0x1.1f8635fc61659p-1, -0x1.2165p-56}, {0x1.22cp-1, 0x1.21b882dd2604p-1, -0x1.ce3482p-55},
    {0x1.214p-1, 0x1.245e78a85f452p-1, -0x1.ce819ep-55}, {0x1.2p-1, 0x1.269621134db92p-1, 0x1.e0efaep-55},
    {0x1.1ecp-1, 0x1.28d041990b0ebp-1, -0x1.5a1b1cp-55}, {0x1.1d8p-1, 0x1.2b0cdfbf7ad03p-1, -0x1.6dbf9ep-55},
    {0x1.1c4p-1, 0x1.2d4c011f1d39ap-1, -0x1.4932ep-55}, {0x1.1bp-1, 0x1.2f8dab636337ap-1, -0x1.98117p-55},
    {0x1.1ap-1, 0x1.315da4434068bp-1, 0x1.6c3a6p-57}, {0x1.18cp-1, 0x1.33a3ed10da62dp-1, -0x1.41af4p-57},
    {0x1.178p-1, 0x1.35eccf0ac61dp-1, -0x1.e6916cp-56}, {0x1.164p-1, 0x1.383850278cfd9p-1, -0x1.75e152p-55},
    {0x1.15p-1, 0x1.3a86767257111p-1, 0x1.700f44p-56}, {0x1.14p-1, 0x1.3c6080c36bfb5p-1, 0x1.19306p-56},
    {0x1.12cp-1, 0x1.3eb37978b85b5p-1, 0x1.9ae16cp-55}, {0x1.11cp-1, 0x1.409167679dd9ap-1, -0x1.4c608p-55},
    {0x1.108p-1, 0x1.42e946de080bfp-1, 0x1.028b26p-60}, {0x1.0f4p-1, 0x1.4543e863c00cap-1, 0x1.1fc3ap-58},
    {0x1.0e4p-1, 0x1.472803f35eaaep-1, -0x1.f291ccp-56}, {0x1.0d4p-1, 0x1.490deaf1a3fc8p-1, -0x1.7244dcp-55},
    {0x1.0cp-1, 0x1.4b6fd6f970c1fp-1, 0x1.c457b6p-55}, {0x1.0bp-1, 0x1.4d59d43fdaba2p-1, -0x1.34d6c8p-57},
    {0x1.09cp-1, 0x1.4fc0e728a3886p-1, -0x1.c1fe76p-56}, {0x1.08cp-1, 0x1.51af0c774a2dp-1, 0x1.72deaep-58},
    {0x1.07cp-1, 0x1.539f107e1d30ap-1, -0x1.57172ap-56}, {0x1.06cp-1, 0x1.5590f6e02f842p-1, -0x1.93c894p-57},
    {0x1.058p-1, 0x1.580202c6c7353p-1, -0x1.e49596p-58}, {0x1.048p-1, 0x1.59f833f9d429p-1, -0x1.654746p-62},
    {0x1.038p-1, 0x1.5bf053a48690ep-1, 0x1.9d1fa2p-59}, {0x1.028p-1, 0x1.5dea65985a35p-1, -0x1.733688p-56},
    {0x1.018p-1, 0x1.5fe66db228992p-1, 0x1.c54626p-58}, {0x1.008p-1, 0x1.61e46fda56467p-1, -0x1.ee18bap-56},
    {0x1.fep-2, 0x1.64e5309aceb06p-1, -0x1.7e2842p-55}, {0x1.fap-2, 0x1.68ed421885c7ap-1, -0x1.102356p-56},
    {0x1.f64p-2, 0x1.6cbc424b69ca3p-1, -0x1.fb093ep-55}, {0x1.f24p-2, 0x1.70d451078a537p-1, -0x1.97ca3cp-57},
    {0x1.ee8p-2, 0x1.74b28a525fd43p-1, -0x1.8ca88ep-56}, {0x1.ebp-2, 0x1.78558c3ba76dep-1, 0x1.1dea2p-56},
    {0x1.e74p-2, 0x1.7c4272ff30835p-1, 0x1.2a9c5ep-57}, {0x1.e3cp-2, 0x1.7ff35c0d7e061p-1, -0x1.6d5656p-58},
    {0x1.ep-2, 0x1.83ef615ae013p-1, 0x1.a36f0ap-59}, {0x1.dccp-2, 0x1.8769dd72eeb3bp-1, -0x1.1beff6p-55},
    {0x1.d94p-2, 0x1.8b2fa9c032326p-1, -0x1.bf0688p-55}, {0x1.d5cp-2, 0x1.8efca16496c7bp-1, -0x1.a32762p-56},
    {0x1.d28p-2, 0x1.928a9cff28c68p-1, 0x1.1c042ap-55}, {0x1.cf4p-2, 0x1.961ef53c6111dp-1, 0x1.bdafeep-59},
    {0x1.ccp-2, 0x1.99b9c10afe553p-1, -0x1.3a208ep-55}, {0x1.c8cp-2, 0x1.9d5b17d69fde3p-1, -0x1.e9ce18p-55},
    {0x1.c58p-2, 0x1.a103118b56c4cp-1, -0x1.9a64fap-55}, {0x1.c28p-2, 0x1.a46904c4d8cb5p-1, 0x1.f1f218p-56},
    {0x1.bf4p-2, 0x1.a81e06c1cb9ebp-1, 0x1.3030c4p-56}, {0x1.bc4p-2, 0x1.ab902ca71304bp-1, 0x1.cb4a3p-55},
    {0x1.b94p-2, 0x1.af084cbedc86ep-1, -0x1.985ce8p-55}, {0x1.b64p-2, 0x1.b2867bea08fa6p-1, -0x1.fadaecp-57},
    {0x1.b38p-2, 0x1.b5bf8beb9c298p-1, 0x1.3383ap-55}, {0x1.b08p-2, 0x1.b94993ec18eacp-1, -0x1.ace6c4p-55},
    {0x1.adcp-2, 0x1.bc8da4fa3253cp-1, 0x1.1f8242p-55}, {0x1.abp-2, 0x1.bfd7140ce2e42p-1, 0x1.815e72p-55},
    {0x1.a84p-2, 0x1.c325f2e591df1p-1, 0x1.9fcf16p-56}, {0x1.a58p-2, 0x1.c67a539e5455fp-1, -0x1.ef15dep-57},
    {0x1.a2cp-2, 0x1.c9d448ac3f8fep-1, -0x1.7c1e12p-56}, {0x1.ap-2, 0x1.cd33e4e1cf068p-1, 0x1.144372p-57},
    {0x1.9d8p-2, 0x1.d049f677f2526p-1, -0x1.45b272p-56}, {0x1.9bp-2, 0x1.d364d29c0385cp-1, 0x1.522b9ap-55},
    {0x1.984p-2, 0x1.d6d4c5b4d312fp-1, -0x1.40809ep-55}, {0x1.95cp-2, 0x1.d9f9e2a8b85c6p-1, -0x1.6cc9e8p-55},
    {0x1.934p-2, 0x1.dd23f978524e1p-1, -0x1.018b8cp-58}, {0x1.90cp-2, 0x1.e05319fbbbc73p-1, -0x1.9775ecp-55},
    {0x1.8e8p-2, 0x1.e335134690c29p-1, -0x1.8d9b22p-57}, {0x1.8cp-2, 0x1.e66df2f20e62p-1, 0x1.bcbdaap-55},
    {0x1.898p-2, 0x1.e9ac0bf9992e6p-1, 0x1.eef5dcp-55}, {0x1.874p-2, 0x1.ec9ba806e4e75p-1, 0x1.5398fep-56},
    {0x1.85p-2, 0x1.ef8f99cc81b6cp-1, 0x1.93b3a6p-55}, {0x1.82cp-2, 0x1.f287ee2a5d35dp-1, -0x1.751acap-55},
    {0x1.808p-2, 0x1.f584b23a16553p-1, -0x1.b2ea5ap-57}, {0x1.7e4p-2, 0x1.f885f35058175p-1, 0x1.fa3e4cp-56},
    {0x1.7cp-2, 0x1.fb8bbefe3e861p-1, 0x1.b9814cp-58}, {0x1.79cp-2, 0x1.fe962312c6421p-1, -0x1.9a868p-55},
    {0x1.778p-2, 0x1.00d296ce23866p+0, 0x1.b6da4ap-55}, {0x1.758p-2, 0x1.023094f7aa688p+0, -0x1.0269f2p-60},
    {0x1.734p-2, 0x1.03bc922ea56b1p+0, -0x1.7f782cp-54}, {0x1.714p-2, 0x1.051e94d293959p+0, -0x1.909918p-54},
    {0x1.6f4p-2, 0x1.068283aac358ap+0, 0x1.87be7ap-54}, {0x1.6dp-2, 0x1.08154366cd4ep+0, -0x1.66f366p-55},
    {0x1.6bp-2, 0x1.097d5a2394173p+0, -0x1.abf61ap-54}, {0x1.69p-2, 0x1.0ae76e2d054fap+0, 0x1.0d711p-54},
    {0x1.67p-2, 0x1.0c53852bd05f7p+0, -0x1.8cd7cp-55}, {0x1.654p-2, 0x1.0d93c43d5ca07p+0, 0x1.309064p-54},
    {0x1.634p-2, 0x1.0f03b05dcaaafp+0, 0x1.d2b57p-56}, {0x1.614p-2, 0x1.1075b041b3414p+0, 0x1.cecec8p-54},
    {0x1.5f8p-2, 0x1.11bb291e148dp+0, 0x1.4ba812p-54}, {0x1.5d8p-2, 0x1.13311e6be621bp+0, 0x1.d42c6p-55},
    {0x1.5bcp-2, 0x1.147a1787d258bp+0, 0x1.f0cbbap-54}, {0x1.59cp-2, 0x1.15f4182b00285p+0, -0x1.2a818cp-59},
    {0x1.58p-2, 0x1.1740a5041f2a3p+0, 0x1.cdc146p-57}, {0x1.564p-2, 0x1.188ee40f23ca6p+0, 0x1.89df16p-54},
    {0x1.548p-2, 0x1.19ded9bfaf4eep+0, 0x1.ac30dp-55}, {0x1.52cp-2, 0x1.1b308a9b00e5p+0, 0x1.bd958ep-54},
    {0x1.51p-2, 0x1.1c83fb3853113p+0, 0x1.6e95acp-54}, {0x1.4f4p-2, 0x1.1dd930413b8d2p+0, 0x1.3d8384p-54},
    {0x1.4d8p-2, 0x1.1f302e720da86p+0, 0x1.9227f4p-56}, {0x1.4bcp-2, 0x1.2088fa9a3f3f6p+0, -0x1.8d6324p-54},
    {0x1.4a4p-2, 0x1.21b1f8699326fp+0, -0x1.7cebf6p-55}, {0x1.488p-2, 0x1.230e2b87d78f6p+0, -0x1.57e168p-54},
    {0x1.46cp-2, 0x1.246c3ac908d02p+0, 0x1.e12504p-55}, {0x1.454p-2, 0x1.2599c6b35c46dp+0, 0x1.f111d4p-54},
    {0x1.43cp-2, 0x1.26c8b7747e496p+0, 0x1.23a374p-56}, {0x1.42p-2, 0x1.282bed190427dp+0, 0x1.40e35ap-57},
    {0x1.408p-2, 0x1.295dee6f74d4fp+0, -0x1.2a396cp-56}, {0x1.3fp-2, 0x1.2a915f448b6d7p+0, 0x1.08c19cp-55},
    {0x1.3d4p-2, 0x1.2bf9e2ab4710fp+0, -0x1.c401bap-55}, {0x1.3bcp-2, 0x1.2d307bb09eb77p+0, 0x1.83d6f2p-54},
    {0x1.3a4p-2, 0x1.2e688f587c923p+0, 0x1.21be24p-54}, {0x1.38cp-2, 0x1.2fa221427293dp+0, -0x1.fb7e5p-56},
    {0x1.374p-2, 0x1.30dd351b73957p+0, -0x1.cecc0cp-55}, {0x1.35cp-2, 0x1.3219ce9e15856p+0, 0x1.e9b21ep-54},
    {0x1.348p-2, 0x1.3322d043421a1p+0, -0x1.11dce8p-54}, {0x1.33p-2, 0x1.34623e05232fbp+0, -0x1.8ef4cep-54},
    {0x1.318p-2, 0x1.35a33c4db4495p+0, -0x1.41618cp-57}, {0x1.3p-2, 0x1.36e5cf0e54775p+0, -0x1.0e55p-54},
    {0x1.2ecp-2, 0x1.37f3d68991729p+0, 0x1.eeb95p-54}, {0x1.2d4p-2, 0x1.3939594071c6fp+0, -0x1.1440fp-55},
    {0x1.2cp-2, 0x1.3a49d9160ca4bp+0, 0x1.a1fb06p-54}, {0x1.2a8p-2, 0x1.3b9259954058p+0, 0x1.da6d1cp-54},
    {0x1.294p-2, 0x1.3ca55d72406c2p+0, 0x1.bac1a6p-54}, {0x1.27cp-2, 0x1.3df0e9ee4dp+0, -0x1.b63eb8p-57},
    {0x1.268p-2, 0x1.3f067dd348197p+0, -0x1.00a43p-55}, {0x1.254p-2, 0x1.401d3ff97f1bdp+0, -0x1.af1084p-58},
    {0x1.24p-2, 0x1.413532f602824p+0, 0x1.14c9c8p-57}, {0x1.22cp-2, 0x1.424e596664d17p+0, 0x1.83d838p-54},
    {0x1.214p-2, 0x1.43a1544c0172p+0, 0x1.83b1aap-54}, {0x1.2p-2, 0x1.44bd288178ac1p+0, -0x1.492b6p-55},
    {0x1.1ecp-2, 0x1.45da38c45756dp+0, -0x1.086c54p-56}, {0x1.1d8p-2, 0x1.46f887d78f379p+0, -0x1.2fb55ap-56},
    {0x1.1c4p-2, 0x1.48181887606c4p+0, 0x1.c65908p-54}, {0x1.1bp-2, 0x1.4938eda9836b4p+0, 0x1.9ee9cp-54},
    {0x1.1ap-2, 0x1.4a20ea197203dp+0, 0x1.30f38ap-55}, {0x1.18cp-2, 0x1.4b440e803f00ep+0, 0x1.0af244p-56},
    {0x1.178p-2, 0x1.4c687f7d34ddfp+0, 0x1.f14e1ep-54}, {0x1.164p-2, 0x1.4d8e400b984e4p+0, -0x1.3ff8cp-56},
    {0x1.15p-2, 0x1.4eb55330fd58p+0, 0x1.8dec94p-55}, {0x1.14p-2, 0x1.4fa2585987cd2p+0, 0x1.627d22p-55},
    {0x1.12cp-2, 0x1.50cbd4b42dfd2p+0, 0x1.38632ep-54}, {0x1.11cp-2, 0x1.51bacbaba0bc4p+0, 0x1.c4c238p-54},
    {0x1.108p-2, 0x1.52e6bb66d5d57p+0, 0x1.bbf296p-56}, {0x1.0f4p-2, 0x1.54140c29b1d5dp+0, -0x1.83114ep-54},
    {0x1.0e4p-2, 0x1.550619f18124ep+0, 0x1.ee4e06p-54}, {0x1.0d4p-2, 0x1.55f90d70a3cdbp+0, 0x1.b1d00cp-54},
    {0x1.0cp-2, 0x1.572a03748a307p+0, 0x1.4d1e54p-54}, {0x1.0bp-2, 0x1.581f0217bf2c9p+0, -0x1.bba86p-54},
    {0x1.09cp-2, 0x1.59528b8c2393ap+0, 0x1.fa72dcp-54}, {0x1.08cp-2, 0x1.5a499e3376e6p+0, -0x1.7ddf9cp-54},
    {0x1.07cp-2, 0x1.5b41a036e067dp+0, -0x1.ead352p-54}, {0x1.06cp-2, 0x1.5c3a9367e9919p+0, -0x1.c7869ap-54},
    {0x1.058p-2, 0x1.5d73195b356a1p+0, 0x1.32a47ep-56}, {0x1.048p-2, 0x1.5e6e31f4bbe4p+0, -0x1.9672cep-54},
    {0x1.038p-2, 0x1.5f6a41ca1517fp+0, -0x1.88248ap-54}, {0x1.028p-2, 0x1.60674ac3feeap+0, -0x1.f1db28p-54},
    {0x1.018p-2, 0x1.61654ed0e61c1p+0, -0x1.78b924p-54}, {0x1.008p-2, 0x1.62644fe4fcf2bp+0, -0x1.093b5cp-58},
    {0x1p-2, 0x1.62e42fefa39efp+0, 0x1.abc9e4p-55},
};

SDCA_EL_HD uint64_t el_bits(double v)
{
    uint64_t b;
    memcpy(&b, &v, sizeof(b));
    return b;
}

SDCA_EL_HD double el_double(uint64_t b)
{
    double v;
    memcpy(&v, &b, sizeof(v));
    return v;
}

// e^x for x <= 0; below -700 e^-700 (1e-304), NaN for NaN
SDCA_EL_HD double exp64(double x, const ExpTab *tab)
{
    const uint32_t xh = (uint32_t)(el_bits(x) >> 32);
    if (xh >= 0xC085E000u && xh <= 0xFFF00000u) x = -700.0;
    // x = k ln2 / 128 + r, |r| <= ln2 / 256; k in the low word of t
    const double magic = 6755399441055744.0;   // 1.5 * 2^52
    const double t = fma(x, 0x1.71547652b82fep+7, magic);
    const int32_t k = (int32_t)(uint32_t)el_bits(t);
    const double kd = t - magic;
    const ExpTab T = tab[k & (EXP_N - 1)];
    double r = fma(kd, -0x1.62e42feep-8, x);
    r = r + fma(kd, -0x1.a39ef35793c76p-40, T.rel);
    const double q = fma(r, fma(r, fma(r, 1.0 / 120, 1.0 / 24), 1.0 / 6), 0.5);
    const double p = fma(r * r, q, r);
    const double s = el_double(el_bits(T.t) + ((uint64_t)(int64_t)(k >> 7) << 52));
    return fma(s, p, s);
}

// log z for 1 <= z <= 4 (NaN for NaN)
SDCA_EL_HD double log64(double z, const LogTab *tab)
{
    uint32_t i = (uint32_t)(el_bits(z) >> 45) - (0x3FF00000u >> 13);
    if (i >= (uint32_t)LOG_N) i = LOG_N - 1;   // (not a number)
    const LogTab T = tab[i];
    const double r = fma(z, T.rc, -1.0);
    double q = fma(r, -1.0 / 8, 1.0 / 7);
    q = fma(r, -q, 1.0 / 6);
    q = fma(r, -q, 1.0 / 5);
    q = fma(r, -q, 1.0 / 4);
    q = fma(r, -q, 1.0 / 3);
    q = fma(r, -q, 0.5);
    return (fma(r * r, -q, T.lo) + r) + T.hi;
}

// 1 / z for 1 <= z <= 4: a single-precision start and one step of third order
SDCA_EL_HD double rcp64(double z)
{
    // z cut to 24 bits and y widened by their bits (conversions are FP64 work too)
    const uint64_t b = el_bits(z);
    uint32_t fb = (uint32_t)(b >> 29) - 0xC0000000u;   // 1023 - 127 exponents: 896 << 23, mod 2^32
    fb = (fb & 0x7fffffffu);
    float zf;
    memcpy(&zf, &fb, sizeof(zf));
#ifdef __CUDA_ARCH__
    const float yf = __frcp_rn(zf);
#else
    const float yf = 1.0f / zf;
#endif
    uint32_t yb;
    memcpy(&yb, &yf, sizeof(yb));
    const double y = el_double(((uint64_t)yb << 29) + ((uint64_t)896 << 52));
    const double e = fma(-z, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

} // namespace sdca
