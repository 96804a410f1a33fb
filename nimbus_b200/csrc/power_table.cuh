// x^y for the two powers of the model in FP64: gamma = c_p / (c_p - R_d) of the
// equation of state and kappa = R_d / c_p of the Exner function.
//
// With y fixed no logarithm is needed: x = 2^e m, m in [1, 2), r = m a - 1 with
// a the inverse of the middle of m's 64th of the interval, and
//   x^y = 2^(e y) a^-y (1 + r)^y,  |r| <= 2^-7,
// the first two factors from tables of hi and lo parts and the third by seven
// terms of the binomial series (table-driven evaluation after Tang, ACM TOMS 16,
// 1990).  14 FP64 operations for the general power's hundred, and an error of
// at most 0.51 ulp against 60 digits over 2^-12 .. 2^12 (the general power: up
// to 2 ulp by its specification).  Continuity and EOS of 3.0 million cells, four
// steps 1.93 -> 1.50 ms, Kessler and EOS 0.68 -> 0.57.  Outside that range, zeros, negative and
// non-finite values among them, and for another gamma, the general power.
#pragma once

#include "stencil_common.cuh"

namespace nimbus
{

constexpr double kGammaDry = kCpd / (kCpd - kRd), kKappaDry = kRd / kCpd;

constexpr int kPowerLowest = -12;  // the smallest exponent of the scales

static __device__ const double kPowerInverse[64] = {
    0.9921875, 0.97705078125, 0.96240234375, 0.9482421875, 0.934326171875, 0.9208984375,
    0.90771484375, 0.89501953125, 0.8828125, 0.870849609375, 0.859130859375, 0.84765625,
    0.836669921875, 0.825927734375, 0.815185546875, 0.804931640625, 0.794921875, 0.78515625,
    0.77587890625, 0.766357421875, 0.75732421875, 0.74853515625, 0.739990234375, 0.7314453125,
    0.72314453125, 0.715087890625, 0.707275390625, 0.699462890625, 0.69189453125, 0.6845703125,
    0.67724609375, 0.670166015625, 0.663330078125, 0.656494140625, 0.649658203125, 0.643310546875,
    0.63671875, 0.630615234375, 0.62451171875, 0.618408203125, 0.612548828125, 0.606689453125,
    0.600830078125, 0.595458984375, 0.58984375, 0.58447265625, 0.5791015625, 0.573974609375,
    0.56884765625, 0.56396484375, 0.558837890625, 0.55419921875, 0.54931640625, 0.544677734375,
    0.5400390625, 0.53564453125, 0.531005859375, 0.52685546875, 0.5224609375, 0.518310546875,
    0.51416015625, 0.510009765625, 0.505859375, 0.501953125};

static __device__ const double2 kPowerGamma[64] = {
    {0x1.02d3b99817251p+0, -0x1.7e31683acc0bep-54}, {0x1.08759267eebecp+0, 0x1.2204e38b7a637p-55},
    {0x1.0e1ce4a03935ep+0, -0x1.03cb780000bfep-54}, {0x1.13c722d1633e8p+0, -0x1.28c0d92055a16p-56},
    {0x1.198bed712d91dp+0, 0x1.f259d001967e8p-55}, {0x1.1f4fd47d90a61p+0, -0x1.67e69ce34167dp-54},
    {0x1.252c07de54db8p+0, 0x1.55ae395ca6250p-54}, {0x1.2b02f14b2fad7p+0, -0x1.436699c371455p-55},
    {0x1.30d127b0eccc1p+0, 0x1.bc45d60409dbap-58}, {0x1.36b24a932a524p+0, 0x1.e5ceca2d7d7d5p-55},
    {0x1.3ca59eab2ccf6p+0, 0x1.8d2e3ea3f153ep-54}, {0x1.42aa5377eb82ep+0, 0x1.8b9ab31d529e5p-54},
    {0x1.489d1f97a5674p+0, 0x1.00456519f45f2p-56}, {0x1.4e9d36fd91f87p+0, -0x1.1f21efb243436p-59},
    {0x1.54ce0529cffdcp+0, 0x1.241a077edd080p-55}, {0x1.5ae6449824bdap+0, -0x1.ea062bcf367e0p-54},
    {0x1.610814d2183f2p+0, -0x1.5d965056a40dap-54}, {0x1.67320429fe79bp+0, 0x1.4cd1b29b96a5dp-54},
    {0x1.6d3951286a1bep+0, -0x1.1bd535c432d69p-56}, {0x1.7397f9a1730f8p+0, -0x1.f279a80db2d92p-54},
    {0x1.79d09bc50c3cap+0, 0x1.431a1d4581817p-54}, {0x1.800a94d4b7572p+0, -0x1.e439dfab5e35ep-54},
    {0x1.8643f1daa9da5p+0, -0x1.dbc69d9c4fa31p-54}, {0x1.8caa17502e0ecp+0, 0x1.4f4b2cc12c765p-54},
    {0x1.930e0691feedap+0, -0x1.73244d1afeccfp-59}, {0x1.996d88959be43p+0, -0x1.e13ecd0e69218p-56},
    {0x1.9fc64c384357fp+0, -0x1.2c9168a43214fp-54}, {0x1.a64ab7c5dd358p+0, 0x1.822f0d048ef44p-54},
    {0x1.acc6374981616p+0, -0x1.3170c105f769ep-54}, {0x1.b33633a9a6612p+0, 0x1.eab803a5eb192p-56},
    {0x1.b9d10f0e9623cp+0, -0x1.c5d520f682ff2p-56}, {0x1.c05dce5d562ccp+0, -0x1.f3a7f8c394342p-55},
    {0x1.c6d9948ba6710p+0, -0x1.c83c00a63b580p-55}, {0x1.cd7eec9ced499p+0, 0x1.c4d5407cbf165p-55},
    {0x1.d44f541ebf42ap+0, 0x1.ef75bc7f9dcd3p-56}, {0x1.dacb0d48d9e5fp+0, -0x1.3aab89370d6c1p-54},
    {0x1.e1b0bb9d766e3p+0, 0x1.fe765c4940917p-57}, {0x1.e83b337c25330p+0, 0x1.ec22e9a56c925p-56},
    {0x1.eeed06c9a3c9bp+0, 0x1.a0e83dfbc3b66p-55}, {0x1.f5c78851337c6p+0, -0x1.c68ab1068a05ep-57},
    {0x1.fc836993385d4p+0, 0x1.2a7cff33a0152p-54}, {0x1.01b3aa7ae65dep+1, -0x1.4b835fd849bdep-53},
    {0x1.053a4f8360112p+1, 0x1.4fdbae3e66509p-53}, {0x1.08887f8ad829ep+1, 0x1.5cf72f7ba4447p-53},
    {0x1.0c10f605e2241p+1, 0x1.a76e9b19b7ff9p-54}, {0x1.0f85a7008414bp+1, -0x1.2891833cd3cdcp-55},
    {0x1.130e134ae70d5p+1, 0x1.719629e5a9e49p-54}, {0x1.16805f7121736p+1, -0x1.ed08a0070568fp-54},
    {0x1.1a05caad0aa4cp+1, 0x1.e3c45578bc9aep-53}, {0x1.1d729adc44450p+1, -0x1.18fdfd3527b86p-53},
    {0x1.211f15db8eeebp+1, 0x1.3ab34eda4b014p-53}, {0x1.248405b4e48e1p+1, 0x1.e01ba74965d2fp-53},
    {0x1.2829c0d5c83eap+1, 0x1.a6dd1c9a29b89p-53}, {0x1.2bb3708e783b4p+1, -0x1.f3a9929ce237cp-54},
    {0x1.2f4fd4b0fde0cp+1, -0x1.1b1dbcac75946p-55}, {0x1.32cd52e1e7313p+1, 0x1.6189047481061p-54},
    {0x1.368fbe484f093p+1, -0x1.d5c6a9c28ae05p-54}, {0x1.39fe1fb5f90c9p+1, 0x1.9bdacf1b1e631p-54},
    {0x1.3db2759be6744p+1, -0x1.9a3fab08df470p-53}, {0x1.4143dc08d6f55p+1, -0x1.461a9decd94e9p-55},
    {0x1.44e6fc552880bp+1, 0x1.ab38ae8ac62f1p-56}, {0x1.489c544645bc2p+1, -0x1.78ad404cf919dp-53},
    {0x1.4c64662de8e0fp+1, -0x1.0c79513c2885ep-53}, {0x1.50051a40a136cp+1, -0x1.b61fc7fca7bc3p-53}};

static __device__ const double2 kPowerKappa[64] = {
    {0x1.0093191dd1558p+0, -0x1.49b108aae85cap-56}, {0x1.01b46282b295bp+0, -0x1.c2e404e9de72ap-58},
    {0x1.02d1e1412ebeap+0, 0x1.00960517894f6p-56}, {0x1.03eb386b0886ap+0, -0x1.eb253792fcc0fp-55},
    {0x1.0505060c2a96cp+0, -0x1.ad14e736497cdp-54}, {0x1.061a1a55c9f03p+0, 0x1.f176c26cf2d80p-54},
    {0x1.072f3ed5dfcd5p+0, -0x1.a49780c41e996p-56}, {0x1.083f0f3d7145cp+0, 0x1.6bff660689310p-54},
    {0x1.094922bcc3859p+0, -0x1.1c1f138fe86cbp-54}, {0x1.0a5285408cf8bp+0, -0x1.fd0678843ffbap-54},
    {0x1.0b5b12fb2fb0ep+0, -0x1.896279576480cp-56}, {0x1.0c62a6b89e8f0p+0, -0x1.597d7a80e7effp-54},
    {0x1.0d6358f5c8c83p+0, 0x1.22a3b7e028e96p-55}, {0x1.0e6290a5ae84cp+0, -0x1.66d196cd1c56dp-54},
    {0x1.0f66164174acep+0, -0x1.0b713caa1e467p-54}, {0x1.1061f2a4659fdp+0, 0x1.5eb5e53bccd57p-56},
    {0x1.115bd2cc07d7bp+0, -0x1.9cb21833d868fp-55}, {0x1.125388d9c3996p+0, -0x1.26641fb616be9p-54},
    {0x1.13428ebd8acc6p+0, 0x1.486d475ef836bp-54}, {0x1.143bb90015f44p+0, 0x1.bfaf46a83e6f5p-54},
    {0x1.152bd14e4acfcp+0, 0x1.a933ce2b8bbd8p-54}, {0x1.1618fc075f210p+0, 0x1.72ff472c74a40p-55},
    {0x1.1703058c4bf09p+0, 0x1.4d6c40c50d11dp-55}, {0x1.17f08f58e4051p+0, 0x1.1319085575396p-55},
    {0x1.18dac0d2ca13bp+0, -0x1.bbf6e93ce14b1p-56}, {0x1.19c1634dc0211p+0, -0x1.6875446be4ceep-54},
    {0x1.1aa43f4128cf0p+0, -0x1.728a4d7fc79a0p-54}, {0x1.1b8a59ff95cbcp+0, -0x1.21d6b2aeedf8cp-54},
    {0x1.1c6c70515fe2ap+0, -0x1.802495c7d8c77p-54}, {0x1.1d4a480105a0ep+0, -0x1.c540df3de7fb0p-54},
    {0x1.1e2b326b3dcd8p+0, -0x1.3ec6803413737p-56}, {0x1.1f079bc98adabp+0, -0x1.61ec083452d47p-55},
    {0x1.1fdf478f6393cp+0, 0x1.a351a9de10cc7p-55}, {0x1.20b9d3dafd6ebp+0, 0x1.e46d022070bc5p-55},
    {0x1.21975252941bbp+0, 0x1.f9881212dd444p-57}, {0x1.2267b1dbfb994p+0, -0x1.85463738fa9fbp-54},
    {0x1.2342e638c21e2p+0, -0x1.8cff01f59b8abp-55}, {0x1.24107bf8942a6p+0, 0x1.504a0531a9754p-56},
    {0x1.24e0a4d3cab7bp+0, 0x1.6e55fb79f45cfp-57}, {0x1.25b36f9bcf213p+0, 0x1.d2addf4c92027p-57},
    {0x1.2680541b474d3p+0, -0x1.6b100819aae9cp-56}, {0x1.274fc1c484c3dp+0, 0x1.4ea0aab2ee109p-54},
    {0x1.2821c70359d39p+0, 0x1.b198a1f1f61acp-56}, {0x1.28e49f77972adp+0, -0x1.f5cc9519bd90cp-55},
    {0x1.29b2c19c1df44p+0, -0x1.1fb381f9595fcp-56}, {0x1.2a7a4d62e711cp+0, -0x1.e6ba9f08bd528p-54},
    {0x1.2b4438645acafp+0, 0x1.27c72a8a9b9afp-54}, {0x1.2c073827cbef9p+0, -0x1.2d81fee1edf1fp-62},
    {0x1.2ccc789a49c5fp+0, 0x1.9710a02db0ceap-55}, {0x1.2d8a77887f75cp+0, 0x1.281f860999e26p-54},
    {0x1.2e5440a848b6bp+0, 0x1.e32c4d31fb126p-56}, {0x1.2f0ce1ec11406p+0, 0x1.e49911fbae0dcp-54},
    {0x1.2fd16390580f6p+0, -0x1.4bfc90e7d500ep-55}, {0x1.308e29634835cp+0, -0x1.f2d230f7cb6efp-56},
    {0x1.314d0356846a2p+0, 0x1.4db345630cc74p-54}, {0x1.3203c6301c857p+0, 0x1.c5db0228f5f3ep-58},
    {0x1.32c6cace8a13bp+0, -0x1.138aa1bda266fp-55}, {0x1.337725e86d655p+0, 0x1.460d2cf415986p-55},
    {0x1.3433d5e73f549p+0, -0x1.99c51c12bd6eep-56}, {0x1.34e7ec7d9fd92p+0, -0x1.22b30e0994bc1p-54},
    {0x1.359de03c72c7cp+0, -0x1.5637e7a113c85p-54}, {0x1.3655b9fd717fep+0, -0x1.bbf0a8add2982p-54},
    {0x1.370f82d73d030p+0, 0x1.740eb4dbc4a24p-54}, {0x1.37c02a9e99ed4p+0, 0x1.57b6bbfb64792p-54}};

static __constant__ double2 kPowerGammaScale[24] = {
    {0x1.2562a242b487cp-17, -0x1.dd8a8579dc018p-71}, {0x1.8332f5f16a209p-16, -0x1.d9e1bac63de3ep-70},
    {0x1.ff02d25c1db08p-15, -0x1.40eef81800119p-70}, {0x1.5134ec9035bc0p-13, -0x1.41697c1d20bd7p-67},
    {0x1.bd08721cb6c6fp-12, 0x1.65608f5f548bap-66}, {0x1.25ab46e6d185bp-10, 0x1.d1aa8fbe46b14p-64},
    {0x1.8392d51a57da7p-9, -0x1.eab08108352d4p-64}, {0x1.ff815983fb41dp-8, -0x1.3b6b40a47b1cep-65},
    {0x1.51886ae3808abp-6, 0x1.5952fa5398a90p-60}, {0x1.bd76a3283b6f9p-5, -0x1.1697875f88c99p-59},
    {0x1.25f3fd8784e2ep-3, -0x1.23823b52e5422p-57}, {0x1.83f2cc003c72dp-2, -0x1.997c6b43351e4p-56},
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.51dbfde3252a3p+1, 0x1.62f606a837007p-53},
    {0x1.bde4ef7c66458p+2, -0x1.f375ebe355e82p-52}, {0x1.263cc62942bb7p+4, -0x1.e1a409d3bc23fp-51},
    {0x1.8452daa8f896ap+5, -0x1.9f527d5f72e51p-49}, {0x1.003f62ebf6ddep+7, 0x1.5ae76d8d8736fp-47},
    {0x1.522fa5944201ap+8, -0x1.a9703b28e3a56p-48}, {0x1.be53571ff8b49p+9, 0x1.802eae4671167p-45},
    {0x1.2685a0d080460p+11, -0x1.d26efcd2bdd68p-44}, {0x1.84b3011a6e676p+12, 0x1.1fb51b5544ab1p-42},
    {0x1.007ed589c418dp+14, -0x1.70cc832683dbfp-42}, {0x1.528361fbf6bc9p+15, -0x1.e544427fdeea4p-39}};

static __constant__ double2 kPowerKappaScale[24] = {
    {0x1.7bf6ee8145b8dp-4, -0x1.e7796874a96eap-58}, {0x1.cf3a49fdaca73p-4, -0x1.efbce4ac22db0p-58},
    {0x1.1a5e4821212dap-3, -0x1.aa9b01fb3e316p-57}, {0x1.583ea7d9e23ddp-3, 0x1.04e9e8912abc5p-58},
    {0x1.a3ae313a06026p-3, 0x1.90ee4f4c925e0p-57}, {0x1.ffa58a7f2cedap-3, 0x1.eac649f68db88p-57},
    {0x1.37e2048298b7ep-2, 0x1.08dba8a84f3d2p-56}, {0x1.7c3a1bfb23898p-2, -0x1.efa0f20d960e0p-57},
    {0x1.cf8c30044885cp-2, 0x1.4673cf17b94dep-56}, {0x1.1a90345360543p-1, 0x1.f8245ca03d0a1p-55},
    {0x1.587b849f18e7fp-1, 0x1.2d29eda3b9d9dp-55}, {0x1.a3f8644594626p-1, -0x1.90ec3b6a468f8p-56},
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.3819288f00936p+0, -0x1.d109ea2179d19p-55},
    {0x1.7c7d555583c25p+0, -0x1.01aa3f318c1c1p-55}, {0x1.cfde2485ae21cp+0, -0x1.97b610935f25ep-54},
    {0x1.1ac22959288ebp+1, 0x1.2ac211492b858p-53}, {0x1.58b86c26fcb0bp+1, -0x1.9c5969d021f6ap-54},
    {0x1.a442a46f7476fp+1, -0x1.453d0cd5ddf6ap-56}, {0x1.002d42bf88584p+2, 0x1.b261c3e6b61b7p-55},
    {0x1.3850565b1f299p+2, -0x1.d13784e9684cfp-53}, {0x1.7cc09a927ff2fp+2, -0x1.4951625b13a05p-54},
    {0x1.d03027846cd70p+2, -0x1.a2bc9c83238bbp-52}, {0x1.1af4273409595p+3, -0x1.f792c1393dc25p-52}};

static __device__ __noinline__ double general_power(double x, double y) { return pow(x, y); }

__device__ __forceinline__ double table_power(double x, double y, const double2* __restrict__ inverse_power,
                                              const double2* __restrict__ scale_power, double c1, double c2, double c3,
                                              double c4, double c5, double c6, double c7)
{
    constexpr unsigned kFirst = (unsigned)(1023 + kPowerLowest) << 20;
    const unsigned high = (unsigned)__double2hiint(x), past = high - kFirst;
    if (past >= 24u << 20) return general_power(x, y);
    const int i = (int)(high >> 14) & 63;
    const double m = __hiloint2double((int)((high & 0xfffffu) | 0x3ff00000u), __double2loint(x));
    const double r = __fma_rn(m, kPowerInverse[i], -1.0);
    const double2 t = inverse_power[i], s = scale_power[past >> 20];
    double p = c7;
    p = __fma_rn(p, r, c6);
    p = __fma_rn(p, r, c5);
    p = __fma_rn(p, r, c4);
    p = __fma_rn(p, r, c3);
    p = __fma_rn(p, r, c2);
    p = __fma_rn(p, r, c1);
    p *= r;
    const double high_part = s.x * t.x;
    const double low_part = __fma_rn(s.y, t.x, __fma_rn(s.x, t.y, __fma_rn(s.x, t.x, -high_part)));
    return high_part + __fma_rn(high_part, p, low_part);
}

// x^gamma.
__device__ __forceinline__ double eos_power(double x, double gamma)
{
    if (gamma != kGammaDry) return general_power(x, gamma);
    return table_power(x, kGammaDry, kPowerGamma, kPowerGammaScale, 1.400278940027894, 0.2802510849288743,
                       -0.056024159237292384, 0.022405756749781855, -0.011649743589398432, 0.006989304557005428,
                       -0.004592693052202411);
}

// x^kappa.
__device__ __forceinline__ double exner_power(double x)
{
    return table_power(x, kKappaDry, kPowerKappa, kPowerKappaScale, 0.2858565737051793, -0.10207129648735735,
                       0.05832161396239774, -0.03957330628673651, 0.029396187080326784, -0.023096307013809207,
                       0.018853658699234978);
}

}  // namespace nimbus
