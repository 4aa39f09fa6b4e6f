// imc_math64.cuh -- the double precision functions of a transport segment,
// with few FP64 operations: GB300 issues FP64 at 1/64 of the FP32 rate (one
// warp instruction in 16 cycles per SM), so an FP64 history costs its FP64
// instructions and little else.
//
//   neglog_k53   -log(k 2^-53) of a 53-bit uniform integer k: table-driven
//                reduction after Tang (ACM TOMS 16, 1990): the mantissa m times
//                a short table reciprocal c leaves r = m c - 1, |r| <= 2^-8;
//                -log v = e ln 2 + log c - log1p(r), with ln 2 and log c split
//                in a high part on the grid 2^-42 (their sum exact) and a low part
//   expm1_neg    exp(-y) - 1 for y >= 0: y = n ln2/64 + r, 0 <= r < ln2/64 (Tang,
//                ACM TOMS 15, 1989), 2^(-n/64) from a two-double table
//   div_r        a / b with r = RN(1/b) at hand: one residual correction
//                (Markstein, IBM J. Res. Dev. 34, 1990), a / b correctly rounded
//   u53, one_minus_2u53   uniforms from their integers without a conversion
//
// Largest errors seen (tests/test_math64.py, against extended precision):
// 0.503 units in the last place for neglog_k53, 1.15 for expm1_neg; div_r
// equals the IEEE quotient.  CUDA's log, exp and expm1 are good to 1 unit each.
// Table entries are the correctly rounded values of the stated expressions,
// computed with 300-bit arithmetic; the polynomials are the Taylor series.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifndef IMC_HD
#define IMC_HD __host__ __device__ __forceinline__
#endif

namespace imc {
namespace m64 {

// one row per 1/256 of the mantissa [1, 2): c, log(c) high and low.  Mantissas
// from 1.5 up are halved, so the rows next to 1 on both sides have c = 1.
struct LogRow { double c, hi, lo, pad; };
struct ExpRow { double hi, lo; };  // 2^(-j/64)
#define IMC_LOG_ROWS \
    {0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0, 0.0}, \
    {0x1.fd00000000000p-1, -0x1.8121214580000p-8, -0x1.ad50382973f27p-46, 0.0}, \
    {0x1.fb00000000000p-1, -0x1.41929f9680000p-7, -0x1.977c755d01368p-46, 0.0}, \
    {0x1.f900000000000p-1, -0x1.c317384c80000p-7, 0x1.41f33fcefb9fep-44, 0.0}, \
    {0x1.f700000000000p-1, -0x1.228fb1fea0000p-6, -0x1.713e3284991fep-45, 0.0}, \
    {0x1.f500000000000p-1, -0x1.63d6178690000p-6, -0x1.7abf389596542p-47, 0.0}, \
    {0x1.f300000000000p-1, -0x1.a55f548c60000p-6, 0x1.de0709f2d03c9p-45, 0.0}, \
    {0x1.f100000000000p-1, -0x1.e72bf28140000p-6, 0x1.8d75149774d47p-45, 0.0}, \
    {0x1.f000000000000p-1, -0x1.0415d89e78000p-5, 0x1.dddc7f461c516p-44, 0.0}, \
    {0x1.ee00000000000p-1, -0x1.252f32f8d0000p-5, -0x1.83e9ae021b67bp-45, 0.0}, \
    {0x1.ec00000000000p-1, -0x1.466aed42e0000p-5, 0x1.c167375bdfd28p-45, 0.0}, \
    {0x1.ea00000000000p-1, -0x1.67c94f2d48000p-5, -0x1.dac20827cca0cp-44, 0.0}, \
    {0x1.e800000000000p-1, -0x1.894aa149f8000p-5, -0x1.9a19a8be97661p-44, 0.0}, \
    {0x1.e600000000000p-1, -0x1.aaef2d0fb0000p-5, -0x1.0fc1a353bb42ep-45, 0.0}, \
    {0x1.e500000000000p-1, -0x1.bbcebfc690000p-5, 0x1.7bf868c317c2ap-46, 0.0}, \
    {0x1.e300000000000p-1, -0x1.dda8adc680000p-5, 0x1.1b1ac64d9e42fp-45, 0.0}, \
    {0x1.e100000000000p-1, -0x1.ffa6911ab8000p-5, -0x1.3008c98381a8fp-45, 0.0}, \
    {0x1.df00000000000p-1, -0x1.10e45b3cb0000p-4, 0x1.7cf69284a3465p-44, 0.0}, \
    {0x1.dd00000000000p-1, -0x1.2207b5c784000p-4, -0x1.49d8cfc10c7bfp-44, 0.0}, \
    {0x1.dc00000000000p-1, -0x1.2aa04a4470000p-4, -0x1.7a48ba8b1cb41p-44, 0.0}, \
    {0x1.da00000000000p-1, -0x1.3bdf5a7d20000p-4, 0x1.19bd0ad125895p-44, 0.0}, \
    {0x1.d800000000000p-1, -0x1.4d3115d208000p-4, 0x1.53a2582f4e1efp-48, 0.0}, \
    {0x1.d700000000000p-1, -0x1.55e10050e0000p-4, -0x1.c1d740c53c72ep-47, 0.0}, \
    {0x1.d500000000000p-1, -0x1.674f089364000p-4, -0x1.a79994c9d3302p-44, 0.0}, \
    {0x1.d300000000000p-1, -0x1.78d02263d8000p-4, -0x1.69b5794b69fb7p-47, 0.0}, \
    {0x1.d200000000000p-1, -0x1.8197e2f410000p-4, 0x1.c0fe460d20041p-44, 0.0}, \
    {0x1.d000000000000p-1, -0x1.9335e5d594000p-4, -0x1.3115c3abd47dap-45, 0.0}, \
    {0x1.ce00000000000p-1, -0x1.a4e7640b1c000p-4, 0x1.e42b6b94407c8p-47, 0.0}, \
    {0x1.cd00000000000p-1, -0x1.adc77ee5b0000p-4, 0x1.573b209c31904p-44, 0.0}, \
    {0x1.cb00000000000p-1, -0x1.bf968769fc000p-4, -0x1.4218c8d824283p-45, 0.0}, \
    {0x1.c900000000000p-1, -0x1.d179788218000p-4, -0x1.36433b5efbeedp-44, 0.0}, \
    {0x1.c800000000000p-1, -0x1.da72763844000p-4, -0x1.a89401fa71733p-46, 0.0}, \
    {0x1.c600000000000p-1, -0x1.ec739830a0000p-4, -0x1.11fcba80cdd10p-44, 0.0}, \
    {0x1.c500000000000p-1, -0x1.f57bc7d900000p-4, -0x1.76a6c9ea8b04ep-46, 0.0}, \
    {0x1.c300000000000p-1, -0x1.03cdc0a51e000p-3, -0x1.81a9cf169fc5cp-44, 0.0}, \
    {0x1.c200000000000p-1, -0x1.08598b59e4000p-3, 0x1.7e5dd7009902cp-45, 0.0}, \
    {0x1.c000000000000p-1, -0x1.1178e8227e000p-3, -0x1.1ef78ce2d07f2p-45, 0.0}, \
    {0x1.bf00000000000p-1, -0x1.160c8024b2000p-3, -0x1.ec2d2a9009e3dp-45, 0.0}, \
    {0x1.bd00000000000p-1, -0x1.1f3b925f26000p-3, 0x1.5f74e9b083633p-46, 0.0}, \
    {0x1.bc00000000000p-1, -0x1.23d712a49c000p-3, -0x1.00d238fd3df5cp-46, 0.0}, \
    {0x1.ba00000000000p-1, -0x1.2d1610c868000p-3, -0x1.39d6ccb81b4a1p-47, 0.0}, \
    {0x1.b900000000000p-1, -0x1.31b994d3a4000p-3, -0x1.f098ee3a50810p-44, 0.0}, \
    {0x1.b700000000000p-1, -0x1.3b08b67580000p-3, 0x1.aade8f29320fbp-44, 0.0}, \
    {0x1.b600000000000p-1, -0x1.3fb45a5992000p-3, -0x1.19713c0cae559p-44, 0.0}, \
    {0x1.b400000000000p-1, -0x1.4913d8333c000p-3, 0x1.53e43558124c4p-44, 0.0}, \
    {0x1.b300000000000p-1, -0x1.4dc7b897bc000p-3, -0x1.c79b60ae1ff0fp-47, 0.0}, \
    {0x1.b100000000000p-1, -0x1.5737cc9018000p-3, -0x1.9baa7a6b887f6p-44, 0.0}, \
    {0x1.b000000000000p-1, -0x1.5bf406b544000p-3, 0x1.27023eb68981cp-46, 0.0}, \
    {0x1.ae00000000000p-1, -0x1.6574ebe8c2000p-3, 0x1.98c1d34f0f462p-44, 0.0}, \
    {0x1.ad00000000000p-1, -0x1.6a399dabbe000p-3, 0x1.8f934e66a15a6p-44, 0.0}, \
    {0x1.ac00000000000p-1, -0x1.6f0128b756000p-3, -0x1.577390d31ef0fp-44, 0.0}, \
    {0x1.aa00000000000p-1, -0x1.7898d85444000p-3, -0x1.8e67be3dbaf3fp-44, 0.0}, \
    {0x1.a900000000000p-1, -0x1.7d6903caf6000p-3, 0x1.4c06b17c301d7p-45, 0.0}, \
    {0x1.a700000000000p-1, -0x1.871213750e000p-3, -0x1.328eb42f9af75p-44, 0.0}, \
    {0x1.a600000000000p-1, -0x1.8beafeb390000p-3, 0x1.73d54aae92cd1p-47, 0.0}, \
    {0x1.a500000000000p-1, -0x1.90c6db9fcc000p-3, 0x1.935f57718d7cap-46, 0.0}, \
    {0x1.a300000000000p-1, -0x1.9a8778deba000p-3, -0x1.470fa3efec390p-44, 0.0}, \
    {0x1.a200000000000p-1, -0x1.9f6c40708a000p-3, 0x1.337d94bcd3f43p-44, 0.0}, \
    {0x1.a100000000000p-1, -0x1.a454082e6a000p-3, -0x1.60a77c81f7171p-44, 0.0}, \
    {0x1.9f00000000000p-1, -0x1.ae2ca6f672000p-3, -0x1.7a8d5ae54f550p-44, 0.0}, \
    {0x1.9e00000000000p-1, -0x1.b31d8575bc000p-3, -0x1.c794e562a63cbp-44, 0.0}, \
    {0x1.9d00000000000p-1, -0x1.b811730b82000p-3, -0x1.e90683b9cd768p-46, 0.0}, \
    {0x1.9c00000000000p-1, -0x1.bd087383be000p-3, 0x1.d4bc4595412b6p-45, 0.0}, \
    {0x1.9a00000000000p-1, -0x1.c6ffbc6f00000p-3, -0x1.ee138d3a69d43p-44, 0.0}, \
    {0x1.9900000000000p-1, -0x1.cc000c9db4000p-3, 0x1.d6d585d57aff9p-46, 0.0}, \
    {0x1.9800000000000p-1, -0x1.d1037f2656000p-3, 0x1.84a7e75b6f6e4p-47, 0.0}, \
    {0x1.9600000000000p-1, -0x1.db13db0d48000p-3, -0x1.2806a847527e6p-44, 0.0}, \
    {0x1.9500000000000p-1, -0x1.e020cc6236000p-3, 0x1.52b00adb91424p-45, 0.0}, \
    {0x1.9400000000000p-1, -0x1.e530effe72000p-3, 0x1.fdbdbb13f7c18p-44, 0.0}, \
    {0x1.9300000000000p-1, -0x1.ea4449f04a000p-3, -0x1.5e91663732a36p-44, 0.0}, \
    {0x1.9100000000000p-1, -0x1.f474b134e0000p-3, 0x1.bae49f1df7b5ep-44, 0.0}, \
    {0x1.9000000000000p-1, -0x1.f991c6cb3c000p-3, 0x1.90d04cd7cc834p-44, 0.0}, \
    {0x1.8f00000000000p-1, -0x1.feb2233ea0000p-3, -0x1.f3418de00938bp-45, 0.0}, \
    {0x1.8e00000000000p-1, -0x1.01eae5626c000p-2, -0x1.a43dcfade85aep-44, 0.0}, \
    {0x1.8d00000000000p-1, -0x1.047e60cde8000p-2, -0x1.dbdf10d397f3cp-45, 0.0}, \
    {0x1.8b00000000000p-1, -0x1.09aa572e6c000p-2, -0x1.b50a1e1734342p-44, 0.0}, \
    {0x1.8a00000000000p-1, -0x1.0c42d67616000p-2, -0x1.7188b163ceae9p-45, 0.0}, \
    {0x1.8900000000000p-1, -0x1.0edd060b78000p-2, -0x1.019b52d8435f5p-47, 0.0}, \
    {0x1.8800000000000p-1, -0x1.1178e8227e000p-2, -0x1.1ef78ce2d07f2p-44, 0.0}, \
    {0x1.8700000000000p-1, -0x1.14167ef367000p-2, -0x1.e0c07824daaf5p-44, 0.0}, \
    {0x1.8600000000000p-1, -0x1.16b5ccbad0000p-2, 0x1.23299042d74bfp-44, 0.0}, \
    {0x1.8400000000000p-1, -0x1.1bf99635a7000p-2, 0x1.1ac89575c2125p-44, 0.0}, \
    {0x1.8300000000000p-1, -0x1.1e9e16788a000p-2, 0x1.82eaed3c8b65ep-44, 0.0}, \
    {0x1.8200000000000p-1, -0x1.214456d0ec000p-2, 0x1.caf0428b728a3p-44, 0.0}, \
    {0x1.8100000000000p-1, -0x1.23ec5991ec000p-2, 0x1.6dbe448a2e522p-44, 0.0}, \
    {0x1.8000000000000p-1, -0x1.269621134e000p-2, 0x1.1b61f10522625p-44, 0.0}, \
    {0x1.7f00000000000p-1, -0x1.2941afb187000p-2, 0x1.210c2b730e28bp-44, 0.0}, \
    {0x1.7e00000000000p-1, -0x1.2bef07cdc9000p-2, -0x1.a9cfa4a5004f4p-45, 0.0}, \
    {0x1.7c00000000000p-1, -0x1.314f1e1d36000p-2, 0x1.8e27ad3213cb8p-45, 0.0}, \
    {0x1.7b00000000000p-1, -0x1.3401e12aed000p-2, 0x1.17c73556e291dp-44, 0.0}, \
    {0x1.7a00000000000p-1, -0x1.36b6776be1000p-2, -0x1.16ecdb0f177c8p-46, 0.0}, \
    {0x1.7900000000000p-1, -0x1.396ce359bc000p-2, 0x1.5839c5663663dp-47, 0.0}, \
    {0x1.7800000000000p-1, -0x1.3c25277333000p-2, -0x1.83b54b606bd5cp-46, 0.0}, \
    {0x1.7700000000000p-1, -0x1.3edf463c17000p-2, 0x1.f067c297f2c3fp-44, 0.0}, \
    {0x1.7600000000000p-1, -0x1.419b423d5f000p-2, 0x1.ce379226de3ecp-44, 0.0}, \
    {0x1.7500000000000p-1, -0x1.44591e053a000p-2, 0x1.6e95892923d88p-47, 0.0}, \
    {0x1.7400000000000p-1, -0x1.4718dc271c000p-2, -0x1.06c18fb4c14c5p-44, 0.0}, \
    {0x1.7300000000000p-1, -0x1.49da7f3bcc000p-2, -0x1.07b334daf4b9ap-44, 0.0}, \
    {0x1.7200000000000p-1, -0x1.4c9e09e173000p-2, 0x1.e20891b0ad8a4p-45, 0.0}, \
    {0x1.7100000000000p-1, -0x1.4f637ebbaa000p-2, 0x1.fc158cb3124b9p-44, 0.0}, \
    {0x1.7000000000000p-1, -0x1.522ae0738a000p-2, -0x1.ebe708164c759p-45, 0.0}, \
    {0x1.6f00000000000p-1, -0x1.54f431b7be000p-2, -0x1.a8954c0910952p-46, 0.0}, \
    {0x1.6e00000000000p-1, -0x1.57bf753c8d000p-2, -0x1.fadedee5d40efp-46, 0.0}, \
    {0x1.6d00000000000p-1, -0x1.5a8cadbbee000p-2, 0x1.7c79b0af7ecf8p-48, 0.0}, \
    {0x1.6c00000000000p-1, -0x1.5d5bddf596000p-2, 0x1.a0b2a08a465dcp-47, 0.0}, \
    {0x1.6b00000000000p-1, -0x1.602d08af09000p-2, -0x1.ebe9176df3f65p-46, 0.0}, \
    {0x1.6a00000000000p-1, -0x1.630030b3ab000p-2, 0x1.db623e731ae00p-45, 0.0}, \
    {0x1.6900000000000p-1, -0x1.65d558d4ce000p-2, -0x1.544fd2dc5bdc0p-51, 0.0}, \
    {0x1.6800000000000p-1, -0x1.68ac83e9c7000p-2, 0x1.7af966c548a30p-44, 0.0}, \
    {0x1.6700000000000p-1, -0x1.6b85b4cffa000p-2, -0x1.fe6750d372503p-45, 0.0}, \
    {0x1.6600000000000p-1, -0x1.6e60ee6af2000p-2, 0x1.a37a6a0f7749ep-44, 0.0}, \
    {0x1.6500000000000p-1, -0x1.713e33a46a000p-2, -0x1.7b9b2617e9472p-46, 0.0}, \
    {0x1.6400000000000p-1, -0x1.741d876c68000p-2, 0x1.13a7b5b11cfa7p-44, 0.0}, \
    {0x1.6300000000000p-1, -0x1.76feecb947000p-2, -0x1.74bb9c9852c57p-46, 0.0}, \
    {0x1.6200000000000p-1, -0x1.79e26687d0000p-2, 0x1.309c168817444p-44, 0.0}, \
    {0x1.6100000000000p-1, -0x1.7cc7f7db47000p-2, 0x1.7c98438023cdcp-44, 0.0}, \
    {0x1.6000000000000p-1, -0x1.7fafa3bd81000p-2, -0x1.46fb79bf6d4cbp-44, 0.0}, \
    {0x1.5f00000000000p-1, -0x1.82996d3ef9000p-2, 0x1.0d52aa30536bbp-44, 0.0}, \
    {0x1.5e00000000000p-1, -0x1.85855776dd000p-2, 0x1.015486666443bp-44, 0.0}, \
    {0x1.5d00000000000p-1, -0x1.8873658328000p-2, 0x1.988e21f7fc497p-45, 0.0}, \
    {0x1.5c00000000000p-1, -0x1.8b639a88b3000p-2, 0x1.05ae1e5e70470p-45, 0.0}, \
    {0x1.5b00000000000p-1, -0x1.8e55f9b34a000p-2, 0x1.1f21d89c89c45p-44, 0.0}, \
    {0x1.5a00000000000p-1, -0x1.914a8635bf000p-2, -0x1.a2652b44673e1p-44, 0.0}, \
    {0x1.5900000000000p-1, -0x1.9441434a03000p-2, -0x1.2cb81c95fff43p-45, 0.0}, \
    {0x1.5800000000000p-1, -0x1.973a343135000p-2, -0x1.ab73b16bf4984p-44, 0.0}, \
    {0x1.5800000000000p-1, -0x1.973a343135000p-2, -0x1.ab73b16bf4984p-44, 0.0}, \
    {0x1.5700000000000p-1, -0x1.9a355c33bd000p-2, -0x1.ae73535438bebp-44, 0.0}, \
    {0x1.5600000000000p-1, -0x1.9d32bea15f000p-2, 0x1.6279e10d0c0b0p-45, 0.0}, \
    {0x1.5500000000000p+0, 0x1.2596010df7000p-2, 0x1.8e7bc224ea3e3p-44, 0.0}, \
    {0x1.5400000000000p+0, 0x1.22941fbcf8000p-2, -0x1.a6976f5eb0963p-44, 0.0}, \
    {0x1.5300000000000p+0, 0x1.1f8ff9e48a000p-2, 0x1.7946c040cbe77p-45, 0.0}, \
    {0x1.5280000000000p+0, 0x1.1e0d0c3371000p-2, 0x1.af8f2a9b0d4a0p-44, 0.0}, \
    {0x1.5180000000000p+0, 0x1.1b05791f08000p-2, -0x1.2dd466dc55e2dp-44, 0.0}, \
    {0x1.5080000000000p+0, 0x1.17fb98e151000p-2, -0x1.a8a8ba74a2684p-44, 0.0}, \
    {0x1.4f80000000000p+0, 0x1.14ef67f887000p-2, -0x1.e97a65dfc9794p-44, 0.0}, \
    {0x1.4f00000000000p+0, 0x1.136870293b000p-2, -0x1.d3e8499d67123p-44, 0.0}, \
    {0x1.4e00000000000p+0, 0x1.1058bf9ae5000p-2, -0x1.4ab9d817d52cdp-44, 0.0}, \
    {0x1.4d00000000000p+0, 0x1.0d46b579ab000p-2, 0x1.d2c81f640e1e6p-44, 0.0}, \
    {0x1.4c00000000000p+0, 0x1.0a324e2739000p-2, 0x1.c6bee7ef4030ep-47, 0.0}, \
    {0x1.4b80000000000p+0, 0x1.08a73667c5000p-2, 0x1.ebc1d40c5a329p-44, 0.0}, \
    {0x1.4a80000000000p+0, 0x1.058f3c703f000p-2, -0x1.0e866bcd236adp-44, 0.0}, \
    {0x1.4980000000000p+0, 0x1.0274dc16c2000p-2, 0x1.979e89cf835c2p-45, 0.0}, \
    {0x1.4900000000000p+0, 0x1.00e6c45ad5000p-2, 0x1.cc68d52e01203p-50, 0.0}, \
    {0x1.4800000000000p+0, 0x1.fb9186d5e4000p-3, -0x1.d572aab993c87p-47, 0.0}, \
    {0x1.4780000000000p+0, 0x1.f871b28956000p-3, -0x1.f75fd6a526efep-44, 0.0}, \
    {0x1.4680000000000p+0, 0x1.f22e5e72f2000p-3, -0x1.f454f1417e41fp-44, 0.0}, \
    {0x1.4580000000000p+0, 0x1.ebe61f4dd8000p-3, -0x1.3d45330fdca4dp-45, 0.0}, \
    {0x1.4500000000000p+0, 0x1.e8c0252aa6000p-3, -0x1.6805b80e8e6ffp-45, 0.0}, \
    {0x1.4400000000000p+0, 0x1.e27076e2b0000p-3, -0x1.a342c2af0003cp-44, 0.0}, \
    {0x1.4300000000000p+0, 0x1.dc1bca0abe000p-3, 0x1.8fac1a628ccc6p-44, 0.0}, \
    {0x1.4280000000000p+0, 0x1.d8ef91af32000p-3, -0x1.5105fc364c784p-46, 0.0}, \
    {0x1.4180000000000p+0, 0x1.d293581b6c000p-3, -0x1.83270128aaa5fp-44, 0.0}, \
    {0x1.4100000000000p+0, 0x1.cf6354e09c000p-3, 0x1.771239a07d55bp-45, 0.0}, \
    {0x1.4000000000000p+0, 0x1.c8ff7c79aa000p-3, -0x1.7794f689f8434p-45, 0.0}, \
    {0x1.3f80000000000p+0, 0x1.c5cba543ae000p-3, 0x1.0929decb454fcp-45, 0.0}, \
    {0x1.3e80000000000p+0, 0x1.bf601bb0e4000p-3, 0x1.386a947c378b5p-45, 0.0}, \
    {0x1.3e00000000000p+0, 0x1.bc286742d8000p-3, 0x1.9ac53f39d121cp-44, 0.0}, \
    {0x1.3d00000000000p+0, 0x1.b5b519e8fc000p-3, -0x1.4b722ec011f31p-44, 0.0}, \
    {0x1.3c00000000000p+0, 0x1.af3c94e80c000p-3, -0x1.a4e633fcd9066p-52, 0.0}, \
    {0x1.3b80000000000p+0, 0x1.abfe5ae462000p-3, -0x1.b68f5395f139dp-44, 0.0}, \
    {0x1.3a80000000000p+0, 0x1.a57df28244000p-3, 0x1.b99c8ca1d9abbp-44, 0.0}, \
    {0x1.3a00000000000p+0, 0x1.a23bc1fe2c000p-3, -0x1.539cd91dc9f0bp-44, 0.0}, \
    {0x1.3900000000000p+0, 0x1.9bb362e7e0000p-3, -0x1.1f2a8a1ce0ffcp-45, 0.0}, \
    {0x1.3880000000000p+0, 0x1.986d322818000p-3, 0x1.93b564dd44000p-48, 0.0}, \
    {0x1.3780000000000p+0, 0x1.91dcc8c340000p-3, 0x1.7bc6abddeff46p-44, 0.0}, \
    {0x1.3700000000000p+0, 0x1.8e928de886000p-3, 0x1.a8154b13d72d5p-44, 0.0}, \
    {0x1.3600000000000p+0, 0x1.87fa06520c000p-3, 0x1.22120401202fcp-44, 0.0}, \
    {0x1.3580000000000p+0, 0x1.84abb75866000p-3, -0x1.d8daadf4e2bd2p-44, 0.0}, \
    {0x1.3500000000000p+0, 0x1.815c0a1436000p-3, -0x1.02a52f9201ce8p-44, 0.0}, \
    {0x1.3400000000000p+0, 0x1.7ab890210e000p-3, -0x1.bdb9072534a58p-45, 0.0}, \
    {0x1.3380000000000p+0, 0x1.7764c128f2000p-3, 0x1.274903479e3d1p-47, 0.0}, \
    {0x1.3280000000000p+0, 0x1.70b8f97a1a000p-3, 0x1.4ea64f6a95befp-44, 0.0}, \
    {0x1.3200000000000p+0, 0x1.6d60fe719e000p-3, -0x1.bc6e557134767p-44, 0.0}, \
    {0x1.3100000000000p+0, 0x1.66acd4272a000p-3, 0x1.aa1bdbfc6c785p-44, 0.0}, \
    {0x1.3080000000000p+0, 0x1.6350a28aaa000p-3, 0x1.d5ec0ab8163afp-45, 0.0}, \
    {0x1.3000000000000p+0, 0x1.5ff3070a7a000p-3, -0x1.8586f183bebf2p-44, 0.0}, \
    {0x1.2f00000000000p+0, 0x1.59338d9982000p-3, 0x1.0ba68b7555d4ap-48, 0.0}, \
    {0x1.2e80000000000p+0, 0x1.55d1ad4232000p-3, 0x1.add94dda647e8p-44, 0.0}, \
    {0x1.2d80000000000p+0, 0x1.4f099f4a24000p-3, -0x1.e9bf2fafeaf27p-44, 0.0}, \
    {0x1.2d00000000000p+0, 0x1.4ba36f39a6000p-3, -0x1.4354bb3f219e5p-44, 0.0}, \
    {0x1.2c80000000000p+0, 0x1.483bccce6e000p-3, 0x1.eea52723f6369p-46, 0.0}, \
    {0x1.2b80000000000p+0, 0x1.41682bf728000p-3, -0x1.10047081f849dp-45, 0.0}, \
    {0x1.2b00000000000p+0, 0x1.3dfc2b0ecc000p-3, 0x1.8a72a62b8c13fp-45, 0.0}, \
    {0x1.2a00000000000p+0, 0x1.371fc201e8000p-3, 0x1.ee8779b2d8abcp-44, 0.0}, \
    {0x1.2980000000000p+0, 0x1.33af575770000p-3, 0x1.c9ecca2fe72a5p-44, 0.0}, \
    {0x1.2900000000000p+0, 0x1.303d718e48000p-3, -0x1.680b5ce3ecb05p-50, 0.0}, \
    {0x1.2800000000000p+0, 0x1.29552f8200000p-3, -0x1.5b967f4471dfcp-44, 0.0}, \
    {0x1.2780000000000p+0, 0x1.25ded0abc6000p-3, 0x1.5a3854f176449p-44, 0.0}, \
    {0x1.2700000000000p+0, 0x1.2266f190a6000p-3, -0x1.4d20ab840e7f6p-45, 0.0}, \
    {0x1.2600000000000p+0, 0x1.1b72ad52f6000p-3, 0x1.e80a41811a396p-45, 0.0}, \
    {0x1.2580000000000p+0, 0x1.17f6458fca000p-3, 0x1.843fad093c8dcp-45, 0.0}, \
    {0x1.2500000000000p+0, 0x1.1478584674000p-3, 0x1.563451027c750p-46, 0.0}, \
    {0x1.2400000000000p+0, 0x1.0d77e7cd08000p-3, 0x1.cb2cd2ee2f482p-44, 0.0}, \
    {0x1.2380000000000p+0, 0x1.09f561ee72000p-3, -0x1.8f3057157d1a8p-45, 0.0}, \
    {0x1.2300000000000p+0, 0x1.0671512ca6000p-3, -0x1.a47579cdc0a3dp-45, 0.0}, \
    {0x1.2280000000000p+0, 0x1.02ebb42bf4000p-3, -0x1.5a8fa5ce00e5dp-46, 0.0}, \
    {0x1.2180000000000p+0, 0x1.f7b79fec38000p-4, -0x1.10987e897ed01p-47, 0.0}, \
    {0x1.2100000000000p+0, 0x1.f0a30c0118000p-4, -0x1.d599e83368e91p-44, 0.0}, \
    {0x1.2080000000000p+0, 0x1.e98b549670000p-4, 0x1.4677489c50e97p-44, 0.0}, \
    {0x1.2000000000000p+0, 0x1.e27076e2b0000p-4, -0x1.a342c2af0003cp-45, 0.0}, \
    {0x1.1f00000000000p+0, 0x1.d4313d66cc000p-4, -0x1.9454379135713p-45, 0.0}, \
    {0x1.1e80000000000p+0, 0x1.cd0cdbf8c0000p-4, 0x1.3e14db50dd743p-44, 0.0}, \
    {0x1.1e00000000000p+0, 0x1.c5e548f5bc000p-4, 0x1.d0c57585fbe06p-46, 0.0}, \
    {0x1.1d00000000000p+0, 0x1.b78c82bb10000p-4, -0x1.25ef7bc3987e7p-44, 0.0}, \
    {0x1.1c80000000000p+0, 0x1.b05b49bee4000p-4, 0x1.ff22c18f84a5ep-47, 0.0}, \
    {0x1.1c00000000000p+0, 0x1.a926d3a4ac000p-4, 0x1.563650bd22a9cp-44, 0.0}, \
    {0x1.1b80000000000p+0, 0x1.a1ef1d8060000p-4, 0x1.cd4176df97bcbp-44, 0.0}, \
    {0x1.1b00000000000p+0, 0x1.9ab4246204000p-4, -0x1.8a64826787061p-45, 0.0}, \
    {0x1.1a00000000000p+0, 0x1.8c345d6318000p-4, 0x1.b20f5acb42a66p-44, 0.0}, \
    {0x1.1980000000000p+0, 0x1.84ef898e84000p-4, -0x1.7d5cd246977c9p-44, 0.0}, \
    {0x1.1900000000000p+0, 0x1.7da766d7b0000p-4, 0x1.2cc844480c89bp-44, 0.0}, \
    {0x1.1880000000000p+0, 0x1.765bf23a6c000p-4, -0x1.ecbc035c4256ap-48, 0.0}, \
    {0x1.1800000000000p+0, 0x1.6f0d28ae58000p-4, -0x1.4b4641b664613p-44, 0.0}, \
    {0x1.1700000000000p+0, 0x1.60658a9374000p-4, 0x1.0c3b1dee9c4f8p-44, 0.0}, \
    {0x1.1680000000000p+0, 0x1.590cafdf00000p-4, 0x1.c284f5722abaap-44, 0.0}, \
    {0x1.1600000000000p+0, 0x1.51b073f060000p-4, 0x1.83f69278e686ap-44, 0.0}, \
    {0x1.1580000000000p+0, 0x1.4a50d3aa1c000p-4, -0x1.f7fe1308973e2p-45, 0.0}, \
    {0x1.1500000000000p+0, 0x1.42edcbea64000p-4, 0x1.bc0eeea7c9acdp-46, 0.0}, \
    {0x1.1400000000000p+0, 0x1.341d7961bc000p-4, 0x1.1d09299837610p-44, 0.0}, \
    {0x1.1380000000000p+0, 0x1.2cb0283f5c000p-4, 0x1.e1ee2ca657021p-44, 0.0}, \
    {0x1.1300000000000p+0, 0x1.253f62f0a0000p-4, 0x1.416f8fb69a701p-44, 0.0}, \
    {0x1.1280000000000p+0, 0x1.1dcb263db0000p-4, 0x1.9444f5e9e8981p-44, 0.0}, \
    {0x1.1200000000000p+0, 0x1.16536eea38000p-4, -0x1.47c5e768fa309p-46, 0.0}, \
    {0x1.1180000000000p+0, 0x1.0ed839b554000p-4, -0x1.901f46d48abb4p-44, 0.0}, \
    {0x1.1100000000000p+0, 0x1.0759835990000p-4, -0x1.b8ecfe4b59987p-44, 0.0}, \
    {0x1.1000000000000p+0, 0x1.f0a30c0118000p-5, -0x1.d599e83368e91p-45, 0.0}, \
    {0x1.0f80000000000p+0, 0x1.e19070c278000p-5, -0x1.fea4664629e86p-45, 0.0}, \
    {0x1.0f00000000000p+0, 0x1.d276b8adb0000p-5, 0x1.6a423c78a64b0p-46, 0.0}, \
    {0x1.0e80000000000p+0, 0x1.c355dd0920000p-5, 0x1.f2ccc9abf8388p-45, 0.0}, \
    {0x1.0e00000000000p+0, 0x1.b42dd71198000p-5, -0x1.c827ae5d6704cp-46, 0.0}, \
    {0x1.0d80000000000p+0, 0x1.a4fe9ffa40000p-5, -0x1.6e584a0402925p-44, 0.0}, \
    {0x1.0d00000000000p+0, 0x1.95c830ec90000p-5, -0x1.c148297c5feb8p-45, 0.0}, \
    {0x1.0c80000000000p+0, 0x1.868a830840000p-5, -0x1.2623a134ac693p-46, 0.0}, \
    {0x1.0c00000000000p+0, 0x1.77458f6330000p-5, -0x1.181dce586af09p-44, 0.0}, \
    {0x1.0b00000000000p+0, 0x1.58a5bafc90000p-5, -0x1.b2b739570ad39p-45, 0.0}, \
    {0x1.0a80000000000p+0, 0x1.494acc34d8000p-5, 0x1.11c78a56fd247p-45, 0.0}, \
    {0x1.0a00000000000p+0, 0x1.39e87b9fe8000p-5, 0x1.eafd480ad9015p-44, 0.0}, \
    {0x1.0980000000000p+0, 0x1.2a7ec22150000p-5, -0x1.78ce77a9163fep-45, 0.0}, \
    {0x1.0900000000000p+0, 0x1.1b0d989240000p-5, -0x1.3401e9ae889bbp-44, 0.0}, \
    {0x1.0880000000000p+0, 0x1.0b94f7c198000p-5, -0x1.e89896f022783p-45, 0.0}, \
    {0x1.0800000000000p+0, 0x1.f829b0e780000p-6, 0x1.980267c7e09e4p-45, 0.0}, \
    {0x1.0780000000000p+0, 0x1.d91a66c540000p-6, 0x1.e61f1658cfb9ap-45, 0.0}, \
    {0x1.0700000000000p+0, 0x1.b9fc027b00000p-6, -0x1.b9a010ae6922ap-44, 0.0}, \
    {0x1.0680000000000p+0, 0x1.9ace7551d0000p-6, -0x1.d75d97ec7c410p-45, 0.0}, \
    {0x1.0600000000000p+0, 0x1.7b91b07d60000p-6, -0x1.3b955b602ace4p-44, 0.0}, \
    {0x1.0580000000000p+0, 0x1.5c45a51b90000p-6, -0x1.63bb6216d87d8p-45, 0.0}, \
    {0x1.0500000000000p+0, 0x1.3cea443470000p-6, -0x1.6a2c432d6a40bp-44, 0.0}, \
    {0x1.0480000000000p+0, 0x1.1d7f7eb9f0000p-6, -0x1.4193a83fcc7a6p-46, 0.0}, \
    {0x1.0400000000000p+0, 0x1.fc0a8b0fc0000p-7, 0x1.f1e7cf6d3a69cp-50, 0.0}, \
    {0x1.0380000000000p+0, 0x1.bcf712c740000p-7, 0x1.c25e097bd9771p-46, 0.0}, \
    {0x1.0300000000000p+0, 0x1.7dc475f820000p-7, -0x1.eb1245b5da1f5p-44, 0.0}, \
    {0x1.0280000000000p+0, 0x1.3e7295d260000p-7, -0x1.609c1ff29a114p-45, 0.0}, \
    {0x1.0200000000000p+0, 0x1.fe02a6b100000p-8, 0x1.9e23f0dda40e4p-46, 0.0}, \
    {0x1.0180000000000p+0, 0x1.7ee11ebd80000p-8, 0x1.749d3c2d23a07p-47, 0.0}, \
    {0x1.0100000000000p+0, 0x1.ff00aa2b00000p-9, 0x1.0bc04a086b56ap-45, 0.0}, \
    {0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0, 0.0}
#define IMC_EXP_ROWS \
    {0x1.0000000000000p+0, 0x0.0p+0}, \
    {0x1.fa7c1819e90d8p-1, 0x1.74853f3a5931ep-56}, \
    {0x1.f50765b6e4540p-1, 0x1.9d3e12dd8a18bp-55}, \
    {0x1.efa1bee615a27p-1, 0x1.dc7f486a4b6b0p-55}, \
    {0x1.ea4afa2a490dap-1, -0x1.e9c23179c2893p-55}, \
    {0x1.e502ee78b3ff6p-1, 0x1.39e8980a9cc8fp-56}, \
    {0x1.dfc97337b9b5fp-1, -0x1.1a5cd4f184b5cp-55}, \
    {0x1.da9e603db3285p-1, 0x1.c2300696db532p-55}, \
    {0x1.d5818dcfba487p-1, 0x1.2ed02d75b3707p-56}, \
    {0x1.d072d4a07897cp-1, -0x1.cbc3743797a9cp-55}, \
    {0x1.cb720dcef9069p-1, 0x1.503cbd1e949dbp-57}, \
    {0x1.c67f12e57d14bp-1, 0x1.2884dff483cadp-55}, \
    {0x1.c199bdd85529cp-1, 0x1.11065895048ddp-56}, \
    {0x1.bcc1e904bc1d2p-1, 0x1.23dd07a2d9e84p-56}, \
    {0x1.b7f76f2fb5e47p-1, -0x1.5584f7e54ac3bp-57}, \
    {0x1.b33a2b84f15fbp-1, -0x1.2805e3084d708p-58}, \
    {0x1.ae89f995ad3adp-1, 0x1.7a1cd345dcc81p-55}, \
    {0x1.a9e6b5579fdbfp-1, 0x1.0fac90ef7fd31p-55}, \
    {0x1.a5503b23e255dp-1, -0x1.d2f6edb8d41e1p-55}, \
    {0x1.a0c667b5de565p-1, -0x1.359495d1cd533p-55}, \
    {0x1.9c49182a3f090p-1, 0x1.c7c46b071f2bep-57}, \
    {0x1.97d829fde4e50p-1, -0x1.d185b7c1b85d1p-55}, \
    {0x1.93737b0cdc5e5p-1, -0x1.75fc781b57ebcp-58}, \
    {0x1.8f1ae99157736p-1, 0x1.5cc13a2e3976cp-56}, \
    {0x1.8ace5422aa0dbp-1, 0x1.6e9f156864b27p-55}, \
    {0x1.868d99b4492edp-1, -0x1.fc6f89bd4f6bap-55}, \
    {0x1.82589994cce13p-1, -0x1.d4c1dd41532d8p-55}, \
    {0x1.7e2f336cf4e62p-1, 0x1.05d02ba15797ep-57}, \
    {0x1.7a11473eb0187p-1, -0x1.41577ee04992fp-56}, \
    {0x1.75feb564267c9p-1, -0x1.0245957316dd3p-55}, \
    {0x1.71f75e8ec5f74p-1, -0x1.16e4786887a99p-56}, \
    {0x1.6dfb23c651a2fp-1, -0x1.bbe3a683c88abp-58}, \
    {0x1.6a09e667f3bcdp-1, -0x1.bdd3413b26456p-55}, \
    {0x1.6623882552225p-1, -0x1.bb60987591c34p-55}, \
    {0x1.6247eb03a5585p-1, -0x1.383c17e40b497p-55}, \
    {0x1.5e76f15ad2148p-1, 0x1.ba6f93080e65ep-55}, \
    {0x1.5ab07dd485429p-1, 0x1.6324c054647adp-55}, \
    {0x1.56f4736b527dap-1, 0x1.9bb2c011d93adp-55}, \
    {0x1.5342b569d4f82p-1, -0x1.07abe1db13cadp-56}, \
    {0x1.4f9b2769d2ca7p-1, -0x1.4b309d25957e3p-55}, \
    {0x1.4bfdad5362a27p-1, 0x1.d4397afec42e2p-57}, \
    {0x1.486a2b5c13cd0p-1, 0x1.3c1a3b69062f0p-57}, \
    {0x1.44e086061892dp-1, 0x1.89b7a04ef80d0p-60}, \
    {0x1.4160a21f72e2ap-1, -0x1.ef3691c309278p-59}, \
    {0x1.3dea64c123422p-1, 0x1.ada0911f09ebcp-56}, \
    {0x1.3a7db34e59ff7p-1, -0x1.5e436d661f5e3p-57}, \
    {0x1.371a7373aa9cbp-1, -0x1.63aeabf42eae2p-55}, \
    {0x1.33c08b26416ffp-1, 0x1.32721843659a6p-55}, \
    {0x1.306fe0a31b715p-1, 0x1.6f46ad23182e4p-56}, \
    {0x1.2d285a6e4030bp-1, 0x1.0024754db41d5p-55}, \
    {0x1.29e9df51fdee1p-1, 0x1.612e8afad1255p-56}, \
    {0x1.26b4565e27cddp-1, 0x1.2bd339940e9d9p-56}, \
    {0x1.2387a6e756238p-1, 0x1.9b07eb6c70573p-55}, \
    {0x1.2063b88628cd6p-1, 0x1.dc775814a8495p-56}, \
    {0x1.1d4873168b9aap-1, 0x1.e016e00a2643cp-55}, \
    {0x1.1a35beb6fcb75p-1, 0x1.e5b4c7b4968e4p-56}, \
    {0x1.172b83c7d517bp-1, -0x1.19041b9d78a76p-56}, \
    {0x1.1429aaea92de0p-1, -0x1.32fbf9af1369ep-55}, \
    {0x1.11301d0125b51p-1, -0x1.6c51039449b3ap-55}, \
    {0x1.0e3ec32d3d1a2p-1, 0x1.03a1727c57b53p-60}, \
    {0x1.0b5586cf9890fp-1, 0x1.8a62e4adc610bp-55}, \
    {0x1.0874518759bc8p-1, 0x1.186be4bb284ffp-58}, \
    {0x1.059b0d3158574p-1, 0x1.d73e2a475b465p-56}, \
    {0x1.02c9a3e778061p-1, -0x1.19083535b085dp-57}

static const LogRow h_log_rows[256] = {IMC_LOG_ROWS};
static const ExpRow h_exp_rows[64] = {IMC_EXP_ROWS};
#ifdef __CUDACC__
static __device__ const LogRow d_log_rows[256] = {IMC_LOG_ROWS};
static __device__ const ExpRow d_exp_rows[64] = {IMC_EXP_ROWS};
#endif
#undef IMC_LOG_ROWS
#undef IMC_EXP_ROWS

constexpr double kLn2Hi = 0x1.62e42fefa3800p-1, kLn2Lo = 0x1.ef35793c76730p-45;          // ln 2: grid 2^-42, rest
constexpr double kStepInv = 0x1.71547652b82fep+6;  // 64 / ln 2
constexpr double kStepHi = 0x1.62e42fefa3800p-7, kStepLo = 0x1.ef35793c76730p-51;  // ln 2 / 64: grid 2^-48, rest
IMC_HD uint64_t bits(double v) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(v);
#else
    uint64_t u; memcpy(&u, &v, 8); return u;
#endif
}
IMC_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double v; memcpy(&v, &u, 8); return v;
#endif
}
IMC_HD uint32_t hi32(double v) { return (uint32_t)(bits(v) >> 32); }

// k 2^-53 (k < 2^53) without an integer conversion: the low 52 bits as the
// fraction of a number in [1/2, 1), whose 1/2 goes unless bit 52 is set
IMC_HD double u53(uint64_t k) {
    const double w = from_bits(0x3FE0000000000000ull | (k & 0xFFFFFFFFFFFFFull));
    return w - ((k >> 52) ? 0.0 : 0.5);
}
// 1 - 2 u53(k): exact, one subtraction
IMC_HD double one_minus_2u53(uint64_t k) {
    const double w = from_bits(0x3FF0000000000000ull | (k & 0xFFFFFFFFFFFFFull));
    return ((k >> 52) ? 1.0 : 2.0) - w;
}

// -log(k 2^-53), 0 < k < 2^53
IMC_HD double neglog_k53(uint64_t k) {
#ifdef __CUDA_ARCH__
    const int z = __clzll((long long)k);  // 11..63
#else
    const int z = __builtin_clzll(k);
#endif
    const uint64_t f = (k << (z - 11)) & 0xFFFFFFFFFFFFFull;  // fraction of the mantissa in [1, 2)
    const int row = (int)(f >> 44);
    const int up = row >> 7;  // mantissa at or above 1.5: halved
    const double m = from_bits(((uint64_t)(0x3FF - up) << 52) | f);
#ifdef __CUDA_ARCH__
    const LogRow &t = d_log_rows[row];
    const double2 t0 = __ldg(reinterpret_cast<const double2 *>(&t));
    const double tc = t0.x, thi = t0.y, tlo = __ldg(&t.lo);
    const double e = __hiloint2double(0x43300000, z - 10 - up) - 0x1p52;
#else
    const LogRow &t = h_log_rows[row];
    const double tc = t.c, thi = t.hi, tlo = t.lo;
    const double e = (double)(z - 10 - up);  // k 2^-53 = m 2^-e
#endif
    const double r = fma(m, tc, -1.0);
    const double hi = fma(e, kLn2Hi, thi);  // exact
    const double lo = fma(e, kLn2Lo, tlo);
    const double r2 = r * r;
    double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
    p = fma(r, p, 1.0 / 5.0);
    p = fma(r, p, -1.0 / 4.0);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -1.0 / 2.0);
    // hi + lo - (r + r2 p), with the rounding of hi - r kept
    const double s = hi - r;
    const double err = (hi - s) - r;
    return s + (fma(-r2, p, lo) + err);
}

// exp(-y) - 1, y >= 0 (NaN gives NaN)
IMC_HD double expm1_neg(double y) {
    // 64 and beyond is -1 to the last bit; a NaN passes
    const uint32_t yh = hi32(y);
    if (yh - 0x40500000u <= 0x7FF00000u - 0x40500000u) y = 64.0;
    // n = floor(64 y / ln 2): the remainder r >= 0 keeps 2^(-n/64) - 1 and
    // exp(-r) - 1 of one sign, so their sum cancels nothing
#ifdef __CUDA_ARCH__
    const double big = __fma_rd(y, kStepInv, 0x1.8p52);
#else
    const double big = std::floor(y * kStepInv) + 0x1.8p52;
#endif
    const double n = big - 0x1.8p52;
    const uint32_t ni = (uint32_t)bits(big);
    double r = fma(-n, kStepHi, y);  // n kStepHi is exact (n < 2^13)
    r = fma(-n, kStepLo, r);
    const double r2 = r * r;
    double q = fma(r, -1.0 / 5040.0, 1.0 / 720.0);
    q = fma(r, q, -1.0 / 120.0);
    q = fma(r, q, 1.0 / 24.0);
    q = fma(r, q, -1.0 / 6.0);
    q = fma(r, q, 1.0 / 2.0);
    const double p = fma(r2, q, -r);  // exp(-r) - 1
    const uint32_t j = ni & 63u;
#ifdef __CUDA_ARCH__
    const double2 t = __ldg(reinterpret_cast<const double2 *>(&d_exp_rows[j]));
    const double th0 = t.x, tl0 = t.y;
#else
    const double th0 = h_exp_rows[j].hi, tl0 = h_exp_rows[j].lo;
#endif
    // times 2^-(n / 64), by the exponents; the low part of row 0 is 0
    const uint64_t sh = (uint64_t)((ni >> 6) & 0x7Fu) << 52;
    const double th = from_bits(bits(th0) - sh), tl = j ? from_bits(bits(tl0) - sh) : 0.0;
    return (th - 1.0) + fma(th, p, tl);
}

// a / b, rb = RN(1 / b): correctly rounded while nothing under- or overflows
IMC_HD double div_r(double a, double b, double rb) {
    const double q = a * rb;
    return fma(fma(-q, b, a), rb, q);
}

}  // namespace m64
}  // namespace imc
