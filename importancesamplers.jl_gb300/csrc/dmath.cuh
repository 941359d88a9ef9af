// dmath.cuh — FP64 exponential and log1p for the mixture kernels, from few FP64
// instructions. An FP64 instruction holds a warp's pipe for 64 cycles on this GPU,
// so the library's exp (19 of them) and log1p (34) are most of a Student-t
// component's cost in low dimensions. Both here are table-driven (P. T. P. Tang,
// "Table-driven implementation of the exponential / logarithm function in IEEE
// floating-point arithmetic", 1989 / 1990): 11 and 21 instructions, the tables 6 KB
// in the L1. Largest errors over a million arguments of the ranges, against 113-bit
// values: exp 0.51 ulp (the library's 0.85), log1p 0.84 (1.49).
#pragma once

#include <cuda_runtime.h>

namespace issm {

// 2^(j / 128), hi and lo
__device__ const double2 kExpTable[128] = {
    {0x1.0000000000000p+0, 0x0p+0},
    {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54},
    {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56},
    {0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55},
    {0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55},
    {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57},
    {0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54},
    {0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54},
    {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59},
    {0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54},
    {0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58},
    {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54},
    {0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55},
    {0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54},
    {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55},
    {0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54},
    {0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54},
    {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55},
    {0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54},
    {0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55},
    {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55},
    {0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55},
    {0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59},
    {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54},
    {0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55},
    {0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55},
    {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54},
    {0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54},
    {0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54},
    {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56},
    {0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55},
    {0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54},
    {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58},
    {0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59},
    {0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54},
    {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56},
    {0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56},
    {0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54},
    {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54},
    {0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55},
    {0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55},
    {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54},
    {0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54},
    {0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60},
    {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54},
    {0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54},
    {0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55},
    {0x1.6623882552225p+0, -0x1.bb60987591c34p-54},
    {0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54},
    {0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56},
    {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57},
    {0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55},
    {0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54},
    {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54},
    {0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55},
    {0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54},
    {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56},
    {0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54},
    {0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55},
    {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54},
    {0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54},
    {0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56},
    {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55},
    {0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57},
    {0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56},
    {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54},
    {0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56},
    {0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56},
    {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54},
    {0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54},
    {0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54},
    {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54},
    {0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54},
    {0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54},
    {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57},
    {0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56},
    {0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54},
    {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55},
    {0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55},
    {0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54},
    {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54},
    {0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56},
    {0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55},
    {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54},
    {0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55},
    {0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54},
    {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54},
    {0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54},
    {0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54},
    {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55},
    {0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54},
    {0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54},
    {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54},
    {0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54},
    {0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54},
    {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55},
    {0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57},
};

// c_j near 1 / (1 + (j + 1/2) / 128) (c_0 = 1), and -log c_j, hi (a multiple of 2^-42) and lo
struct LogEntry {
    double c, hi, lo;
};
__device__ const LogEntry kLogTable[128] = {
    {0x1.0000000000000p+0, 0x0p+0, 0x0p+0},
    {0x1.fa11c00000000p-1, 0x1.7dc725f820000p-7, -0x1.03f24279a767ap-44},
    {0x1.f631000000000p-1, 0x1.3ceba43470000p-6, -0x1.e0b0fed853743p-46},
    {0x1.f25f600000000p-1, 0x1.b9fc8e7b00000p-6, -0x1.9358107695779p-44},
    {0x1.ee9c800000000p-1, 0x1.1b0d909240000p-5, -0x1.3381e9ae9df10p-44},
    {0x1.eae8000000000p-1, 0x1.58a63afc90000p-5, -0x1.656e6d58c041cp-46},
    {0x1.e741a00000000p-1, 0x1.95c8deec90000p-5, 0x1.7c7dd367a2fd4p-49},
    {0x1.e3a9200000000p-1, 0x1.d2762aadb0000p-5, 0x1.f0311a9843dc5p-45},
    {0x1.e01e000000000p-1, 0x1.0759935990000p-4, -0x1.b0ecfe4604432p-44},
    {0x1.dca0200000000p-1, 0x1.253f4ff0a0000p-4, 0x1.4cb78fadac1acp-44},
    {0x1.d92f200000000p-1, 0x1.42eddeea64000p-4, 0x1.e92eeecb83024p-46},
    {0x1.d5cac00000000p-1, 0x1.6065d09374000p-4, 0x1.a55b1fad39aa8p-44},
    {0x1.d272c00000000p-1, 0x1.7da7c0d7b4000p-4, -0x1.d617b802bb66bp-44},
    {0x1.cf26e00000000p-1, 0x1.9ab4576204000p-4, -0x1.cfa9021c2a05bp-46},
    {0x1.cbe6e00000000p-1, 0x1.b78c47bb10000p-4, -0x1.724ef99e084c6p-45},
    {0x1.c8b2600000000p-1, 0x1.d4317066cc000p-4, -0x1.e3886c6f86dc0p-46},
    {0x1.c589400000000p-1, 0x1.f0a3820118000p-4, -0x1.13cefec05b2c1p-47},
    {0x1.c26b600000000p-1, 0x1.067118aca6000p-3, 0x1.799a7784b454ap-45},
    {0x1.bf58400000000p-1, 0x1.1478534674000p-3, 0x1.62b450fd471fbp-46},
    {0x1.bc4fe00000000p-1, 0x1.2266c510a6000p-3, 0x1.43de9aa02c927p-46},
    {0x1.b951e00000000p-1, 0x1.303d7e0e48000p-3, 0x1.bcfa541914558p-49},
    {0x1.b65e200000000p-1, 0x1.3dfc6d8ece000p-3, -0x1.11fea0f2e5561p-44},
    {0x1.b374800000000p-1, 0x1.4ba38539a6000p-3, -0x1.06d4bad036f2cp-44},
    {0x1.b094c00000000p-1, 0x1.5933509982000p-3, 0x1.e1da5f7af2e77p-44},
    {0x1.adbe800000000p-1, 0x1.66acfa272c000p-3, -0x1.a16421c7fe2a6p-44},
    {0x1.aaf1e00000000p-1, 0x1.740f50d404000p-3, 0x1.b9c259018bcafp-45},
    {0x1.a82e600000000p-1, 0x1.815c229436000p-3, -0x1.6f3a5df1a2efap-45},
    {0x1.a574200000000p-1, 0x1.8e92426888000p-3, 0x1.c274e643554fbp-46},
    {0x1.a2c2a00000000p-1, 0x1.9bb38c67e0000p-3, 0x1.1ecaf7684cd87p-46},
    {0x1.a01a000000000p-1, 0x1.a8bed7c882000p-3, 0x1.eb185cf770f25p-44},
    {0x1.9d7a000000000p-1, 0x1.b5b4d1e8fc000p-3, 0x1.3c8dc20fee737p-44},
    {0x1.9ae2400000000p-1, 0x1.c296ce58c2000p-3, 0x1.b23470dd26c50p-44},
    {0x1.9853000000000p-1, 0x1.cf6308e09e000p-3, -0x1.c9dbd431ae023p-46},
    {0x1.95cbc00000000p-1, 0x1.dc1b7d0ac0000p-3, 0x1.d3301f3bfff48p-46},
    {0x1.934c600000000p-1, 0x1.e8c04daaa6000p-3, 0x1.90526acb3d24ap-48},
    {0x1.90d5000000000p-1, 0x1.f5505964ba000p-3, -0x1.c71f2ee13a436p-44},
    {0x1.8e65200000000p-1, 0x1.00e6d81ad5000p-2, 0x1.94734bad64c64p-45},
    {0x1.8bfce00000000p-1, 0x1.071b9abcd6000p-2, -0x1.cae16eaafbd62p-45},
    {0x1.899c000000000p-1, 0x1.0d46dd79ac000p-2, 0x1.e5906872c81ffp-45},
    {0x1.8742800000000p-1, 0x1.136865293b000p-2, -0x1.97684a0c51bbfp-44},
    {0x1.84f0000000000p-1, 0x1.1980f2dd43000p-2, -0x1.24262183a4308p-44},
    {0x1.82a4a00000000p-1, 0x1.1f8ffa248a000p-2, 0x1.7956c040cc921p-45},
    {0x1.8060200000000p-1, 0x1.2595ebcdf8000p-2, -0x1.8fbc40faba0acp-44},
    {0x1.7e22600000000p-1, 0x1.2b92e66b8a000p-2, 0x1.e9dec249274f0p-45},
    {0x1.7beb400000000p-1, 0x1.31870a1544000p-2, 0x1.0c5eac43989bep-44},
    {0x1.79baa00000000p-1, 0x1.3772786bfe000p-2, -0x1.42bb68cab2a61p-44},
    {0x1.7790800000000p-1, 0x1.3d54fd5c1f000p-2, 0x1.c861cd9c795e3p-44},
    {0x1.756ca00000000p-1, 0x1.432f13e04f000p-2, 0x1.6dab962f1a293p-47},
    {0x1.734f000000000p-1, 0x1.49008a0401000p-2, 0x1.6c6619d3695c5p-45},
    {0x1.7137800000000p-1, 0x1.4ec9862600000p-2, 0x1.4eebd7b3bbe57p-44},
    {0x1.6f26000000000p-1, 0x1.548a303add000p-2, 0x1.4167e63b2c7a2p-45},
    {0x1.6d1a600000000p-1, 0x1.5a42b1cf4d000p-2, 0x1.e5e289c46230cp-49},
    {0x1.6b14a00000000p-1, 0x1.5ff2dbca7a000p-2, 0x1.3874054563596p-45},
    {0x1.6914800000000p-1, 0x1.659b34303f000p-2, -0x1.1edf97322c132p-44},
    {0x1.671a000000000p-1, 0x1.6b3b8e235a000p-2, -0x1.a276de1b31cc1p-46},
    {0x1.6525000000000p-1, 0x1.70d4182789000p-2, 0x1.7f756624a1cd3p-44},
    {0x1.6335600000000p-1, 0x1.766502639e000p-2, 0x1.1c785548a2250p-44},
    {0x1.614b400000000p-1, 0x1.7bedc5237b000p-2, 0x1.6a0780fe33f82p-44},
    {0x1.5f66400000000p-1, 0x1.816f4b5a0d000p-2, 0x1.528d6e0ad25fcp-44},
    {0x1.5d86800000000p-1, 0x1.86e90ea331000p-2, -0x1.b6fb02717958bp-45},
    {0x1.5babc00000000p-1, 0x1.8c5ba1058c000p-2, -0x1.0cf7eb82eb8c2p-46},
    {0x1.59d6200000000p-1, 0x1.91c67bf45b000p-2, -0x1.ecd60e0c9ddf5p-44},
    {0x1.5805600000000p-1, 0x1.972a345135000p-2, 0x1.588970274a832p-46},
    {0x1.5639800000000p-1, 0x1.9c86a32dc1000p-2, -0x1.92d918a5cbf17p-44},
    {0x1.5472600000000p-1, 0x1.a1dc018d5c000p-2, -0x1.8f5efee084c9bp-44},
    {0x1.52b0000000000p-1, 0x1.a72a2966be000p-2, 0x1.ea167cc070d2ep-46},
    {0x1.50f2200000000p-1, 0x1.ac71b6e58c000p-2, -0x1.a9a71e4d025a3p-47},
    {0x1.4f39000000000p-1, 0x1.b1b1c2ebe0000p-2, 0x1.b1b4775ec1774p-45},
    {0x1.4d84400000000p-1, 0x1.b6eb4d53cf000p-2, 0x1.258751a070247p-44},
    {0x1.4bd3e00000000p-1, 0x1.bc1e3370dc000p-2, -0x1.2ba7480a472edp-44},
    {0x1.4a28000000000p-1, 0x1.c149ef115f000p-2, 0x1.135665be33dc9p-45},
    {0x1.4880600000000p-1, 0x1.c66f22fff8000p-2, -0x1.6af8929e68dfdp-46},
    {0x1.46dce00000000p-1, 0x1.cb8e1184d8000p-2, -0x1.18f8a3ea0f655p-44},
    {0x1.453da00000000p-1, 0x1.d0a6352722000p-2, -0x1.59baa6a33c51ep-46},
    {0x1.43a2800000000p-1, 0x1.d5b7d0ae2d000p-2, 0x1.d2e5573933b8ep-45},
    {0x1.420b600000000p-1, 0x1.dac328a2c6000p-2, 0x1.fc50a9448b37fp-44},
    {0x1.4078200000000p-1, 0x1.dfc883506e000p-2, 0x1.a9b06b8804bb0p-45},
    {0x1.3ee9000000000p-1, 0x1.e4c6f48688000p-2, 0x1.261643d8e9c89p-45},
    {0x1.3d5da00000000p-1, 0x1.e9bf901986000p-2, 0x1.74e11819da403p-44},
    {0x1.3bd6000000000p-1, 0x1.eeb238640f000p-2, -0x1.75e50518d1183p-45},
    {0x1.3a52400000000p-1, 0x1.f39e674812000p-2, -0x1.3765fb27f4393p-47},
    {0x1.38d2200000000p-1, 0x1.f884ceafeb000p-2, -0x1.505999f7bcfe8p-45},
    {0x1.3755c00000000p-1, 0x1.fd64e88f61000p-2, 0x1.899292332bee8p-44},
    {0x1.35dce00000000p-1, 0x1.011fb4f260000p-1, 0x1.102815e13541ap-45},
    {0x1.3467a00000000p-1, 0x1.0389e65ce6800p-1, -0x1.cd99ec4f6bb26p-44},
    {0x1.32f5c00000000p-1, 0x1.05f1649265000p-1, -0x1.a36a2c59ebf6ap-46},
    {0x1.3187800000000p-1, 0x1.0855b704b4800p-1, 0x1.d75bfa1fe489ap-45},
    {0x1.301c800000000p-1, 0x1.0ab7706ce1800p-1, -0x1.6e9fd68c7544ep-44},
    {0x1.2eb4e00000000p-1, 0x1.0d164deb9d800p-1, 0x1.a6784f46d0b8cp-44},
    {0x1.2d50a00000000p-1, 0x1.0f7241e9b4800p-1, 0x1.7d5ea110ef217p-45},
    {0x1.2befa00000000p-1, 0x1.11cb75587d000p-1, -0x1.775ef65428028p-46},
    {0x1.2a91c00000000p-1, 0x1.1422121244000p-1, 0x1.2532abe82b0a9p-45},
    {0x1.2937200000000p-1, 0x1.1675d49aba800p-1, -0x1.afb178d0d746fp-47},
    {0x1.27dfa00000000p-1, 0x1.18c6e71f5d000p-1, -0x1.8f91310e24f19p-47},
    {0x1.268b400000000p-1, 0x1.1b153d17da800p-1, -0x1.1a68107ebbc57p-44},
    {0x1.2539e00000000p-1, 0x1.1d6101c677000p-1, 0x1.908c1fff70c3dp-44},
    {0x1.23eb800000000p-1, 0x1.1faa293870800p-1, 0x1.ae8601f8534edp-44},
    {0x1.22a0200000000p-1, 0x1.21f0a7665c800p-1, 0x1.a38c7d0d3cc7cp-48},
    {0x1.2157a00000000p-1, 0x1.2434a8d484000p-1, -0x1.d706fd332d0b8p-44},
    {0x1.2012000000000p-1, 0x1.2676221343000p-1, 0x1.df9a55bf74e3dp-46},
    {0x1.1ecf400000000p-1, 0x1.28b5079f60800p-1, 0x1.c77820c474cb2p-48},
    {0x1.1d8f600000000p-1, 0x1.2af14de264800p-1, -0x1.5ee9b4e1f4314p-44},
    {0x1.1c52200000000p-1, 0x1.2d2b5c72ee800p-1, 0x1.323c317205db0p-45},
    {0x1.1b17c00000000p-1, 0x1.2f62b55509800p-1, -0x1.2324d5003be04p-46},
    {0x1.19e0200000000p-1, 0x1.319786da80800p-1, 0x1.142d066ab3cf9p-45},
    {0x1.18ab000000000p-1, 0x1.33ca3aa329000p-1, -0x1.739be9c131d48p-44},
    {0x1.1778a00000000p-1, 0x1.35fa51bd37000p-1, -0x1.3eedb0378097cp-45},
    {0x1.1648e00000000p-1, 0x1.3827fbc588000p-1, -0x1.69840b4615f56p-48},
    {0x1.151ba00000000p-1, 0x1.3a536947ec000p-1, -0x1.0b8da8747dd69p-47},
    {0x1.13f0e00000000p-1, 0x1.3c7c905f73800p-1, -0x1.c9a7b93d0622fp-45},
    {0x1.12c8c00000000p-1, 0x1.3ea32b76b3000p-1, 0x1.27e1e6181c35dp-44},
    {0x1.11a3000000000p-1, 0x1.40c7a7880e000p-1, -0x1.796eb0cb21802p-44},
    {0x1.107fc00000000p-1, 0x1.42e9bf1df8000p-1, 0x1.af6cad4c4f7bcp-45},
    {0x1.0f5ee00000000p-1, 0x1.4509a4733b800p-1, 0x1.85f01fc4e0b05p-44},
    {0x1.0e40600000000p-1, 0x1.47274e133b000p-1, -0x1.dc5f267d03cb9p-44},
    {0x1.0d24400000000p-1, 0x1.4942b27a30000p-1, -0x1.2a225ba789d59p-44},
    {0x1.0c0a800000000p-1, 0x1.4b5bc8156e800p-1, -0x1.21b91731425cdp-44},
    {0x1.0af3000000000p-1, 0x1.4d72c2a3a0000p-1, 0x1.84471b9e5b308p-45},
    {0x1.09ddc00000000p-1, 0x1.4f87993502800p-1, 0x1.6d8b8dc9a7a23p-46},
    {0x1.08cac00000000p-1, 0x1.519a42cba3800p-1, -0x1.31ac9bcd50da3p-44},
    {0x1.07ba000000000p-1, 0x1.53aab65b9a800p-1, -0x1.f355cdb6bbe6bp-45},
    {0x1.06ab600000000p-1, 0x1.55b9292b41000p-1, -0x1.e6b3861979d0ep-45},
    {0x1.059ee00000000p-1, 0x1.57c592d36f800p-1, -0x1.aba8b62c55569p-47},
    {0x1.0494a00000000p-1, 0x1.59cfabffae800p-1, 0x1.2087455e6b565p-45},
    {0x1.038c600000000p-1, 0x1.5bd7e9ae72800p-1, -0x1.c6a9e569c3d17p-44},
    {0x1.0286400000000p-1, 0x1.5dde04b14a800p-1, 0x1.96df76005f243p-47},
    {0x1.0182400000000p-1, 0x1.5fe1f46d18800p-1, 0x1.cecd5ec1cc7ddp-45},
    {0x1.0080400000000p-1, 0x1.61e3f01a46800p-1, -0x1.cc9436e4fb135p-44},
};

// e^x for -60 < x <= 0: x = k ln 2 / 128 + r, |r| <= ln 2 / 256, e^r - 1 to degree 5
__device__ __forceinline__ double table_exp(double x) {
    const double t = fma(x, 0x1.71547652b82fep+7, 0x1.8p52);  // 128 / ln 2: k in the low mantissa bits
    const int k = __double2loint(t);
    const double kd = t - 0x1.8p52;
    double r = fma(-kd, 0x1.62e42fefa4000p-8, x);  // ln 2 / 128 in 39 bits, so k times it is exact
    r = fma(-kd, -0x1.8432a1b0e2634p-50, r);
    const double2 T = kExpTable[k & 127];
    double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    q = fma(r, q, 1.0 / 6.0);
    q = fma(r, q, 0.5);
    const double p = fma(r * r, q, r);
    const double v = T.x + fma(T.x, p, T.y);
    return __hiloint2double(__double2hiint(v) + (k >> 7) * (1 << 20), __double2loint(v));
}

// log(1 + z) for finite z >= 0: u + c = 1 + z exactly, u = 2^k m, r = (m + c 2^-k) c_j - 1,
// |r| < 2^-7, log(1 + r) to degree 8. c_0 = 1 keeps a small z's relative accuracy.
__device__ __forceinline__ double table_log1p(double z) {
    const bool big = __double2hiint(z) >= 0x3ff00000;
    const double u = 1.0 + z;
    const double a = big ? z : 1.0, b = big ? 1.0 : z;
    const double c = b - (u - a);
    const int hi = __double2hiint(u), k = (hi >> 20) - 1023;
    const LogEntry *e = kLogTable + ((hi >> 13) & 127);
    const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(u));
    // c 2^-k: c is 0, z (k = 0) or a multiple of 2^-52, and beyond k = 60 it does not count
    const int chi = __double2hiint(c);
    const double cs = (chi & 0x7ff00000) == 0 && k > 0 || k > 60 ? 0.0
                                                                 : __hiloint2double(chi - k * (1 << 20), __double2loint(c));
    double r = fma(m, e->c, -1.0);
    r = fma(cs, e->c, r);
    double p = fma(r, -1.0 / 8.0, 1.0 / 7.0);
    p = fma(r, p, -1.0 / 6.0);
    p = fma(r, p, 1.0 / 5.0);
    p = fma(r, p, -1.0 / 4.0);
    p = fma(r, p, 1.0 / 3.0);
    p = fma(r, p, -0.5);
    const double kd = __hiloint2double(0x43380000, k) - 0x1.8p52;  // k >= 0
    const double h = fma(kd, 0x1.62e42fefa3800p-1, e->hi);  // exact: both are multiples of 2^-42
    const double l = fma(kd, 0x1.ef35793c76730p-45, e->lo);
    const double s = h + r;  // h = 0 or h > |r|
    return s + (((h - s) + r) + fma(r * r, p, l));
}

}  // namespace issm
