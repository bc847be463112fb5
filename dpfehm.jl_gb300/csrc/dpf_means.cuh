// dpf_means.cuh -- FP64 exponentials, powers, reciprocals and face means with few FP64 instructions (a B300 SM issues 1.6 FP64
// lanes a clock, against 128 FP32 and 64 integer ones, so every kernel that evaluates them is bound by them).
#pragma once
#include "dpf_internal.h"

namespace dpf {

// 2^(j/256) as an unevaluated sum of two doubles, each the nearest one
static __device__ const double2 kExp2Table[256] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.00b1afa5abcbfp+0, -0x1.4f6b2a7609f71p-55}, {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54},
    {0x1.02168143b0281p+0, -0x1.2bf310fc54eb6p-55}, {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56}, {0x1.037d42e11bbccp+0, 0x1.56811eeade11ap-57},
    {0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54}, {0x1.04e5f72f654b1p+0, 0x1.4c3793aa0d08dp-55}, {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55},
    {0x1.0650a0e3c1f89p+0, -0x1.5cb7b5799c397p-54}, {0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55}, {0x1.07bd42b72a836p+0, 0x1.3233454458700p-55},
    {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57}, {0x1.092bdf66607e0p+0, -0x1.68063800a3fd1p-54}, {0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54},
    {0x1.0a9c79b1f3919p+0, 0x1.5d16c873d1d38p-55}, {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0c0f145e46c85p+0, 0x1.4f98906d21cefp-54},
    {0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54}, {0x1.0d83b23395decp+0, -0x1.bc14de43f316ap-54}, {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59},
    {0x1.0efa55fdfa9c5p+0, -0x1.49db9bc54021bp-54}, {0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57}, {0x1.1073028d7233ep+0, 0x1.d46eb1692fdd5p-55},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.11edbab5e2ab6p+0, -0x1.ca454f703fb72p-54}, {0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58},
    {0x1.136a814f204abp+0, -0x1.7108fba48dcf0p-57}, {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54}, {0x1.14e95934f312ep+0, -0x1.b91e839bf44abp-55},
    {0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55}, {0x1.166a45471c3c2p+0, 0x1.8f23b82ea1a32p-58}, {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55},
    {0x1.17ed48695bbc0p+0, 0x1.09e3fe2ac5a64p-56}, {0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54}, {0x1.1972658375d2fp+0, 0x1.4aadd85f17e08p-54},
    {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55}, {0x1.1af99f8138a1cp+0, 0x1.7bf85a4b69280p-54}, {0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54},
    {0x1.1c82f95281c6bp+0, 0x1.009778010f8c9p-54}, {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.1e0e75eb44027p+0, -0x1.6fdd8088cb6dep-54},
    {0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54}, {0x1.1f9c18438ce4dp+0, -0x1.bf524a097af5cp-54}, {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55},
    {0x1.212be3578a819p+0, 0x1.3592d2cfcaac9p-54}, {0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55}, {0x1.22bdda27912d1p+0, 0x1.d34fb5577d69fp-55},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.2451ffb82140ap+0, 0x1.acfcc911ca996p-55}, {0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55},
    {0x1.25e85711ece75p+0, 0x1.3e1a24ac31b2cp-54}, {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55}, {0x1.2780e341ddf29p+0, 0x1.e067c05f9e76cp-54},
    {0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54}, {0x1.291ba7591bb70p+0, -0x1.2cc7228401cbdp-55}, {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55},
    {0x1.2ab8a66d10f13p+0, -0x1.95743191690a7p-54}, {0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59}, {0x1.2c57e39771b2fp+0, -0x1.50145a6eb5124p-54},
    {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54}, {0x1.2df961f641589p+0, 0x1.d16cffbbce198p-54}, {0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56},
    {0x1.2f9d24abd886bp+0, -0x1.53c55532bda93p-57}, {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.31432edeeb2fdp+0, 0x1.959a3f3f3fcd1p-55},
    {0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55}, {0x1.32eb83ba8ea32p+0, -0x1.c45e83cb4f318p-54}, {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54},
    {0x1.3496266e3fa2dp+0, -0x1.35a75930881a4p-55}, {0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55}, {0x1.36431a2de883bp+0, -0x1.c3144a06cb85ep-55},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.37f26231e754ap+0, -0x1.9f5ca9eceb23cp-54}, {0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54},
    {0x1.39a401b7140efp+0, -0x1.9a9a5fc8e2934p-54}, {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56}, {0x1.3b57fbfec6cf4p+0, 0x1.54c66e26fff18p-54},
    {0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54}, {0x1.3d0e544ede173p+0, 0x1.fe8d08c284c71p-56}, {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55},
    {0x1.3ec70df1c5175p+0, -0x1.af6637b8c9bcap-55}, {0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54}, {0x1.40822c367a024p+0, 0x1.bddf8b6f4d048p-55},
    {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58}, {0x1.423fb2709468ap+0, -0x1.8462dc0b314ddp-54}, {0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55},
    {0x1.43ffa3f84b9d4p+0, 0x1.880be9704c003p-55}, {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.45c2042a7d232p+0, -0x1.8641982fb1f8ep-57},
    {0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54}, {0x1.4786d668b3237p+0, -0x1.c20f0ed445733p-54}, {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56},
    {0x1.494e1e192aed2p+0, -0x1.3b2895e499ea0p-55}, {0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54}, {0x1.4b17dea6db7d7p+0, -0x1.125b87f2897f0p-55},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4ce41b817c114p+0, 0x1.05e29690abd5dp-54}, {0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54},
    {0x1.4eb2d81d8abffp+0, -0x1.5257d2e5d7a52p-54}, {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54}, {0x1.508417f4531eep+0, 0x1.a249b49b7465fp-56},
    {0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55}, {0x1.5257de83f4eefp+0, -0x1.c998d43efef71p-56}, {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55},
    {0x1.542e2f4f6ad27p+0, 0x1.7926d192d5f7ep-55}, {0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55}, {0x1.56070dde910d2p+0, -0x1.0fb6e168eebf0p-54},
    {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54}, {0x1.57e27dbe2c4cfp+0, -0x1.0b98c8a57b9c4p-54}, {0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55},
    {0x1.59c0827ff07ccp+0, -0x1.7e2cee467e60fp-54}, {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5ba11fba87a03p+0, -0x1.b77a14c233e1ap-54},
    {0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60}, {0x1.5d84590998b93p+0, -0x1.cd6a7a8b45643p-54}, {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54},
    {0x1.5f6a320dceb71p+0, -0x1.9eadde3cdcf92p-55}, {0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54}, {0x1.6152ae6cdf6f4p+0, 0x1.e4b3e4ab84c27p-54},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.633dd1d1929fdp+0, 0x1.84710beb964e5p-54}, {0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55},
    {0x1.652b9febc8fb7p+0, -0x1.ae3d5c9a73e09p-54}, {0x1.6623882552225p+0, -0x1.bb60987591c34p-54}, {0x1.671c1c70833f6p+0, -0x1.e8732586c6134p-55},
    {0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57}, {0x1.690f4b19e9538p+0, 0x1.804bd9aeb445dp-55}, {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54},
    {0x1.6b052fa75173ep+0, 0x1.a38f52c9a9d0ep-56}, {0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56}, {0x1.6cfdcddd47645p+0, 0x1.c7aa9b6f17309p-54},
    {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57}, {0x1.6ef9298593ae5p+0, -0x1.0b9749e1ac8b2p-54}, {0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55},
    {0x1.70f7466f42e87p+0, 0x1.9d644d45aa65fp-58}, {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.72f8286ead08ap+0, -0x1.20aa02cd62c72p-54},
    {0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54}, {0x1.74fbd35d7cbfdp+0, 0x1.047fd618a6e1cp-54}, {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54},
    {0x1.77024b1ab6e09p+0, 0x1.b7877169147f8p-54}, {0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54}, {0x1.790b938ac1cf6p+0, 0x1.349a862aadd3ep-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7b17b0976cfdbp+0, -0x1.bebb58468dc88p-54}, {0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54},
    {0x1.7d26a62ff86f0p+0, 0x1.1bddbfb72b8b4p-54}, {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56}, {0x1.7f3878491c491p+0, -0x1.07f11cf9311aep-55},
    {0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54}, {0x1.814d2add106d9p+0, 0x1.464370d151d4dp-54}, {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54},
    {0x1.8364c1eb941f7p+0, 0x1.99b9a31df2bd5p-54}, {0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55}, {0x1.857f4179f5b21p+0, -0x1.ba748f8b216d0p-58},
    {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54}, {0x1.879cad931a436p+0, 0x1.5d2d7d2db47bdp-55}, {0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54},
    {0x1.89bd0a478580fp+0, 0x1.d53954475202bp-54}, {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8be05bad61778p+0, 0x1.ecb5efc43446ep-54},
    {0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56}, {0x1.8e06a5e0866d9p+0, -0x1.7114a6fc9b2e6p-54}, {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55},
    {0x1.902fed0282c8ap+0, 0x1.592ca85fe3fd2p-54}, {0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54}, {0x1.925c353aa2fe2p+0, -0x1.3455fa639db7fp-55},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.948b82b5f98e5p+0, -0x1.dc3d6797d2d99p-55}, {0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56},
    {0x1.96bdd9a7670b3p+0, -0x1.ba5967f19c896p-58}, {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54}, {0x1.98f33e47a22a2p+0, 0x1.cabdaa24c78edp-56},
    {0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54}, {0x1.9b2bb4d53fe0dp+0, -0x1.dd84e4df6d518p-54}, {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56},
    {0x1.9d674194bb8d5p+0, -0x1.516bea3dd8233p-54}, {0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56}, {0x1.9fa5e8d07f29ep+0, -0x1.4a9ceaaf1facep-55},
    {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54}, {0x1.a1e7aed8eb8bbp+0, 0x1.c6618ee8be70ep-54}, {0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54},
    {0x1.a42c980460ad8p+0, -0x1.aa780589fb120p-54}, {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a674a8af46052p+0, 0x1.50f5630670366p-57},
    {0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54}, {0x1.a8bfe53c12e59p+0, -0x1.4f867b2ba15a9p-54}, {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54},
    {0x1.ab0e521356ebap+0, 0x1.89c31dae94545p-55}, {0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55}, {0x1.ad5ff3a3c2774p+0, 0x1.7ef3bb6b1b8e5p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.afb4ce622f2ffp+0, -0x1.4b2fc0f315ecdp-54}, {0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54},
    {0x1.b20ce6c9a8952p+0, 0x1.4dd024a0756ccp-54}, {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57}, {0x1.b468415b749b1p+0, -0x1.f763de9df7c90p-56},
    {0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54}, {0x1.b6c6e29f1c52ap+0, 0x1.2a8f352883f6ep-54}, {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56},
    {0x1.b928cf22749e4p+0, -0x1.b721654cb65c6p-54}, {0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54}, {0x1.bb8e0b79a6f1fp+0, -0x1.f52d1c9696205p-60},
    {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55}, {0x1.bdf69c3f3a207p+0, -0x1.c262360ea5b52p-60}, {0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54},
    {0x1.c06286141b33dp+0, -0x1.d8a5aa1fbca34p-55}, {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c2d1cd9fa652cp+0, -0x1.6e51617c8a5d7p-54},
    {0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54}, {0x1.c544778fafb22p+0, 0x1.12f072493b5afp-54}, {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54},
    {0x1.c7ba88988c933p+0, -0x1.e76bbbe255559p-55}, {0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56}, {0x1.ca3405751c4dbp+0, -0x1.7f2bed10d08f5p-55},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.ccb0f2e6d1675p+0, -0x1.d220f86009093p-56}, {0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55},
    {0x1.cf3155b5bab74p+0, -0x1.a08e9b86dff57p-54}, {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54}, {0x1.d1b532b08c968p+0, 0x1.55636219a36eep-54},
    {0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54}, {0x1.d43c8eacaa1d6p+0, 0x1.3db53bf5a1614p-54}, {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55},
    {0x1.d6c76e862e6d3p+0, 0x1.fe87a4a8165a0p-58}, {0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54}, {0x1.d955d71ff6075p+0, 0x1.a052dbb9af6bep-54},
    {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54}, {0x1.dbe7cd63a8315p+0, -0x1.b76f1926b8be4p-54}, {0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54},
    {0x1.de7d5641c0658p+0, -0x1.ca5528e79ba8fp-54}, {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e11676b197d17p+0, -0x1.2b529bd5c7f44p-56},
    {0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54}, {0x1.e3b333b16ee12p+0, -0x1.9f4a431fdc68bp-54}, {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55},
    {0x1.e653924676d76p+0, -0x1.63ff87522b735p-55}, {0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54}, {0x1.e8f7977cdb740p+0, -0x1.1089480b054b1p-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.eb9f4867cca6ep+0, 0x1.4832f2293e4f2p-54}, {0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54},
    {0x1.ee4aaa2188510p+0, 0x1.1c68da487568dp-54}, {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54}, {0x1.f0f9c1cb6412ap+0, -0x1.3220065181d45p-54},
    {0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54}, {0x1.f3ac948dd7274p+0, -0x1.95a5a3ed837dep-56}, {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54},
    {0x1.f6632798844f8p+0, 0x1.fa37b3539343ep-54}, {0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54}, {0x1.f91d802243c89p+0, -0x1.12ea8a779f689p-57},
    {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55}, {0x1.fbdba3692d514p+0, -0x1.9677315098eb6p-56}, {0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57},
    {0x1.fe9d96b2a23d9p+0, 0x1.4a6037442fde3p-56},
};

// exp(kHalf ? x / 2 : x) by Tang's table-driven method (P. T. P. Tang, ACM TOMS 15, 1989): x' = (256 k + j) ln2/256
// + r, |r| <= R, e^x' = 2^k (T_j + (T_j p(r) + t_j)), p = e^r - 1 to degree 4 with r^5/120 economised (its
// Chebyshev remainder R^5/1920 is 2e-18). Eight
// FP64 instructions (the integer part comes from an FP32 product, whose error only widens r); ln2/256 is split
// after 34 bits, so that n ln2/256 is exact in its leading part. The table's low part keeps the error at 0.51 ulp. Arguments beyond
// +-700 (and infinities and NaN) take the library's function.
template <bool kHalf>
__device__ __forceinline__ double exp64(double x) {
    const float xf = (float)x;
    if (!(fabsf(xf) < (kHalf ? 1400.0f : 700.0f))) return exp(kHalf ? 0.5 * x : x);
    const float nf = rintf(xf * (kHalf ? 184.66497f : 369.32994f));
    const double nd = (double)nf;
    constexpr double s = kHalf ? 2.0 : 1.0;  // r is s times the reduced argument, |r| <= s R
    constexpr double R = 0x1.63p-10;         // 1.0001 ln2/512
    double r = fma(nd, -s * 0x1.62e42fef80000p-9, x);
    r = fma(nd, -s * 0x1.1cf79abc9e3b4p-44, r);
    double p = fma(r, 1.0 / (24.0 * s * s * s * s), (1.0 / 6.0 + R * R / 96.0) / (s * s * s));
    p = fma(p, r, 1.0 / (2.0 * s * s));
    p = fma(p, r, (1.0 - R * R * R * R / 384.0) / s);
    p *= r;
    const int n = (int)nf;
    const double2 t = kExp2Table[n & 255];
    const double v = t.x + fma(t.x, p, t.y);
    return __longlong_as_double(__double_as_longlong(v) + ((long long)(n >> 8) << 52));
}

// log x of a normal x as hi + lo with an absolute error near 2^-61, table-driven (P. T. P. Tang, ACM TOMS 16,
// 1990): x = 2^k m, c_j about 1 / m to 9 bits, log x = k ln2 - log c_j + log1p(m c_j - 1); ln2 and the table
// are split at 2^-42, so that the sum of their leading parts is exact. 16 FP64 instructions.
struct LogDD {
    double hi, lo;
};
static __device__ const double kLogTable[128][3] = {  // c, -log c rounded to a multiple of 2^-42, the rest
    {0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0}, {0x1.fa00000000000p-1, 0x1.82448a3880000p-7, 0x1.4554412c584e0p-44},
    {0x1.f600000000000p-1, 0x1.432a925980000p-6, 0x1.98139928637fep-47}, {0x1.f200000000000p-1, 0x1.c63d2ec150000p-6, -0x1.5439ce030a687p-44},
    {0x1.ef00000000000p-1, 0x1.149e3e4008000p-5, -0x1.2b98a9a4168fdp-44}, {0x1.eb00000000000p-1, 0x1.5715c4c040000p-5, -0x1.8888ddfc47628p-44},
    {0x1.e700000000000p-1, 0x1.9a187b5740000p-5, -0x1.0c22e4ec4d90dp-44}, {0x1.e400000000000p-1, 0x1.ccb73cddd8000p-5, 0x1.965c36e09f5fep-44},
    {0x1.e000000000000p-1, 0x1.08598b59e4000p-4, -0x1.7e5dd7009902cp-46}, {0x1.dd00000000000p-1, 0x1.2207b5c784000p-4, 0x1.49d8cfc10c7bfp-44},
    {0x1.d900000000000p-1, 0x1.4485e03dbc000p-4, 0x1.fad46e8d26ab7p-44}, {0x1.d600000000000p-1, 0x1.5e95a4d978000p-4, 0x1.1cb7ce1d17171p-44},
    {0x1.d200000000000p-1, 0x1.8197e2f410000p-4, -0x1.c0fe460d20041p-44}, {0x1.cf00000000000p-1, 0x1.9c0c32d4d4000p-4, -0x1.ab7c09e838668p-44},
    {0x1.cc00000000000p-1, 0x1.b6ac88dad4000p-4, 0x1.b1bdff50225c7p-44}, {0x1.c900000000000p-1, 0x1.d179788218000p-4, 0x1.36433b5efbeedp-44},
    {0x1.c600000000000p-1, 0x1.ec739830a0000p-4, 0x1.11fcba80cdd10p-44}, {0x1.c200000000000p-1, 0x1.08598b59e4000p-3, -0x1.7e5dd7009902cp-45},
    {0x1.bf00000000000p-1, 0x1.160c8024b2000p-3, 0x1.ec2d2a9009e3dp-45}, {0x1.bc00000000000p-1, 0x1.23d712a49c000p-3, 0x1.00d238fd3df5cp-46},
    {0x1.b900000000000p-1, 0x1.31b994d3a4000p-3, 0x1.f098ee3a50810p-44}, {0x1.b600000000000p-1, 0x1.3fb45a5992000p-3, 0x1.19713c0cae559p-44},
    {0x1.b300000000000p-1, 0x1.4dc7b897bc000p-3, 0x1.c79b60ae1ff0fp-47}, {0x1.b100000000000p-1, 0x1.5737cc9018000p-3, 0x1.9baa7a6b887f6p-44},
    {0x1.ae00000000000p-1, 0x1.6574ebe8c2000p-3, -0x1.98c1d34f0f462p-44}, {0x1.ab00000000000p-1, 0x1.73cb9074fe000p-3, -0x1.d66a90d0005a6p-44},
    {0x1.a800000000000p-1, 0x1.823c16551a000p-3, 0x1.e0ddb9a631e83p-46}, {0x1.a500000000000p-1, 0x1.90c6db9fcc000p-3, -0x1.935f57718d7cap-46},
    {0x1.a300000000000p-1, 0x1.9a8778deba000p-3, 0x1.470fa3efec390p-44}, {0x1.a000000000000p-1, 0x1.a93ed3c8ae000p-3, -0x1.8724350562169p-45},
    {0x1.9d00000000000p-1, 0x1.b811730b82000p-3, 0x1.e90683b9cd768p-46}, {0x1.9b00000000000p-1, 0x1.c2028ab180000p-3, -0x1.92e0ee55c7ac6p-45},
    {0x1.9800000000000p-1, 0x1.d1037f2656000p-3, -0x1.84a7e75b6f6e4p-47}, {0x1.9600000000000p-1, 0x1.db13db0d48000p-3, 0x1.2806a847527e6p-44},
    {0x1.9300000000000p-1, 0x1.ea4449f04a000p-3, 0x1.5e91663732a36p-44}, {0x1.9100000000000p-1, 0x1.f474b134e0000p-3, -0x1.bae49f1df7b5ep-44},
    {0x1.8e00000000000p-1, 0x1.01eae5626c000p-2, 0x1.a43dcfade85aep-44}, {0x1.8c00000000000p-1, 0x1.07138604d6000p-2, -0x1.e76324e912b17p-44},
    {0x1.8a00000000000p-1, 0x1.0c42d67616000p-2, 0x1.7188b163ceae9p-45}, {0x1.8700000000000p-1, 0x1.14167ef367000p-2, 0x1.e0c07824daaf5p-44},
    {0x1.8500000000000p-1, 0x1.1956d3b9bc000p-2, 0x1.7d2f73ad1aa14p-45}, {0x1.8300000000000p-1, 0x1.1e9e16788a000p-2, -0x1.82eaed3c8b65ep-44},
    {0x1.8000000000000p-1, 0x1.269621134e000p-2, -0x1.1b61f10522625p-44}, {0x1.7e00000000000p-1, 0x1.2bef07cdc9000p-2, 0x1.a9cfa4a5004f4p-45},
    {0x1.7c00000000000p-1, 0x1.314f1e1d36000p-2, -0x1.8e27ad3213cb8p-45}, {0x1.7a00000000000p-1, 0x1.36b6776be1000p-2, 0x1.16ecdb0f177c8p-46},
    {0x1.7800000000000p-1, 0x1.3c25277333000p-2, 0x1.83b54b606bd5cp-46}, {0x1.7500000000000p-1, 0x1.44591e053a000p-2, -0x1.6e95892923d88p-47},
    {0x1.7300000000000p-1, 0x1.49da7f3bcc000p-2, 0x1.07b334daf4b9ap-44}, {0x1.7100000000000p-1, 0x1.4f637ebbaa000p-2, -0x1.fc158cb3124b9p-44},
    {0x1.6f00000000000p-1, 0x1.54f431b7be000p-2, 0x1.a8954c0910952p-46}, {0x1.6d00000000000p-1, 0x1.5a8cadbbee000p-2, -0x1.7c79b0af7ecf8p-48},
    {0x1.6b00000000000p-1, 0x1.602d08af09000p-2, 0x1.ebe9176df3f65p-46}, {0x1.6900000000000p-1, 0x1.65d558d4ce000p-2, 0x1.544fd2dc5bdc0p-51},
    {0x1.6700000000000p-1, 0x1.6b85b4cffa000p-2, 0x1.fe6750d372503p-45}, {0x1.6500000000000p-1, 0x1.713e33a46a000p-2, 0x1.7b9b2617e9472p-46},
    {0x1.6300000000000p-1, 0x1.76feecb947000p-2, 0x1.74bb9c9852c57p-46}, {0x1.6100000000000p-1, 0x1.7cc7f7db47000p-2, -0x1.7c98438023cdcp-44},
    {0x1.5f00000000000p-1, 0x1.82996d3ef9000p-2, -0x1.0d52aa30536bbp-44}, {0x1.5e00000000000p-1, 0x1.85855776dd000p-2, -0x1.015486666443bp-44},
    {0x1.5c00000000000p-1, 0x1.8b639a88b3000p-2, -0x1.05ae1e5e70470p-45}, {0x1.5a00000000000p-1, 0x1.914a8635bf000p-2, 0x1.a2652b44673e1p-44},
    {0x1.5800000000000p-1, 0x1.973a343135000p-2, 0x1.ab73b16bf4984p-44}, {0x1.5600000000000p-1, 0x1.9d32bea15f000p-2, -0x1.6279e10d0c0b0p-45},
    {0x1.5400000000000p-1, 0x1.a334402250000p-2, -0x1.61cdd40314305p-44}, {0x1.5300000000000p-1, 0x1.a63865fabd000p-2, 0x1.d7bae3eeaa2e6p-47},
    {0x1.5100000000000p-1, 0x1.ac478d0205000p-2, 0x1.bc0e8cc8a54afp-48}, {0x1.4f00000000000p-1, 0x1.b25fefb60d000p-2, -0x1.347cf9c45db45p-44},
    {0x1.4e00000000000p-1, 0x1.b56fa04463000p-2, -0x1.bdab6b49ef99bp-44}, {0x1.4c00000000000p-1, 0x1.bb9611b80e000p-2, 0x1.7d85bf40a666dp-45},
    {0x1.4a00000000000p-1, 0x1.c1c60693fa000p-2, 0x1.cec807fe8e180p-45}, {0x1.4900000000000p-1, 0x1.c4e19b8472000p-2, 0x1.e0d23293066a0p-45},
    {0x1.4700000000000p-1, 0x1.cb200d2ceb000p-2, 0x1.90b9d9a2cb517p-44}, {0x1.4500000000000p-1, 0x1.d1684d49f4000p-2, 0x1.ab9d98a582718p-44},
    {0x1.4400000000000p-1, 0x1.d490246df0000p-2, -0x1.652280b2c4c2cp-44}, {0x1.4200000000000p-1, 0x1.dae75484c9000p-2, 0x1.856f4a7c8e7a6p-44},
    {0x1.4000000000000p-1, 0x1.e148a1a272000p-2, 0x1.b36537e3375b2p-44}, {0x1.3f00000000000p-1, 0x1.e47d1d32e6000p-2, 0x1.df865b95578b8p-44},
    {0x1.3d00000000000p-1, 0x1.eaedd2eaca000p-2, -0x1.bcf314a1b2d37p-44}, {0x1.3c00000000000p-1, 0x1.ee2a156b41000p-2, 0x1.f27f45a470251p-45},
    {0x1.3a00000000000p-1, 0x1.f4aa7ee032000p-2, -0x1.b4c86a43fad5dp-44}, {0x1.3900000000000p-1, 0x1.f7eeae6b57000p-2, 0x1.873001acabb96p-44},
    {0x1.3700000000000p-1, 0x1.fe7f18eb04000p-2, -0x1.60f51ceb37e7ap-45}, {0x1.3600000000000p-1, 0x1.00e5ae5b20800p-1, -0x1.53ba3b1727b1cp-47},
    {0x1.3400000000000p-1, 0x1.04360be760000p-1, 0x1.d6774030d58c4p-44}, {0x1.3300000000000p-1, 0x1.05e04c1aa3000p-1, -0x1.fcfe79d1ac1c7p-44},
    {0x1.3200000000000p-1, 0x1.078bf0533c800p-1, -0x1.4bf6edf090501p-44}, {0x1.3000000000000p-1, 0x1.0ae76e2d05800p-1, -0x1.82de51de06076p-44},
    {0x1.2f00000000000p-1, 0x1.0c974c8943000p-1, 0x1.cdc0a7cdcbb87p-45}, {0x1.2d00000000000p-1, 0x1.0ffb54213a800p-1, -0x1.c5108822a3283p-44},
    {0x1.2c00000000000p-1, 0x1.11af823c75800p-1, 0x1.53cdc223111a7p-44}, {0x1.2b00000000000p-1, 0x1.1365252bf0800p-1, 0x1.930b4c43a97c2p-47},
    {0x1.2900000000000p-1, 0x1.16d4d38c11800p-1, 0x1.fa75d42395d88p-45}, {0x1.2800000000000p-1, 0x1.188ee40f24000p-1, -0x1.accec41d52e6cp-44},
    {0x1.2700000000000p-1, 0x1.1a4a738b7a000p-1, 0x1.9e2b126042793p-44}, {0x1.2500000000000p-1, 0x1.1dc619de06800p-1, 0x1.441b50bb38388p-45},
    {0x1.2400000000000p-1, 0x1.1f8635fc61800p-1, -0x1.a7242c9fe81d3p-45}, {0x1.2300000000000p-1, 0x1.2147dba47a000p-1, 0x1.c9d579851b8b6p-44},
    {0x1.2100000000000p-1, 0x1.24cfce6f81000p-1, -0x1.32cb5b2e5bdd7p-44}, {0x1.2000000000000p-1, 0x1.269621134d800p-1, 0x1.c93c1df5bb3b6p-44},
    {0x1.1f00000000000p-1, 0x1.285e0842ca000p-1, 0x1.c1c4d866d5f22p-44}, {0x1.1e00000000000p-1, 0x1.2a2786d0ec000p-1, 0x1.06d2be797882dp-45},
    {0x1.1c00000000000p-1, 0x1.2dbf557b0e000p-1, -0x1.7a6e507b9dc11p-46}, {0x1.1b00000000000p-1, 0x1.2f8dab6363000p-1, 0x1.bcccfdd1febc9p-44},
    {0x1.1a00000000000p-1, 0x1.315da44340800p-1, -0x1.74e93c5a0ed9cp-45}, {0x1.1900000000000p-1, 0x1.332f4314ad800p-1, -0x1.a96c3d4e8a818p-47},
    {0x1.1700000000000p-1, 0x1.36d77e9d35000p-1, -0x1.4a061506115f9p-48}, {0x1.1600000000000p-1, 0x1.38ae217197800p-1, -0x1.18b7abb5569a4p-45},
    {0x1.1500000000000p-1, 0x1.3a86767257000p-1, 0x1.112e01e8919cap-45}, {0x1.1400000000000p-1, 0x1.3c6080c36c000p-1, -0x1.2b7367cfe13c2p-47},
    {0x1.1300000000000p-1, 0x1.3e3c43918f800p-1, -0x1.27534c617cda4p-46}, {0x1.1200000000000p-1, 0x1.4019c2125c800p-1, 0x1.498c367879c5ap-44},
    {0x1.1000000000000p-1, 0x1.43d9ff2f92000p-1, 0x1.e267b0b7efae1p-44}, {0x1.0f00000000000p-1, 0x1.45bcc464c8800p-1, 0x1.3a145b00234d8p-45},
    {0x1.0e00000000000p-1, 0x1.47a1527e8a000p-1, 0x1.69a4a83594fabp-44}, {0x1.0d00000000000p-1, 0x1.4987ace0da800p-1, 0x1.d83ed15c6b2f4p-44},
    {0x1.0c00000000000p-1, 0x1.4b6fd6f971000p-1, -0x1.f047750959d5fp-44}, {0x1.0b00000000000p-1, 0x1.4d59d43fda800p-1, 0x1.d0f65949c0a34p-44},
    {0x1.0a00000000000p-1, 0x1.4f45a835a5000p-1, -0x1.e6c516d93b8fbp-45}, {0x1.0900000000000p-1, 0x1.5133566680000p-1, -0x1.d46359b33c2adp-44},
    {0x1.0800000000000p-1, 0x1.5322e26867800p-1, 0x1.5ccc45d257531p-47}, {0x1.0700000000000p-1, 0x1.55144fdbcc000p-1, -0x1.4ec532b35ba3ep-44},
    {0x1.0600000000000p-1, 0x1.5707a26bb9000p-1, -0x1.cccfe80199f84p-44}, {0x1.0500000000000p-1, 0x1.58fcddce00800p-1, -0x1.9e3900345a85dp-44},
    {0x1.0400000000000p-1, 0x1.5af405c364800p-1, 0x1.dfa63ac10c9fbp-45}, {0x1.0300000000000p-1, 0x1.5ced1e17c3800p-1, -0x1.1d52fdabeaa73p-44},
    {0x1.0200000000000p-1, 0x1.5ee82aa241800p-1, 0x1.202380cda46bep-45}, {0x1.0000000000000p-1, 0x1.62e42fefa3800p-1, 0x1.ef35793c76730p-45},
};
__device__ __forceinline__ LogDD log_dd(double x) {
    const long long u = __double_as_longlong(x);
    const double *t = kLogTable[(u >> 45) & 127];
    const double m = __longlong_as_double((u & 0xFFFFFFFFFFFFFll) | 0x3FF0000000000000ll);
    const double k = (double)((float)((int)(u >> 52) - 1023));
    const double r = fma(m, t[0], -1.0);  // |r| <= 2^-7, rounded at 2^-61
    const double h = fma(k, 0x1.62e42fefa3800p-1, t[1]);
    const double s = h + r, e = r - (s - h);
    double p = fma(r, -1.0 / 8.0, 1.0 / 7.0);
    p = fma(p, r, -1.0 / 6.0);
    p = fma(p, r, 1.0 / 5.0);
    p = fma(p, r, -1.0 / 4.0);
    p = fma(p, r, 1.0 / 3.0);
    p = fma(p, r, -1.0 / 2.0);
    p *= r * r;
    return {s, e + (p + fma(k, 0x1.ef35793c76730p-45, t[2]))};
}
// x^y for x >= 0, and log x beside it, in 28 FP64 instructions against about 75 of the library's power; error
// 0.61 ulp (0.56 for the logarithm). |y| above 6 takes the library's: y lo, up to |y| 2^-15, takes r beyond the range R
// that p is made for (0.66 ulp at |y| = 8, 1.0 at 16, 97 at 100, 2e6 at 1000; the library's is within 2), and so do
// zero, subnormal, infinite and NaN x and results beyond e^+-700.
__device__ __forceinline__ double pow64(double x, double y, LogDD &lx) {
    const unsigned ex = (unsigned)(__double2hiint(x) >> 20);
    if (ex - 23u > 2000u) {
        lx = {log(x), 0.0};
        return pow(x, y);
    }
    lx = log_dd(x);
    if ((__double2hiint(y) & 0x7FFFFFFF) > 0x40180000) return pow(x, y);  // 6.0, to 2^-18
    const double z = y * lx.hi;
    const float zf = (float)z;
    if (!(fabsf(zf) < 700.0f)) return pow(x, y);
    const double zl = fma(y, lx.lo, fma(y, lx.hi, -z));
    constexpr double R = 0x1.63p-10;  // as in exp64
    const float nf = rintf(zf * 369.32994f);
    const double nd = (double)nf;
    double r = fma(nd, -0x1.62e42fef80000p-9, z);
    r = fma(nd, -0x1.1cf79abc9e3b4p-44, r) + zl;
    double p = fma(r, 1.0 / 24.0, 1.0 / 6.0 + R * R / 96.0);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0 - R * R * R * R / 384.0);
    p *= r;
    const int n = (int)nf;
    const double2 t = kExp2Table[n & 255];
    const double v = t.x + fma(t.x, p, t.y);
    return __longlong_as_double(__double_as_longlong(v) + ((long long)(n >> 8) << 52));
}

// kc of a cell for the face means: exp(logK / 2) (geometric) or exp(logK) (harmonic), once per cell
__device__ __forceinline__ double cell_k(double logK, int kind) {
    return kind == DPF_MEAN_GEOMETRIC ? exp64<true>(logK) : exp64<false>(logK);
}

// num / den for 0 <= num <= 2^240 and positive den, correctly rounded but for rare ties' neighbours: a Newton
// step on a float reciprocal (error 2^-44), then Markstein's correction of the quotient by its exact remainder
// (P. Markstein, IBM J. Res. Dev. 34, 1990). Five FP64 instructions. den outside 2^+-120 or num below 2^-900
// take the division.
__device__ __forceinline__ double div64(double num, double den) {
    const unsigned en = (unsigned)(__double2hiint(num) >> 20), ed = (unsigned)(__double2hiint(den) >> 20);
    if (ed - 903u > 240u || en - 123u > 1140u) return num / den;
    const double r0 = (double)__fdividef(1.0f, (float)den);
    const double r = fma(fma(-den, r0, 1.0), r0, r0);
    const double q = num * r;
    return fma(fma(-den, q, num), r, q);
}

// 1 / p for a positive p: the reciprocal of p's significand from a float division, then one
// third-order Householder step r (1 + e + e^2), e = 1 - m r (|e| < 2^-22, so its error is below
// 2^-66 before rounding). Three FP64 instructions in a chain that a column's or a pivot's threads wait for; the
// division the compiler emits has about ten, 70 clocks each from a single warp. Exponents outside
// +-500 (and zero, infinity, NaN) take the division.
__device__ __forceinline__ double recip(double p) {
    const long long u = __double_as_longlong(p);
    const int ex = (int)((u >> 52) & 0x7FF);
    if (ex < 523 || ex > 1523) return 1.0 / p;
    const double m = __longlong_as_double((u & 0xFFFFFFFFFFFFFll) | 0x3FF0000000000000ll);
    const double r = (double)(1.0f / (float)m);
    const double e = fma(-m, r, 1.0);
    const double q = fma(r, fma(e, e, e), r);
    return __longlong_as_double(__double_as_longlong(q) + ((long long)(1023 - ex) << 52));
}

// Face conductances from the cell values kc:
//   geometric  kc = exp(logK / 2):  K_f = exp((logK_a + logK_b)/2) = kc_a kc_b
//   harmonic   kc = exp(logK):      K_f = 2 / (1/K_a + 1/K_b) = 2 kc_a kc_b / (kc_a + kc_b)
// (harmonic as twice the smaller value times a quotient in [1/2, 1]: the product kc_a kc_b could overflow; the
// same for both orders; the values are not negative, so their bits order them)
__device__ __forceinline__ double face_mean_k(double ka, double kb, int kind) {
    if (kind == DPF_MEAN_GEOMETRIC) return ka * kb;
    const long long ia = __double_as_longlong(ka), ib = __double_as_longlong(kb);
    const double lo = __longlong_as_double(ia < ib ? ia : ib), hi = __longlong_as_double(ia < ib ? ib : ia);
    return lo * (2.0 * div64(hi, ka + kb));
}

// dK_f / dlogK_a = dlogk_scale(ka) dlogk_weight(ka, kb), the scale applied once per cell, to the sum over its faces.
//   geometric  K_f / 2: the weight is kb times ka's power of two, the scale half its significand, so that the weight is
//              within a factor of two of K_f: kb alone times dK_f overflows or vanishes for cells hundreds of e-folds
//              apart. Integer additions to the exponent; the FP64 instructions are those of kb alone.
//   harmonic   K_f^2 / (2 ka) = 2 (ka t) t with t = kb / (ka + kb), in this order since t^2 could underflow
__device__ __forceinline__ bool normal_exponent(int e) { return (unsigned)(e - 1) < 2046u; }
__device__ __forceinline__ double dlogk_weight(double ka, double kb, int kind) {
    if (kind == DPF_MEAN_GEOMETRIC) {
        const int ea = __double2hiint(ka) >> 20, eb = __double2hiint(kb) >> 20;
        if (normal_exponent(ea) && normal_exponent(eb) && normal_exponent(ea + eb - 1023))
            return __longlong_as_double(__double_as_longlong(kb) + ((long long)(ea - 1023) << 52));
        return (normal_exponent(ea) ? __longlong_as_double((long long)ea << 52) : ka) * kb;
    }
    const double t = div64(kb, ka + kb);
    return ka * t * t;
}
__device__ __forceinline__ double dlogk_scale(double ka, int kind) {
    if (kind != DPF_MEAN_GEOMETRIC) return 2.0;
    const long long u = __double_as_longlong(ka);
    return normal_exponent((int)(u >> 52)) ? __longlong_as_double((u & 0xFFFFFFFFFFFFFll) | 0x3FE0000000000000ll) : 0.5;
}

}  // namespace dpf
