// FP64 exponential and quotient with few FP64-pipe operations.
//
// The HH rates are six exponentials and three quotients per compartment, and GB300's FP64 pipe
// takes 16 cycles per warp instruction (2 lanes per clock per SM), so their count of FP64
// operations sets the time of every FP64 kernel here.  Both functions do what FP32 and integer
// arithmetic can do exactly or to more than enough digits there, and only the rest in FP64:
//   exp64: table-driven reduction after Tang (ACM TOMS 15, 1989), x = k ln2/512 + r with
//     |r| < 0.00068, e^x = 2^(k/512) (1 + r + r^2 (1/2 + r/6 + r^2/24)).  The bracket after the
//     1/2 is below 1.2e-4 and is multiplied by r^2 < 4.6e-7, so evaluating it in FP32 costs
//     less than 1e-17 of the result.  9 FP64 operations.
//   div64: Newton's iteration from an FP32 reciprocal and a residual correction of the quotient
//     (Markstein, IBM J. R&D 34, 1990).  5 FP64 operations.
// Against 80-bit arithmetic over 4e7 arguments exp64 is within 0.56 ulp and div64 correctly
// rounded, no further off than CUDA's own exp (1 ulp) and division.  Arguments outside the short path
// (overflow, underflow, zero divisors, infinities, NaN) go to CUDA's functions.
#pragma once
#include "cvt.cuh"

namespace nrt {

// 2^(j/512) and what its rounding left over.
static __device__ const double2 kExp2Frac[512] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.0058c86da1c0ap+0, -0x1.5e00e62d6b30dp-56},
    {0x1.00b1afa5abcbfp+0, -0x1.4f6b2a7609f71p-55}, {0x1.010ab5b2cbd11p+0, 0x1.c1d0660524e08p-54},
    {0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54}, {0x1.01bd1e77170b4p+0, 0x1.5e7626621eb5bp-56},
    {0x1.02168143b0281p+0, -0x1.2bf310fc54eb6p-55}, {0x1.027003103b10ep+0, -0x1.082ef51b61d7ep-56},
    {0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56}, {0x1.032363d42b027p+0, 0x1.fea8d61ed6016p-54},
    {0x1.037d42e11bbccp+0, 0x1.56811eeade11ap-57}, {0x1.03d7411915a8ap+0, 0x1.b7c00e7b751dap-54},
    {0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54}, {0x1.048b9b35659d8p+0, 0x1.21cd53d5e8b66p-57},
    {0x1.04e5f72f654b1p+0, 0x1.4c3793aa0d08dp-55}, {0x1.0540727fc1762p+0, -0x1.abcae24b819dfp-54},
    {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55}, {0x1.05f5c74f0bec2p+0, 0x1.996d5009d00dep-54},
    {0x1.0650a0e3c1f89p+0, -0x1.5cb7b5799c397p-54}, {0x1.06ab99fa6407cp+0, -0x1.a5e905f7c7ebep-55},
    {0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55}, {0x1.0761ead925493p+0, -0x1.d856655af086ap-55},
    {0x1.07bd42b72a836p+0, 0x1.3233454458700p-55}, {0x1.0818ba42e7d30p+0, -0x1.ba46408f85fd6p-54},
    {0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57}, {0x1.08d0088f8093fp+0, 0x1.dd1f1d8a47bbcp-58},
    {0x1.092bdf66607e0p+0, -0x1.68063800a3fd1p-54}, {0x1.0987d61701716p+0, -0x1.d05b3e26abfd6p-55},
    {0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54}, {0x1.0a402331b9715p+0, 0x1.c01f59d7db7cfp-55},
    {0x1.0a9c79b1f3919p+0, 0x1.5d16c873d1d38p-55}, {0x1.0af8f03834e52p+0, 0x1.bb2180f5f5219p-54},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.0bb23d833d93fp+0, -0x1.6b8089b07909fp-55},
    {0x1.0c0f145e46c85p+0, 0x1.4f98906d21cefp-54}, {0x1.0c6c0b6bdae53p+0, -0x1.4e8a80969d886p-54},
    {0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54}, {0x1.0d265a4b520bap+0, -0x1.db361584e6300p-54},
    {0x1.0d83b23395decp+0, -0x1.bc14de43f316ap-54}, {0x1.0de12a7b26300p+0, 0x1.e181a9425ebcbp-54},
    {0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59}, {0x1.0e9c7c55189c6p+0, 0x1.3140927decdabp-55},
    {0x1.0efa55fdfa9c5p+0, -0x1.49db9bc54021bp-54}, {0x1.0f58503328e6dp+0, -0x1.6058ab1a46f1ap-55},
    {0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57}, {0x1.1014a66f951cep+0, 0x1.7bef21c9dea63p-55},
    {0x1.1073028d7233ep+0, 0x1.d46eb1692fdd5p-55}, {0x1.10d17f64d9ef1p+0, 0x1.431762073e535p-57},
    {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54}, {0x1.118edb6db2dc1p+0, -0x1.ce5fc87c4dd8ep-57},
    {0x1.11edbab5e2ab6p+0, -0x1.ca454f703fb72p-54}, {0x1.124cbae51a5c8p+0, -0x1.512b949cc76f8p-54},
    {0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58}, {0x1.130b1e264a0e9p+0, -0x1.a70f11e89fb52p-54},
    {0x1.136a814f204abp+0, -0x1.7108fba48dcf0p-57}, {0x1.13ca058cbae1ep+0, -0x1.43684aabe72bdp-56},
    {0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54}, {0x1.1489717425438p+0, -0x1.01720e2fc037dp-56},
    {0x1.14e95934f312ep+0, -0x1.b91e839bf44abp-55}, {0x1.154962388149ep+0, 0x1.821afe3f2bf25p-59},
    {0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55}, {0x1.1609d83606e12p+0, -0x1.8105d66c7d0ccp-54},
    {0x1.166a45471c3c2p+0, 0x1.8f23b82ea1a32p-58}, {0x1.16cad3c92df73p+0, 0x1.0c17504ffdddfp-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.178c554eaea89p+0, 0x1.00be0ed2710c9p-54},
    {0x1.17ed48695bbc0p+0, 0x1.09e3fe2ac5a64p-56}, {0x1.184e5d23816c9p+0, -0x1.f62a4b061b797p-54},
    {0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54}, {0x1.1910eba4df41fp+0, 0x1.e94c19df12feep-55},
    {0x1.1972658375d2fp+0, 0x1.4aadd85f17e08p-54}, {0x1.19d4013041dc2p+0, -0x1.d020f4d703c9fp-54},
    {0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55}, {0x1.1a979e2363cf8p+0, 0x1.23a7a004a48aep-58},
    {0x1.1af99f8138a1cp+0, 0x1.7bf85a4b69280p-54}, {0x1.1b5bc2dc40bf0p+0, 0x1.d8392ae90ce4ep-55},
    {0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54}, {0x1.1c206fb91588fp+0, 0x1.d338944c9a0e8p-55},
    {0x1.1c82f95281c6bp+0, 0x1.009778010f8c9p-54}, {0x1.1ce5a51860746p+0, -0x1.ad03a21404840p-57},
    {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54}, {0x1.1dab6358e15e8p+0, -0x1.8b44056589d61p-54},
    {0x1.1e0e75eb44027p+0, -0x1.6fdd8088cb6dep-54}, {0x1.1e71aad999e82p+0, 0x1.a63f5c1b1dd1fp-56},
    {0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54}, {0x1.1f387bf9cda38p+0, 0x1.1e4b090a54f7dp-54},
    {0x1.1f9c18438ce4dp+0, -0x1.bf524a097af5cp-54}, {0x1.1fffd7190241ep+0, 0x1.42a3cf9a6e318p-54},
    {0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55}, {0x1.20c7bc96ffc18p+0, -0x1.1130fe76aad5cp-59},
    {0x1.212be3578a819p+0, 0x1.3592d2cfcaac9p-54}, {0x1.21902cd3d09b9p+0, -0x1.d6583a1ed89bdp-61},
    {0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55}, {0x1.2259282fc1f27p+0, 0x1.b283a7a9a2022p-55},
    {0x1.22bdda27912d1p+0, 0x1.d34fb5577d69fp-55}, {0x1.2322af0b63bffp+0, 0x1.487fd27e5a7b2p-59},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.23ecc1c78903ap+0, -0x1.cdd7a05f66fd8p-54},
    {0x1.2451ffb82140ap+0, 0x1.acfcc911ca996p-55}, {0x1.24b760c547f15p+0, 0x1.68f656fed356ep-56},
    {0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55}, {0x1.25828c65fa1ffp+0, 0x1.447d93c478783p-54},
    {0x1.25e85711ece75p+0, 0x1.3e1a24ac31b2cp-54}, {0x1.264e450b3cb82p+0, -0x1.2a34ff432e733p-54},
    {0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55}, {0x1.271a8b16f0a30p+0, -0x1.88846a8172bc5p-56},
    {0x1.2780e341ddf29p+0, 0x1.e067c05f9e76cp-54}, {0x1.27e75eeb3ab98p+0, 0x1.05117e5c88fb1p-55},
    {0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54}, {0x1.28b4c0ea83f36p+0, -0x1.6c190554e071ap-54},
    {0x1.291ba7591bb70p+0, -0x1.2cc7228401cbdp-55}, {0x1.2982b17779965p+0, 0x1.0f41c1ae6b7b2p-54},
    {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55}, {0x1.2a5130f50d65cp+0, -0x1.a7281af95a0a4p-56},
    {0x1.2ab8a66d10f13p+0, -0x1.95743191690a7p-54}, {0x1.2b203fc675d1fp+0, 0x1.3fc477099b71ap-55},
    {0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59}, {0x1.2befde4f2e280p+0, 0x1.4e5c6fb4ca905p-57},
    {0x1.2c57e39771b2fp+0, -0x1.50145a6eb5124p-54}, {0x1.2cc00cf2f6c18p+0, -0x1.51cc74f1651e2p-54},
    {0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54}, {0x1.2d90cc15d5346p+0, 0x1.9676bdb1b6915p-56},
    {0x1.2df961f641589p+0, 0x1.d16cffbbce198p-54}, {0x1.2e621c1c14833p+0, 0x1.b28aedee223bcp-55},
    {0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56}, {0x1.2f33fd6a454d2p+0, -0x1.33b50add83bc9p-54},
    {0x1.2f9d24abd886bp+0, -0x1.53c55532bda93p-57}, {0x1.300670653dfe4p+0, 0x1.02bf2a6597e23p-55},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.30d975721b004p+0, 0x1.8b02cef625aa4p-56},
    {0x1.31432edeeb2fdp+0, 0x1.959a3f3f3fcd1p-55}, {0x1.31ad0cf63eeacp+0, -0x1.edae36238f255p-54},
    {0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55}, {0x1.3281375752b40p+0, -0x1.854137c374413p-58},
    {0x1.32eb83ba8ea32p+0, -0x1.c45e83cb4f318p-54}, {0x1.3355f4fb45e20p+0, 0x1.c3f8de75651c2p-55},
    {0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54}, {0x1.342b46484ebb4p+0, -0x1.d8deede0553fdp-55},
    {0x1.3496266e3fa2dp+0, -0x1.35a75930881a4p-55}, {0x1.35012ba4ea77dp+0, -0x1.731012edb1079p-54},
    {0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55}, {0x1.35d7a577dd72bp+0, 0x1.9ad8b9afdb485p-55},
    {0x1.36431a2de883bp+0, -0x1.c3144a06cb85ep-55}, {0x1.36aeb428335b4p+0, 0x1.7e20a76092403p-55},
    {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54}, {0x1.3786581d3f669p+0, -0x1.7849f7db479d2p-55},
    {0x1.37f26231e754ap+0, -0x1.9f5ca9eceb23cp-54}, {0x1.385e91be9c811p+0, 0x1.68effa66ed3d2p-56},
    {0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54}, {0x1.393761742d808p+0, 0x1.bd89f516d2f1dp-55},
    {0x1.39a401b7140efp+0, -0x1.9a9a5fc8e2934p-54}, {0x1.3a10c7a61d55bp+0, 0x1.e218b6b52d59ep-55},
    {0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56}, {0x1.3aeac4bcdf3eap+0, -0x1.fc8195f57f1d7p-55},
    {0x1.3b57fbfec6cf4p+0, 0x1.54c66e26fff18p-54}, {0x1.3bc559212ef89p+0, -0x1.c069167914572p-56},
    {0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54}, {0x1.3ca0853c10f28p+0, 0x1.9b612c9a97edcp-54},
    {0x1.3d0e544ede173p+0, 0x1.fe8d08c284c71p-56}, {0x1.3d7c4976d27fap+0, -0x1.6a8b6efe6c152p-57},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.3e58a63b0a09bp+0, -0x1.7e0252b7a548ap-54},
    {0x1.3ec70df1c5175p+0, -0x1.af6637b8c9bcap-55}, {0x1.3f359bf29743fp+0, -0x1.b6502050c36aap-54},
    {0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54}, {0x1.40132b07a35dfp+0, -0x1.76a483355fa84p-56},
    {0x1.40822c367a024p+0, 0x1.bddf8b6f4d048p-55}, {0x1.40f153e4a136ap+0, -0x1.976147d73afd4p-55},
    {0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58}, {0x1.41d016f44d8f5p+0, -0x1.edd01519b2f84p-55},
    {0x1.423fb2709468ap+0, -0x1.8462dc0b314ddp-54}, {0x1.42af74a1af3f1p+0, 0x1.391233bcfaea7p-55},
    {0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55}, {0x1.438f6d5817663p+0, -0x1.5f4a55726d308p-57},
    {0x1.43ffa3f84b9d4p+0, 0x1.880be9704c003p-55}, {0x1.4470018321a1ap+0, -0x1.1db72ba02c9f7p-54},
    {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59}, {0x1.4551318eb43ecp+0, -0x1.c6c6a45fd2998p-55},
    {0x1.45c2042a7d232p+0, -0x1.8641982fb1f8ep-57}, {0x1.4632fde7006f4p+0, -0x1.35fc2fa6ed511p-54},
    {0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54}, {0x1.471566f8827d0p+0, -0x1.f88fcd7beb2f5p-59},
    {0x1.4786d668b3237p+0, -0x1.c20f0ed445733p-54}, {0x1.47f86d3001fe5p+0, 0x1.31d56d5833416p-57},
    {0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56}, {0x1.48dc10fa920a1p+0, 0x1.71f91caab9615p-54},
    {0x1.494e1e192aed2p+0, -0x1.3b2895e499ea0p-55}, {0x1.49c052c5916c4p+0, 0x1.beb7d6865bab2p-57},
    {0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54}, {0x1.4aa532feaada6p+0, -0x1.be0fe368141a0p-54},
    {0x1.4b17dea6db7d7p+0, -0x1.125b87f2897f0p-55}, {0x1.4b8ab213d5283p+0, -0x1.1a553a430a16cp-54},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.4c70d073537cap+0, 0x1.37586fcd9083ap-56},
    {0x1.4ce41b817c114p+0, 0x1.05e29690abd5dp-54}, {0x1.4d578e8bb586bp+0, 0x1.efb0d287c6e23p-54},
    {0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54}, {0x1.4e3eeccbd7b2ap+0, 0x1.89a81e193b611p-57},
    {0x1.4eb2d81d8abffp+0, -0x1.5257d2e5d7a52p-54}, {0x1.4f26eba2e35f0p+0, 0x1.470a97853189bp-54},
    {0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54}, {0x1.500f8b804f127p+0, -0x1.5ef3f782a2391p-55},
    {0x1.508417f4531eep+0, 0x1.a249b49b7465fp-56}, {0x1.50f8ccd3deb0dp+0, -0x1.1f895f0e2f60fp-56},
    {0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55}, {0x1.51e2b00da3b14p+0, -0x1.09dc978c2d695p-57},
    {0x1.5257de83f4eefp+0, -0x1.c998d43efef71p-56}, {0x1.52cd359dfd53dp+0, -0x1.cec6446cbd1a3p-55},
    {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55}, {0x1.53b85df598d78p+0, -0x1.fe83ad1154a1ap-54},
    {0x1.542e2f4f6ad27p+0, 0x1.7926d192d5f7ep-55}, {0x1.54a4298571b06p+0, -0x1.a08b582efaca3p-55},
    {0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55}, {0x1.559098bed1bdfp+0, 0x1.4bccce5904465p-54},
    {0x1.56070dde910d2p+0, -0x1.0fb6e168eebf0p-54}, {0x1.567dac1351819p+0, -0x1.6cc9b92f9338dp-54},
    {0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54}, {0x1.576b63f4d854cp+0, 0x1.cd4fad1261866p-54},
    {0x1.57e27dbe2c4cfp+0, -0x1.0b98c8a57b9c4p-54}, {0x1.5859c0d59ca07p+0, 0x1.70f80f6d151b8p-55},
    {0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55}, {0x1.5948c32824135p+0, -0x1.34e9078187b25p-59},
    {0x1.59c0827ff07ccp+0, -0x1.7e2cee467e60fp-54}, {0x1.5a386b5f43d92p+0, 0x1.f6069380b8d75p-56},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.5b28b9ee20d1ep+0, -0x1.687aca30682a8p-54},
    {0x1.5ba11fba87a03p+0, -0x1.b77a14c233e1ap-54}, {0x1.5c19af482fc8fp+0, -0x1.8e5770aa82b0ep-54},
    {0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60}, {0x1.5d0b4be135accp+0, -0x1.b8ded2fcd487ap-54},
    {0x1.5d84590998b93p+0, -0x1.cd6a7a8b45643p-54}, {0x1.5dfd902d47c65p+0, -0x1.d4927bc94f4ccp-54},
    {0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54}, {0x1.5ef07ca0cbf0fp+0, 0x1.7b7b016f3ade2p-54},
    {0x1.5f6a320dceb71p+0, -0x1.9eadde3cdcf92p-55}, {0x1.5fe411b078d26p+0, 0x1.fc4c5337e4394p-54},
    {0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54}, {0x1.60d84fd15612ap+0, 0x1.5baf387937330p-55},
    {0x1.6152ae6cdf6f4p+0, 0x1.e4b3e4ab84c27p-54}, {0x1.61cd3778bc944p+0, 0x1.63633ea778bf9p-56},
    {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54}, {0x1.62c2c91c56acdp+0, 0x1.de5927c1708a2p-54},
    {0x1.633dd1d1929fdp+0, 0x1.84710beb964e5p-54}, {0x1.63b90532205d8p+0, -0x1.b04ea96997c15p-54},
    {0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55}, {0x1.64afec30678b7p+0, -0x1.2a2f3bd4177d3p-54},
    {0x1.652b9febc8fb7p+0, -0x1.ae3d5c9a73e09p-54}, {0x1.65a77e8dcc390p+0, -0x1.91671c41cc2bdp-54},
    {0x1.6623882552225p+0, -0x1.bb60987591c34p-54}, {0x1.669fbcc140be7p+0, 0x1.872063cf6798fp-54},
    {0x1.671c1c70833f6p+0, -0x1.e8732586c6134p-55}, {0x1.6798a7420a036p+0, -0x1.0c928caabd378p-55},
    {0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57}, {0x1.68923e87bfb7ap+0, 0x1.f6854973b742cp-54},
    {0x1.690f4b19e9538p+0, 0x1.804bd9aeb445dp-55}, {0x1.698c830a4c8d4p+0, -0x1.a24fd076a2899p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.6a877541ee718p+0, 0x1.11dd76fdd6672p-54},
    {0x1.6b052fa75173ep+0, 0x1.a38f52c9a9d0ep-56}, {0x1.6b8315a736c75p+0, -0x1.35f1acc6972ebp-54},
    {0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56}, {0x1.6c7f64b30aa09p+0, -0x1.6453f83de632ap-58},
    {0x1.6cfdcddd47645p+0, 0x1.c7aa9b6f17309p-54}, {0x1.6d7c62dea2f8ap+0, 0x1.e624bfec2908fp-54},
    {0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57}, {0x1.6e7a10a38cee8p+0, -0x1.4022c7d2819e1p-54},
    {0x1.6ef9298593ae5p+0, -0x1.0b9749e1ac8b2p-54}, {0x1.6f786e7ba9fefp+0, -0x1.6886a4d66bc2ep-54},
    {0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55}, {0x1.70777ce1303f6p+0, -0x1.370766994643fp-55},
    {0x1.70f7466f42e87p+0, 0x1.9d644d45aa65fp-58}, {0x1.71773c4eaa988p+0, -0x1.2a825be6cfe24p-54},
    {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55}, {0x1.7277ad3ef9011p+0, -0x1.9f65bb8417329p-54},
    {0x1.72f8286ead08ap+0, -0x1.20aa02cd62c72p-54}, {0x1.7378d02d50b8fp+0, 0x1.8b41ecebff89fp-54},
    {0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54}, {0x1.747aa5953c849p+0, -0x1.8f873623619b2p-54},
    {0x1.74fbd35d7cbfdp+0, 0x1.047fd618a6e1cp-54}, {0x1.757d2df29ce7cp+0, 0x1.19527ae80ec89p-55},
    {0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54}, {0x1.768069c1a861dp+0, 0x1.d62703a28cf99p-54},
    {0x1.77024b1ab6e09p+0, 0x1.b7877169147f8p-54}, {0x1.7784597eeba8fp+0, -0x1.d6763647d9ca2p-54},
    {0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54}, {0x1.7888fda749e5dp+0, 0x1.110a476eb9526p-54},
    {0x1.790b938ac1cf6p+0, 0x1.349a862aadd3ep-54}, {0x1.798e56b7fcf03p+0, 0x1.ee11e10ef0644p-54},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.7a94652e958aap+0, -0x1.73ce2886ce405p-54},
    {0x1.7b17b0976cfdbp+0, -0x1.bebb58468dc88p-54}, {0x1.7b9b2988fb9ecp+0, 0x1.25e05bb469b48p-57},
    {0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54}, {0x1.7ca2a4456e7a3p+0, -0x1.25c3a2377fadbp-54},
    {0x1.7d26a62ff86f0p+0, 0x1.1bddbfb72b8b4p-54}, {0x1.7daad5e2850acp+0, -0x1.33a50c0ce4ba0p-56},
    {0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56}, {0x1.7eb3bedf2e1b9p+0, 0x1.1a92fd166cab9p-54},
    {0x1.7f3878491c491p+0, -0x1.07f11cf9311aep-55}, {0x1.7fbd5fbab091fp+0, 0x1.efa4a3a96ff7fp-54},
    {0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54}, {0x1.80c7b8f4abaa9p+0, -0x1.ae7c35d63d803p-55},
    {0x1.814d2add106d9p+0, 0x1.464370d151d4dp-54}, {0x1.81d2cb0d1736ap+0, 0x1.422251b07b086p-58},
    {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54}, {0x1.82de968443d9ap+0, 0x1.3bc166320d9ccp-54},
    {0x1.8364c1eb941f7p+0, 0x1.99b9a31df2bd5p-54}, {0x1.83eb1bdadb46dp+0, 0x1.f48b2f8c93e44p-54},
    {0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55}, {0x1.84f85b91e07f1p+0, 0x1.40292415699dap-55},
    {0x1.857f4179f5b21p+0, -0x1.ba748f8b216d0p-58}, {0x1.8606562ab00ecp+0, 0x1.a8521803ef3cap-54},
    {0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54}, {0x1.87150c27004c2p+0, 0x1.3cbb932ba1d2ep-54},
    {0x1.879cad931a436p+0, 0x1.5d2d7d2db47bdp-55}, {0x1.88247e08e1957p+0, -0x1.3d58ca4ad8933p-57},
    {0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54}, {0x1.8934ac52be8f7p+0, 0x1.98181a63ad2a8p-54},
    {0x1.89bd0a478580fp+0, 0x1.d53954475202bp-54}, {0x1.8a4597875c644p+0, 0x1.a508d46fb2c1dp-56},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.8b574029db01ep+0, 0x1.1709939065e99p-54},
    {0x1.8be05bad61778p+0, 0x1.ecb5efc43446ep-54}, {0x1.8c69a6bdb5598p+0, -0x1.816caef5dfec0p-55},
    {0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56}, {0x1.8d7ccbc6c19e6p+0, 0x1.adaa8b3e778e2p-57},
    {0x1.8e06a5e0866d9p+0, -0x1.7114a6fc9b2e6p-54}, {0x1.8e90afc931857p+0, 0x1.ba4c54c1b1faap-55},
    {0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55}, {0x1.8fa553499284bp+0, -0x1.815b6ec103d0cp-54},
    {0x1.902fed0282c8ap+0, 0x1.592ca85fe3fd2p-54}, {0x1.90bab6ccce12cp+0, -0x1.5a36b1812f7afp-54},
    {0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54}, {0x1.91d0dad829e70p+0, -0x1.f5e0d8cd2f3bcp-54},
    {0x1.925c353aa2fe2p+0, -0x1.3455fa639db7fp-55}, {0x1.92e7bff148396p+0, -0x1.72d01639e7220p-54},
    {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57}, {0x1.93ff669e2802bp+0, 0x1.53b769dad8e6ep-56},
    {0x1.948b82b5f98e5p+0, -0x1.dc3d6797d2d99p-55}, {0x1.9517cf65253d1p+0, -0x1.f5d0450666694p-54},
    {0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56}, {0x1.9630faccf9243p+0, 0x1.0bec0c0f91530p-56},
    {0x1.96bdd9a7670b3p+0, -0x1.ba5967f19c896p-58}, {0x1.974ae95cba768p+0, 0x1.02e9ebb071962p-57},
    {0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54}, {0x1.98659b9bddb5bp+0, 0x1.279adf9fd115bp-54},
    {0x1.98f33e47a22a2p+0, 0x1.cabdaa24c78edp-56}, {0x1.9981121235681p+0, -0x1.a180aa7583e5ep-54},
    {0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54}, {0x1.9a9d4d47f2598p+0, -0x1.4d609893222adp-54},
    {0x1.9b2bb4d53fe0dp+0, -0x1.dd84e4df6d518p-54}, {0x1.9bba4dc5a3dd3p+0, 0x1.66c912c5f1786p-55},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.9cd81414380f2p+0, 0x1.a6bd173ec7862p-54},
    {0x1.9d674194bb8d5p+0, -0x1.516bea3dd8233p-54}, {0x1.9df6a0bcfc15ep+0, 0x1.4bcb245c8e7c9p-64},
    {0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56}, {0x1.9f15f4499c647p+0, 0x1.432f731487969p-54},
    {0x1.9fa5e8d07f29ep+0, -0x1.4a9ceaaf1facep-55}, {0x1.a0360f4424fcbp+0, -0x1.548de0c885750p-55},
    {0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54}, {0x1.a156f23701b15p+0, 0x1.4ffcb1c953fd2p-54},
    {0x1.a1e7aed8eb8bbp+0, 0x1.c6618ee8be70ep-54}, {0x1.a2789dacfe68cp+0, -0x1.9e2f2608ff33fp-57},
    {0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54}, {0x1.a39b1231475f7p+0, 0x1.8360ad75bf0e9p-55},
    {0x1.a42c980460ad8p+0, -0x1.aa780589fb120p-54}, {0x1.a4be504f696b1p+0, -0x1.0e534b216c6a8p-54},
    {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54}, {0x1.a5e25893523d4p+0, 0x1.ddc8ca9dffa72p-55},
    {0x1.a674a8af46052p+0, 0x1.50f5630670366p-57}, {0x1.a7072b8950a73p+0, -0x1.c6cd81ecd5c5ep-57},
    {0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54}, {0x1.a82cc9be14dcap+0, 0x1.5778678031c65p-54},
    {0x1.a8bfe53c12e59p+0, -0x1.4f867b2ba15a9p-54}, {0x1.a95333beb0b7ep+0, -0x1.ad46b150cf4fap-54},
    {0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54}, {0x1.aa7a6a1897fd2p+0, 0x1.725ec3c304e53p-61},
    {0x1.ab0e521356ebap+0, 0x1.89c31dae94545p-55}, {0x1.aba26d59a09eep+0, 0x1.cd1ec41e524a9p-54},
    {0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55}, {0x1.accb3e100301ep+0, -0x1.7f505bf57ecf5p-54},
    {0x1.ad5ff3a3c2774p+0, 0x1.7ef3bb6b1b8e5p-54}, {0x1.adf4dcca5a413p+0, 0x1.791fa997ef90fp-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.af1f4a17a4735p+0, -0x1.915f95760eb2fp-56},
    {0x1.afb4ce622f2ffp+0, -0x1.4b2fc0f315ecdp-54}, {0x1.b04a868742ee4p+0, 0x1.c1a01c43d2693p-57},
    {0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54}, {0x1.b17692a8fa8cdp+0, 0x1.d63160ee10297p-54},
    {0x1.b20ce6c9a8952p+0, 0x1.4dd024a0756ccp-54}, {0x1.b2a36f0cf3f3ap+0, -0x1.0a8720b3e06bdp-54},
    {0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57}, {0x1.b3d11c43bbd62p+0, -0x1.3467d87ff2174p-54},
    {0x1.b468415b749b1p+0, -0x1.f763de9df7c90p-56}, {0x1.b4ff9ade433c6p+0, -0x1.fa2f8e36fef82p-54},
    {0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54}, {0x1.b62eeb6ddfc87p+0, -0x1.9f7c84a9a3b9fp-56},
    {0x1.b6c6e29f1c52ap+0, 0x1.2a8f352883f6ep-54}, {0x1.b75f0e844bfc6p+0, 0x1.a1b9e0bd95b2ap-54},
    {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56}, {0x1.b89004b3a7804p+0, -0x1.90c333ffb24afp-54},
    {0x1.b928cf22749e4p+0, -0x1.b721654cb65c6p-54}, {0x1.b9c1ce8e77680p+0, 0x1.a3307ae543910p-54},
    {0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54}, {0x1.baf46ca7a67a7p+0, 0x1.8d19c3ebe1ea1p-54},
    {0x1.bb8e0b79a6f1fp+0, -0x1.f52d1c9696205p-60}, {0x1.bc27df9285775p+0, 0x1.6f58bca6ba32bp-55},
    {0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55}, {0x1.bd5c27e2cb5e5p+0, -0x1.25c5473ec3e56p-56},
    {0x1.bdf69c3f3a207p+0, -0x1.c262360ea5b52p-60}, {0x1.be91462c95b60p+0, -0x1.879e57f67afecp-55},
    {0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54}, {0x1.bfc73b0468d30p+0, -0x1.7fc2bd9bc7402p-54},
    {0x1.c06286141b33dp+0, -0x1.d8a5aa1fbca34p-55}, {0x1.c0fe06ff301f4p+0, 0x1.ff2f06da8099ap-54},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.c235aab23e61ep+0, -0x1.64601deb2b32cp-54},
    {0x1.c2d1cd9fa652cp+0, -0x1.6e51617c8a5d7p-54}, {0x1.c36e26b34e065p+0, 0x1.29e63e337f8a9p-54},
    {0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54}, {0x1.c4a77b9881650p+0, -0x1.915ef6cdef8d0p-54},
    {0x1.c544778fafb22p+0, 0x1.12f072493b5afp-54}, {0x1.c5e1a9f8630adp+0, -0x1.9caa2e00697a7p-56},
    {0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54}, {0x1.c71cb269e601fp+0, -0x1.7f6ecb95815f0p-55},
    {0x1.c7ba88988c933p+0, -0x1.e76bbbe255559p-55}, {0x1.c8589584661a1p+0, -0x1.0f3af432cdc42p-54},
    {0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56}, {0x1.c99553dfa8313p+0, 0x1.4b0255f572675p-54},
    {0x1.ca3405751c4dbp+0, -0x1.7f2bed10d08f5p-55}, {0x1.cad2ee13da7cbp+0, 0x1.87d521ba089f4p-55},
    {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56}, {0x1.cc1164b994d23p+0, -0x1.e9ffb7156580ap-55},
    {0x1.ccb0f2e6d1675p+0, -0x1.d220f86009093p-56}, {0x1.cd50b869d8f0fp+0, 0x1.20abfc58a6591p-54},
    {0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55}, {0x1.ce90e9be12cb9p+0, 0x1.2a13fc0b63e9fp-57},
    {0x1.cf3155b5bab74p+0, -0x1.a08e9b86dff57p-54}, {0x1.cfd1f95018d17p+0, -0x1.166c435088969p-54},
    {0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54}, {0x1.d113e7ba2c38cp+0, 0x1.2785752b6f21bp-56},
    {0x1.d1b532b08c968p+0, 0x1.55636219a36eep-54}, {0x1.d256b596f948cp+0, -0x1.a3e4ea3b2f7a4p-54},
    {0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54}, {0x1.d39a638197a3cp+0, -0x1.85b78c128cd7ep-54},
    {0x1.d43c8eacaa1d6p+0, 0x1.3db53bf5a1614p-54}, {0x1.d4def2158a91fp+0, -0x1.cdf2e68e10b59p-54},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.d62461eec14bep+0, 0x1.223aa2bd32658p-54},
    {0x1.d6c76e862e6d3p+0, 0x1.fe87a4a8165a0p-58}, {0x1.d76ab3a99745bp+0, -0x1.84b279b977de0p-57},
    {0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54}, {0x1.d8b1e7e2d479dp+0, -0x1.0ecc71e1dd728p-55},
    {0x1.d955d71ff6075p+0, 0x1.a052dbb9af6bep-54}, {0x1.d9f9ff37adb4ap+0, -0x1.0b22123ad1988p-54},
    {0x1.da9e603db3285p+0, 0x1.c2300696db532p-54}, {0x1.db42fa45c4dfdp+0, 0x1.464497a1b4103p-55},
    {0x1.dbe7cd63a8315p+0, -0x1.b76f1926b8be4p-54}, {0x1.dc8cd9ab294e4p+0, 0x1.751d3390c4ab9p-54},
    {0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54}, {0x1.ddd79e065807dp+0, 0x1.1e846990935d0p-54},
    {0x1.de7d5641c0658p+0, -0x1.ca5528e79ba8fp-54}, {0x1.df2347f63c159p+0, -0x1.1cb486bfb8ea4p-55},
    {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54}, {0x1.e06fd81a2ece1p+0, -0x1.0d77a4789fc84p-54},
    {0x1.e11676b197d17p+0, -0x1.2b529bd5c7f44p-56}, {0x1.e1bd4f11f8220p+0, 0x1.53855b6c7ee95p-55},
    {0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54}, {0x1.e30bad7dcee90p+0, 0x1.4036d1ded17acp-54},
    {0x1.e3b333b16ee12p+0, -0x1.9f4a431fdc68bp-54}, {0x1.e45af3fe592e8p+0, -0x1.2623713eaad2ep-55},
    {0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55}, {0x1.e5ab2334ac7eep+0, -0x1.06b148ae42258p-56},
    {0x1.e653924676d76p+0, -0x1.63ff87522b735p-55}, {0x1.e6fc3bc24e350p+0, 0x1.c80ff0defb85bp-54},
    {0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54}, {0x1.e84e3e4933c7ep+0, -0x1.41295a3f6ff00p-54},
    {0x1.e8f7977cdb740p+0, -0x1.1089480b054b1p-54}, {0x1.e9a12b6bc3181p+0, 0x1.8b73d3d8d0823p-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.eaf503ccd2be5p+0, 0x1.79cf665c76b10p-56},
    {0x1.eb9f4867cca6ep+0, 0x1.4832f2293e4f2p-54}, {0x1.ec49c80faa594p+0, -0x1.91db1fa5e4e64p-57},
    {0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54}, {0x1.ed9f78d802dc2p+0, -0x1.e9293de204116p-56},
    {0x1.ee4aaa2188510p+0, 0x1.1c68da487568dp-54}, {0x1.eef616ca06dd6p+0, 0x1.2d876b0b940d3p-55},
    {0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54}, {0x1.f04da28a52e59p+0, 0x1.69a19a4a2daadp-54},
    {0x1.f0f9c1cb6412ap+0, -0x1.3220065181d45p-54}, {0x1.f1a61cbdf5be7p+0, -0x1.3a0db8e45753dp-55},
    {0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54}, {0x1.f2ff860a70c22p+0, -0x1.bf9d712240136p-54},
    {0x1.f3ac948dd7274p+0, -0x1.95a5a3ed837dep-56}, {0x1.f459df15b82acp+0, 0x1.3819ce47a2d42p-54},
    {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54}, {0x1.f5b5288633625p+0, 0x1.e4fe7272853d5p-54},
    {0x1.f6632798844f8p+0, 0x1.fa37b3539343ep-54}, {0x1.f7116302bd526p+0, 0x1.0871fa5acb04ep-54},
    {0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54}, {0x1.f86e8f32a4b45p+0, 0x1.2baee59d08d56p-54},
    {0x1.f91d802243c89p+0, -0x1.12ea8a779f689p-57}, {0x1.f9ccadbdac61dp+0, -0x1.ab8cdee7db21ap-55},
    {0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55}, {0x1.fb2bbf4c0ba54p+0, 0x1.5e25207ff7e4fp-55},
    {0x1.fbdba3692d514p+0, -0x1.9677315098eb6p-56}, {0x1.fc8bc4866e8adp+0, 0x1.5cb1f0c14583bp-55},
    {0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57}, {0x1.fdecbe15f6314p+0, 0x1.e511aca9f0528p-54},
    {0x1.fe9d96b2a23d9p+0, 0x1.4a6037442fde3p-56}, {0x1.ff4eaca4391b6p+0, -0x1.2e60c5e4b7047p-55}};

// e^x 2^scale.
__device__ __forceinline__ double exp64(double x, int scale = 0) {
  if (fabsf(__int_as_float(__double2hiint(x))) <= __int_as_float(0x40860800)) {  // |x| <= 705
    const double t = fma(x, 0x1.71547652b82fep+9, 0x1.8p52);  // 512/ln2: k in the low word
    const int k = __double2loint(t);
    const double kd = t - 0x1.8p52;
    const double r = fma(-kd, 0x1.473de6af278edp-43, fma(-kd, 0x1.62e42fef00000p-10, x));
    const double2 T = __ldg(&kExp2Frac[k & 511]);
    const float rf = d2f(r);
    const float q = rf * fmaf(rf, 1.0f / 24, 1.0f / 6);
    const double p = fma(r * r, 0.5 + f2d(q), r);
    const double e = T.x + fma(T.x, p, T.y);
    return __hiloint2double(__double2hiint(e) + (((k >> 9) + scale) << 20), __double2loint(e));
  }
  return ldexp(exp(x), scale);
}

// Brings the table (64 lines) into L1: for kernels whose whole run is one short chain.
__device__ __forceinline__ void exp64_prefetch() {
  const char *p = (const char *)kExp2Frac;
  for (int q = threadIdx.x; q < (int)(sizeof(kExp2Frac) / 128); q += blockDim.x)
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 128 * q));
}

// n / d.
__device__ __forceinline__ double div64(double n, double d) {
  const uint32_t hn = (uint32_t)__double2hiint(n) & 0x7fffffffu;
  const uint32_t hd = (uint32_t)__double2hiint(d) & 0x7fffffffu;
  // |d| in [2^-100, 2^100), |n| in [2^-800, 2^800): nothing below leaves the normal range
  if (hd - 0x39b00000u < 0x0c800000u && hn - 0x0df00000u < 0x64000000u) {
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(d2f(d)));
    const double r0 = f2d(rf);
    const double r = fma(r0, fma(-d, r0, 1.0), r0);
    const double q = n * r;
    return fma(fma(-d, q, n), r, q);
  }
  return n / d;
}

}  // namespace nrt
