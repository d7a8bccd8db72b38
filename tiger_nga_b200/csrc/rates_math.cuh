// FP64 exponential, logarithm and quotient of the generated rate kernels.
//
// A rate kernel is straight-line code that every warp reads once per cell (0.6 MB for GRI with the library's
// functions inlined), and its time follows the number of instructions: these forms have no branch and
// few of them (exp 15 against 32 inlined, log 22 against 83, quotient 8 against 23). Constants are
// operands from constant memory (an FP64 literal takes two moves at every use), tables are in shared
// memory, staged by the kernel. Arguments are limited as each function states; the generator keeps them so.
#pragma once
#include <cuda_runtime.h>

namespace tng {

constexpr int kExpTab = 256, kLogTab = 129;
constexpr int kMathTab = kExpTab + 2 * kLogTab;  // doubles: 2^(j/256), then the logarithm's pairs

static __device__ const double c_math_tab[kMathTab] = {
    // 2^(j/256)
    0x1.0000000000000p+0, 0x1.00b1afa5abcbfp+0, 0x1.0163da9fb3335p+0, 0x1.02168143b0281p+0, 0x1.02c9a3e778061p+0,
    0x1.037d42e11bbccp+0, 0x1.04315e86e7f85p+0, 0x1.04e5f72f654b1p+0, 0x1.059b0d3158574p+0, 0x1.0650a0e3c1f89p+0,
    0x1.0706b29ddf6dep+0, 0x1.07bd42b72a836p+0, 0x1.0874518759bc8p+0, 0x1.092bdf66607e0p+0, 0x1.09e3ecac6f383p+0,
    0x1.0a9c79b1f3919p+0, 0x1.0b5586cf9890fp+0, 0x1.0c0f145e46c85p+0, 0x1.0cc922b7247f7p+0, 0x1.0d83b23395decp+0,
    0x1.0e3ec32d3d1a2p+0, 0x1.0efa55fdfa9c5p+0, 0x1.0fb66affed31bp+0, 0x1.1073028d7233ep+0, 0x1.11301d0125b51p+0,
    0x1.11edbab5e2ab6p+0, 0x1.12abdc06c31ccp+0, 0x1.136a814f204abp+0, 0x1.1429aaea92de0p+0, 0x1.14e95934f312ep+0,
    0x1.15a98c8a58e51p+0, 0x1.166a45471c3c2p+0, 0x1.172b83c7d517bp+0, 0x1.17ed48695bbc0p+0, 0x1.18af9388c8deap+0,
    0x1.1972658375d2fp+0, 0x1.1a35beb6fcb75p+0, 0x1.1af99f8138a1cp+0, 0x1.1bbe084045cd4p+0, 0x1.1c82f95281c6bp+0,
    0x1.1d4873168b9aap+0, 0x1.1e0e75eb44027p+0, 0x1.1ed5022fcd91dp+0, 0x1.1f9c18438ce4dp+0, 0x1.2063b88628cd6p+0,
    0x1.212be3578a819p+0, 0x1.21f49917ddc96p+0, 0x1.22bdda27912d1p+0, 0x1.2387a6e756238p+0, 0x1.2451ffb82140ap+0,
    0x1.251ce4fb2a63fp+0, 0x1.25e85711ece75p+0, 0x1.26b4565e27cddp+0, 0x1.2780e341ddf29p+0, 0x1.284dfe1f56381p+0,
    0x1.291ba7591bb70p+0, 0x1.29e9df51fdee1p+0, 0x1.2ab8a66d10f13p+0, 0x1.2b87fd0dad990p+0, 0x1.2c57e39771b2fp+0,
    0x1.2d285a6e4030bp+0, 0x1.2df961f641589p+0, 0x1.2ecafa93e2f56p+0, 0x1.2f9d24abd886bp+0, 0x1.306fe0a31b715p+0,
    0x1.31432edeeb2fdp+0, 0x1.32170fc4cd831p+0, 0x1.32eb83ba8ea32p+0, 0x1.33c08b26416ffp+0, 0x1.3496266e3fa2dp+0,
    0x1.356c55f929ff1p+0, 0x1.36431a2de883bp+0, 0x1.371a7373aa9cbp+0, 0x1.37f26231e754ap+0, 0x1.38cae6d05d866p+0,
    0x1.39a401b7140efp+0, 0x1.3a7db34e59ff7p+0, 0x1.3b57fbfec6cf4p+0, 0x1.3c32dc313a8e5p+0, 0x1.3d0e544ede173p+0,
    0x1.3dea64c123422p+0, 0x1.3ec70df1c5175p+0, 0x1.3fa4504ac801cp+0, 0x1.40822c367a024p+0, 0x1.4160a21f72e2ap+0,
    0x1.423fb2709468ap+0, 0x1.431f5d950a897p+0, 0x1.43ffa3f84b9d4p+0, 0x1.44e086061892dp+0, 0x1.45c2042a7d232p+0,
    0x1.46a41ed1d0057p+0, 0x1.4786d668b3237p+0, 0x1.486a2b5c13cd0p+0, 0x1.494e1e192aed2p+0, 0x1.4a32af0d7d3dep+0,
    0x1.4b17dea6db7d7p+0, 0x1.4bfdad5362a27p+0, 0x1.4ce41b817c114p+0, 0x1.4dcb299fddd0dp+0, 0x1.4eb2d81d8abffp+0,
    0x1.4f9b2769d2ca7p+0, 0x1.508417f4531eep+0, 0x1.516daa2cf6642p+0, 0x1.5257de83f4eefp+0, 0x1.5342b569d4f82p+0,
    0x1.542e2f4f6ad27p+0, 0x1.551a4ca5d920fp+0, 0x1.56070dde910d2p+0, 0x1.56f4736b527dap+0, 0x1.57e27dbe2c4cfp+0,
    0x1.58d12d497c7fdp+0, 0x1.59c0827ff07ccp+0, 0x1.5ab07dd485429p+0, 0x1.5ba11fba87a03p+0, 0x1.5c9268a5946b7p+0,
    0x1.5d84590998b93p+0, 0x1.5e76f15ad2148p+0, 0x1.5f6a320dceb71p+0, 0x1.605e1b976dc09p+0, 0x1.6152ae6cdf6f4p+0,
    0x1.6247eb03a5585p+0, 0x1.633dd1d1929fdp+0, 0x1.6434634ccc320p+0, 0x1.652b9febc8fb7p+0, 0x1.6623882552225p+0,
    0x1.671c1c70833f6p+0, 0x1.68155d44ca973p+0, 0x1.690f4b19e9538p+0, 0x1.6a09e667f3bcdp+0, 0x1.6b052fa75173ep+0,
    0x1.6c012750bdabfp+0, 0x1.6cfdcddd47645p+0, 0x1.6dfb23c651a2fp+0, 0x1.6ef9298593ae5p+0, 0x1.6ff7df9519484p+0,
    0x1.70f7466f42e87p+0, 0x1.71f75e8ec5f74p+0, 0x1.72f8286ead08ap+0, 0x1.73f9a48a58174p+0, 0x1.74fbd35d7cbfdp+0,
    0x1.75feb564267c9p+0, 0x1.77024b1ab6e09p+0, 0x1.780694fde5d3fp+0, 0x1.790b938ac1cf6p+0, 0x1.7a11473eb0187p+0,
    0x1.7b17b0976cfdbp+0, 0x1.7c1ed0130c132p+0, 0x1.7d26a62ff86f0p+0, 0x1.7e2f336cf4e62p+0, 0x1.7f3878491c491p+0,
    0x1.80427543e1a12p+0, 0x1.814d2add106d9p+0, 0x1.82589994cce13p+0, 0x1.8364c1eb941f7p+0, 0x1.8471a4623c7adp+0,
    0x1.857f4179f5b21p+0, 0x1.868d99b4492edp+0, 0x1.879cad931a436p+0, 0x1.88ac7d98a6699p+0, 0x1.89bd0a478580fp+0,
    0x1.8ace5422aa0dbp+0, 0x1.8be05bad61778p+0, 0x1.8cf3216b5448cp+0, 0x1.8e06a5e0866d9p+0, 0x1.8f1ae99157736p+0,
    0x1.902fed0282c8ap+0, 0x1.9145b0b91ffc6p+0, 0x1.925c353aa2fe2p+0, 0x1.93737b0cdc5e5p+0, 0x1.948b82b5f98e5p+0,
    0x1.95a44cbc8520fp+0, 0x1.96bdd9a7670b3p+0, 0x1.97d829fde4e50p+0, 0x1.98f33e47a22a2p+0, 0x1.9a0f170ca07bap+0,
    0x1.9b2bb4d53fe0dp+0, 0x1.9c49182a3f090p+0, 0x1.9d674194bb8d5p+0, 0x1.9e86319e32323p+0, 0x1.9fa5e8d07f29ep+0,
    0x1.a0c667b5de565p+0, 0x1.a1e7aed8eb8bbp+0, 0x1.a309bec4a2d33p+0, 0x1.a42c980460ad8p+0, 0x1.a5503b23e255dp+0,
    0x1.a674a8af46052p+0, 0x1.a799e1330b358p+0, 0x1.a8bfe53c12e59p+0, 0x1.a9e6b5579fdbfp+0, 0x1.ab0e521356ebap+0,
    0x1.ac36bbfd3f37ap+0, 0x1.ad5ff3a3c2774p+0, 0x1.ae89f995ad3adp+0, 0x1.afb4ce622f2ffp+0, 0x1.b0e07298db666p+0,
    0x1.b20ce6c9a8952p+0, 0x1.b33a2b84f15fbp+0, 0x1.b468415b749b1p+0, 0x1.b59728de5593ap+0, 0x1.b6c6e29f1c52ap+0,
    0x1.b7f76f2fb5e47p+0, 0x1.b928cf22749e4p+0, 0x1.ba5b030a1064ap+0, 0x1.bb8e0b79a6f1fp+0, 0x1.bcc1e904bc1d2p+0,
    0x1.bdf69c3f3a207p+0, 0x1.bf2c25bd71e09p+0, 0x1.c06286141b33dp+0, 0x1.c199bdd85529cp+0, 0x1.c2d1cd9fa652cp+0,
    0x1.c40ab5fffd07ap+0, 0x1.c544778fafb22p+0, 0x1.c67f12e57d14bp+0, 0x1.c7ba88988c933p+0, 0x1.c8f6d9406e7b5p+0,
    0x1.ca3405751c4dbp+0, 0x1.cb720dcef9069p+0, 0x1.ccb0f2e6d1675p+0, 0x1.cdf0b555dc3fap+0, 0x1.cf3155b5bab74p+0,
    0x1.d072d4a07897cp+0, 0x1.d1b532b08c968p+0, 0x1.d2f87080d89f2p+0, 0x1.d43c8eacaa1d6p+0, 0x1.d5818dcfba487p+0,
    0x1.d6c76e862e6d3p+0, 0x1.d80e316c98398p+0, 0x1.d955d71ff6075p+0, 0x1.da9e603db3285p+0, 0x1.dbe7cd63a8315p+0,
    0x1.dd321f301b460p+0, 0x1.de7d5641c0658p+0, 0x1.dfc97337b9b5fp+0, 0x1.e11676b197d17p+0, 0x1.e264614f5a129p+0,
    0x1.e3b333b16ee12p+0, 0x1.e502ee78b3ff6p+0, 0x1.e653924676d76p+0, 0x1.e7a51fbc74c83p+0, 0x1.e8f7977cdb740p+0,
    0x1.ea4afa2a490dap+0, 0x1.eb9f4867cca6ep+0, 0x1.ecf482d8e67f1p+0, 0x1.ee4aaa2188510p+0, 0x1.efa1bee615a27p+0,
    0x1.f0f9c1cb6412ap+0, 0x1.f252b376bba97p+0, 0x1.f3ac948dd7274p+0, 0x1.f50765b6e4540p+0, 0x1.f6632798844f8p+0,
    0x1.f7bfdad9cbe14p+0, 0x1.f91d802243c89p+0, 0x1.fa7c1819e90d8p+0, 0x1.fbdba3692d514p+0, 0x1.fd3c22b8f71f1p+0,
    0x1.fe9d96b2a23d9p+0,
    // v_j = 1 / (1 + j/128) rounded, -ln v_j
    0x1.0000000000000p+0, 0x0.0p+0, 0x1.fc07f01fc07f0p-1, 0x1.fe02a6b106799p-8,
    0x1.f81f81f81f820p-1, 0x1.fc0a8b0fc03c4p-7, 0x1.f44659e4a4271p-1, 0x1.7b91b07d5b126p-6,
    0x1.f07c1f07c1f08p-1, 0x1.f829b0e7832f8p-6, 0x1.ecc07b301ecc0p-1, 0x1.39e87b9febd68p-5,
    0x1.e9131abf0b767p-1, 0x1.77458f632dcffp-5, 0x1.e573ac901e574p-1, 0x1.b42dd711971b9p-5,
    0x1.e1e1e1e1e1e1ep-1, 0x1.f0a30c01162a8p-5, 0x1.de5d6e3f8868ap-1, 0x1.16536eea37ae3p-4,
    0x1.dae6076b981dbp-1, 0x1.341d7961bd1d0p-4, 0x1.d77b654b82c34p-1, 0x1.51b073f06183cp-4,
    0x1.d41d41d41d41dp-1, 0x1.6f0d28ae56b4ep-4, 0x1.d0cb58f6ec074p-1, 0x1.8c345d6319b23p-4,
    0x1.cd85689039b0bp-1, 0x1.a926d3a4ad562p-4, 0x1.ca4b3055ee191p-1, 0x1.c5e548f5bc743p-4,
    0x1.c71c71c71c71cp-1, 0x1.e27076e2af2eap-4, 0x1.c3f8f01c3f8f0p-1, 0x1.fec9131dbeabcp-4,
    0x1.c0e070381c0e0p-1, 0x1.0d77e7cd08e5bp-3, 0x1.bdd2b899406f7p-1, 0x1.1b72ad52f67a2p-3,
    0x1.bacf914c1bad0p-1, 0x1.29552f81ff521p-3, 0x1.b7d6c3dda338bp-1, 0x1.371fc201e8f75p-3,
    0x1.b4e81b4e81b4fp-1, 0x1.44d2b6ccb7d1cp-3, 0x1.b2036406c80d9p-1, 0x1.526e5e3a1b438p-3,
    0x1.af286bca1af28p-1, 0x1.5ff3070a793d6p-3, 0x1.ac5701ac5701bp-1, 0x1.6d60fe719d21bp-3,
    0x1.a98ef606a63bep-1, 0x1.7ab890210d907p-3, 0x1.a6d01a6d01a6dp-1, 0x1.87fa06520c911p-3,
    0x1.a41a41a41a41ap-1, 0x1.9525a9cf456b6p-3, 0x1.a16d3f97a4b02p-1, 0x1.a23bc1fe2b561p-3,
    0x1.9ec8e951033d9p-1, 0x1.af3c94e80bff3p-3, 0x1.9c2d14ee4a102p-1, 0x1.bc286742d8cd4p-3,
    0x1.999999999999ap-1, 0x1.c8ff7c79a9a20p-3, 0x1.970e4f80cb872p-1, 0x1.d5c216b4fbb94p-3,
    0x1.948b0fcd6e9e0p-1, 0x1.e27076e2af2e8p-3, 0x1.920fb49d0e229p-1, 0x1.ef0adcbdc5935p-3,
    0x1.8f9c18f9c18fap-1, 0x1.fb9186d5e3e29p-3, 0x1.8d3018d3018d3p-1, 0x1.0402594b4d041p-2,
    0x1.8acb90f6bf3aap-1, 0x1.0a324e27390e2p-2, 0x1.886e5f0abb04ap-1, 0x1.1058bf9ae4ad4p-2,
    0x1.8618618618618p-1, 0x1.1675cababa60fp-2, 0x1.83c977ab2beddp-1, 0x1.1c898c16999fbp-2,
    0x1.8181818181818p-1, 0x1.22941fbcf7966p-2, 0x1.7f405fd017f40p-1, 0x1.2895a13de86a4p-2,
    0x1.7d05f417d05f4p-1, 0x1.2e8e2bae11d31p-2, 0x1.7ad2208e0ecc3p-1, 0x1.347dd9a987d56p-2,
    0x1.78a4c8178a4c8p-1, 0x1.3a64c556945eap-2, 0x1.767dce434a9b1p-1, 0x1.404308686a7e4p-2,
    0x1.745d1745d1746p-1, 0x1.4618bc21c5ec2p-2, 0x1.724287f46debcp-1, 0x1.4be5f957778a1p-2,
    0x1.702e05c0b8170p-1, 0x1.51aad872df82ep-2, 0x1.6e1f76b4337c7p-1, 0x1.5767717455a6cp-2,
    0x1.6c16c16c16c17p-1, 0x1.5d1bdbf5809cap-2, 0x1.6a13cd1537290p-1, 0x1.62c82f2b9c796p-2,
    0x1.6816816816817p-1, 0x1.686c81e9b14adp-2, 0x1.661ec6a5122f9p-1, 0x1.6e08eaa2ba1e4p-2,
    0x1.642c8590b2164p-1, 0x1.739d7f6bbd007p-2, 0x1.623fa77016240p-1, 0x1.792a55fdd47a1p-2,
    0x1.6058160581606p-1, 0x1.7eaf83b82afc2p-2, 0x1.5e75bb8d015e7p-1, 0x1.842d1da1e8b18p-2,
    0x1.5c9882b931057p-1, 0x1.89a3386c1425bp-2, 0x1.5ac056b015ac0p-1, 0x1.8f11e873662c8p-2,
    0x1.58ed2308158edp-1, 0x1.947941c2116fbp-2, 0x1.571ed3c506b3ap-1, 0x1.99d958117e08ap-2,
    0x1.5555555555555p-1, 0x1.9f323ecbf984dp-2, 0x1.5390948f40febp-1, 0x1.a484090e5bb09p-2,
    0x1.51d07eae2f815p-1, 0x1.a9cec9a9a084ap-2, 0x1.5015015015015p-1, 0x1.af1293247786bp-2,
    0x1.4e5e0a72f0539p-1, 0x1.b44f77bcc8f64p-2, 0x1.4cab88725af6ep-1, 0x1.b9858969310fdp-2,
    0x1.4afd6a052bf5bp-1, 0x1.beb4d9da71b7ap-2, 0x1.49539e3b2d067p-1, 0x1.c3dd7a7cdad4dp-2,
    0x1.47ae147ae147bp-1, 0x1.c8ff7c79a9a21p-2, 0x1.460cbc7f5cf9ap-1, 0x1.ce1af0b85f3ecp-2,
    0x1.446f86562d9fbp-1, 0x1.d32fe7e00ebd5p-2, 0x1.42d6625d51f87p-1, 0x1.d83e7258a2f3ep-2,
    0x1.4141414141414p-1, 0x1.dd46a04c1c4a1p-2, 0x1.3fb013fb013fbp-1, 0x1.e24881a7c6c26p-2,
    0x1.3e22cbce4a902p-1, 0x1.e744261d68789p-2, 0x1.3c995a47babe7p-1, 0x1.ec399d2468cc1p-2,
    0x1.3b13b13b13b14p-1, 0x1.f128f5faf06ecp-2, 0x1.3991c2c187f63p-1, 0x1.f6123fa7028adp-2,
    0x1.3813813813814p-1, 0x1.faf588f78f31dp-2, 0x1.3698df3de0748p-1, 0x1.ffd2e0857f497p-2,
    0x1.3521cfb2b78c1p-1, 0x1.02552a5a5d0ffp-1, 0x1.33ae45b57bcb2p-1, 0x1.04bdf9da926d2p-1,
    0x1.323e34a2b10bfp-1, 0x1.0723e5c1cdf41p-1, 0x1.30d190130d190p-1, 0x1.0986f4f573521p-1,
    0x1.2f684bda12f68p-1, 0x1.0be72e4252a83p-1, 0x1.2e025c04b8097p-1, 0x1.0e44985d1cc8cp-1,
    0x1.2c9fb4d812ca0p-1, 0x1.109f39e2d4c96p-1, 0x1.2b404ad012b40p-1, 0x1.12f719593efbdp-1,
    0x1.29e4129e4129ep-1, 0x1.154c3d2f4d5eap-1, 0x1.288b01288b013p-1, 0x1.179eabbd899a0p-1,
    0x1.27350b8812735p-1, 0x1.19ee6b467c96fp-1, 0x1.25e22708092f1p-1, 0x1.1c3b81f713c25p-1,
    0x1.2492492492492p-1, 0x1.1e85f5e7040d1p-1, 0x1.23456789abcdfp-1, 0x1.20cdcd192ab6ep-1,
    0x1.21fb78121fb78p-1, 0x1.23130d7bebf43p-1, 0x1.20b470c67c0d9p-1, 0x1.2555bce98f7cap-1,
    0x1.1f7047dc11f70p-1, 0x1.2795e1289b11bp-1, 0x1.1e2ef3b3fb874p-1, 0x1.29d37fec2b08bp-1,
    0x1.1cf06ada2811dp-1, 0x1.2c0e9ed448e8cp-1, 0x1.1bb4a4046ed29p-1, 0x1.2e47436e40268p-1,
    0x1.1a7b9611a7b96p-1, 0x1.307d7334f10bep-1, 0x1.19453808ca29cp-1, 0x1.32b1339121d71p-1,
    0x1.1811811811812p-1, 0x1.34e289d9ce1d2p-1, 0x1.16e0689427379p-1, 0x1.37117b54747b6p-1,
    0x1.15b1e5f75270dp-1, 0x1.393e0d3562a1ap-1, 0x1.1485f0e0acd3bp-1, 0x1.3b68449fffc23p-1,
    0x1.135c81135c811p-1, 0x1.3d9026a7156fbp-1, 0x1.12358e75d3033p-1, 0x1.3fb5b84d16f43p-1,
    0x1.1111111111111p-1, 0x1.41d8fe84672afp-1, 0x1.0fef010fef011p-1, 0x1.43f9fe2f9ce67p-1,
    0x1.0ecf56be69c90p-1, 0x1.4618bc21c5ec2p-1, 0x1.0db20a88f4696p-1, 0x1.48353d1ea88dfp-1,
    0x1.0c9714fbcda3bp-1, 0x1.4a4f85db03ebbp-1, 0x1.0b7e6ec259dc8p-1, 0x1.4c679afccee39p-1,
    0x1.0a6810a6810a7p-1, 0x1.4e7d811b75bb0p-1, 0x1.0953f39010954p-1, 0x1.50913cc01686bp-1,
    0x1.0842108421084p-1, 0x1.52a2d265bc5abp-1, 0x1.073260a47f7c6p-1, 0x1.54b2467999498p-1,
    0x1.0624dd2f1a9fcp-1, 0x1.56bf9d5b3f399p-1, 0x1.05197f7d73404p-1, 0x1.58cadb5cd7989p-1,
    0x1.0410410410410p-1, 0x1.5ad404c359f2dp-1, 0x1.03091b51f5e1ap-1, 0x1.5cdb1dc6c1765p-1,
    0x1.0204081020408p-1, 0x1.5ee02a9241676p-1, 0x1.0101010101010p-1, 0x1.60e32f44788d9p-1,
    0x1.0000000000000p-1, 0x1.62e42fefa39efp-1};

// 0..4: 256/ln2, -ln2/256 in two parts (the first with 32 bits), 1/24, 1/6;  5..9: ln2, -1/6, 1/5, 1/3, 2^52 + 2^31
static __constant__ double c_math_k[10] = {0x1.71547652b82fep+8, -0x1.62e42fee00000p-9, -0x1.a39ef35793c76p-41, 1.0 / 24.0, 1.0 / 6.0,
                                           0x1.62e42fefa39efp-1, -1.0 / 6.0, 0.2, 1.0 / 3.0, 4503601774854144.0};

__device__ __forceinline__ void stage_math_tab(double* xt) {
  for (int j = threadIdx.x; j < kMathTab; j += blockDim.x) xt[j] = c_math_tab[j];
  __syncthreads();
}

// e^x by table (P. T. P. Tang, "Table-driven implementation of the exponential function in IEEE
// floating-point arithmetic", ACM TOMS 15, 1989): with x = (256 k + j) ln2/256 + r, |r| <= ln2/512,
//   e^x = 2^k (T_j + T_j p(r)),  T_j = 2^(j/256),  p(r) = e^r - 1
// and p's Taylor polynomial of degree 4 (the next term is below 4e-17 of the result). r carries no
// rounding of the reduction; what is left are the roundings of T_j, of its product with p and of the sum: at
// most 1.34 units in the last place (rms 0.61 of 2^-53; more than one unit for 0.3 % of arguments). The power
// of two goes into T_j's exponent (a NaN passes through p). Below the normal range the result is zero or a
// denormal, above it infinity or NaN, or with SAT at least 2^1023 and finite. |x| < 5e6 (an infinity gives NaN).
template <bool SAT = false>
__device__ __forceinline__ double tng_exp(const double x, const double* xt) {
  const double t = fma(x, c_math_k[0], 6755399441055744.0);  // 1.5 * 2^52: the integer in the low word
  const int n = min(__double2loint(t), SAT ? 1023 * 256 + 255 : 1024 * 256);
  const double kd = t - 6755399441055744.0;
  const double r = fma(kd, c_math_k[2], fma(kd, c_math_k[1], x));
  const double p = fma(r * r, fma(r, fma(r, c_math_k[3], c_math_k[4]), 0.5), r);
  const double e = xt[n & (kExpTab - 1)];
  const int hi = n < -1022 * 256 ? 0 : __double2hiint(e) + ((n >> 8) << 20);
  const double s = __hiloint2double(hi, __double2loint(e));
  return fma(s, p, s);
}

// ln x by table (P. T. P. Tang, "Table-driven implementation of the logarithm function in IEEE
// floating-point arithmetic", ACM TOMS 16, 1990): x = 2^m z, 1 <= z < 2, v_j z = 1 + r for the table's
// reciprocal v_j nearest 1/z, |r| <= 1/250 with one rounding (FMA),
//   ln x = m ln2 - ln v_j + ln(1 + r)
// and the series of ln(1 + r) to r^6 (the next term is below 3e-18). The error is within two units in the last
// place where |ln x| > 0.4 and within 1e-16 nearer to one, where the result vanishes: below one -ln 2 and
// -ln v_j cancel (x just below it takes m = -1, v = 1/2, whose constants cancel exactly), which leaves up to 83
// units of a small result (5 above one). The uses are addends of an exponent, to which that is nothing.
// Zero and denormal arguments give a value near -709; negative, infinite and NaN ones give NaN.
__device__ __forceinline__ double tng_log(const double x, const double* xt) {
  const int hx = __double2hiint(x);
  const double z = __hiloint2double((hx & 0xfffff) | 0x3ff00000, __double2loint(x));
  const int j = ((hx & 0xfffff) + 0x1000) >> 13;
  const double2 c = *reinterpret_cast<const double2*>(xt + kExpTab + 2 * j);
  // m + 2^52 + 2^31 as an integer in the low word; m = exponent - 1023
  const int m = (hx >> 20) - 1023;
  const double md = __hiloint2double(0x43300000, m ^ (int)0x80000000) - c_math_k[9];
  const double r = fma(c.x, z, -1.0);
  double q = fma(r, c_math_k[6], c_math_k[7]);
  q = fma(r, q, -0.25);
  q = fma(r, q, c_math_k[8]);
  q = fma(r, q, -0.5);
  const double base = fma(md, c_math_k[5], c.y);
  const double y = base + fma(r * r, q, r);
  return (unsigned)hx >= 0x7ff00000u ? __longlong_as_double(0x7ff8000000000000ll) : y;
}

// 1 / b from the hardware's approximate reciprocal (relative error below 2^-20, result 0 for b > 2^1022)
// and one third-order iteration (Householder): with e = 1 - b r, r (1 + e + e^2) leaves e^3. Within 0.51 units.
__device__ __forceinline__ double tng_rcp(const double b) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  const double e = fma(-b, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// a / b for operands whose quotient and its parts are in the normal range: the product with the reciprocal and
// one correction by its FMA residual (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990), correctly rounded but near a tie
__device__ __forceinline__ double tng_quot(const double a, const double b) {
  const double r = tng_rcp(b), q = a * r;
  return fma(fma(-b, q, a), r, q);
}

}  // namespace tng
