// fpmath_tables.h -- generated by gen_fpmath_tables.py; do not edit.
#pragma once

#define PDAC_LN2_HI 0x1.62e42fefa3800p-1
#define PDAC_LN2_LO 0x1.ef35793c76730p-45
#define PDAC_LN2_32_HI 0x1.62e42fefa3800p-6
#define PDAC_LN2_32_LO 0x1.ef35793c76730p-50
#define PDAC_INV_LN2_32 0x1.71547652b82fep+5

// 2^(j/32), j = 0 .. 31: hi, lo
#define PDAC_EXP2_TABLE { \
    0x1.0000000000000p+0, 0x0.0p+0, \
    0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55, \
    0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54, \
    0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54, \
    0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55, \
    0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54, \
    0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54, \
    0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55, \
    0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55, \
    0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54, \
    0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55, \
    0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59, \
    0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56, \
    0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55, \
    0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54, \
    0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54, \
    0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54, \
    0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55, \
    0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55, \
    0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54, \
    0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54, \
    0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57, \
    0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56, \
    0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54, \
    0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54, \
    0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56, \
    0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55, \
    0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56, \
    0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55, \
    0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54, \
    0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54, \
    0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54, \
}

// log(1 + j/128), j = 0 .. 128: hi, lo
#define PDAC_LOG_TABLE { \
    0x0.0p+0, 0x0.0p+0, \
    0x1.fe02a6b106789p-8, -0x1.e44b7e3711ebfp-67, \
    0x1.fc0a8b0fc03e4p-7, -0x1.83092c59642a1p-62, \
    0x1.7b91b07d5b11bp-6, -0x1.5b602ace3a510p-60, \
    0x1.f829b0e783300p-6, 0x1.33e3f04f1ef23p-60, \
    0x1.39e87b9febd60p-5, -0x1.5bfa937f551bbp-59, \
    0x1.77458f632dcfcp-5, 0x1.18d3ca87b9296p-59, \
    0x1.b42dd711971bfp-5, -0x1.eb9759c130499p-60, \
    0x1.f0a30c01162a6p-5, 0x1.85f325c5bbacdp-59, \
    0x1.16536eea37ae1p-4, -0x1.79da3e8c22cdap-60, \
    0x1.341d7961bd1d1p-4, -0x1.b599f227becbbp-58, \
    0x1.51b073f06183fp-4, 0x1.a49e39a1a8be4p-58, \
    0x1.6f0d28ae56b4cp-4, -0x1.906d99184b992p-58, \
    0x1.8c345d6319b21p-4, -0x1.4a697ab3424a9p-61, \
    0x1.a926d3a4ad563p-4, 0x1.942f48aa70ea9p-58, \
    0x1.c5e548f5bc743p-4, 0x1.5d617ef8161b1p-60, \
    0x1.e27076e2af2e6p-4, -0x1.61578001e0162p-60, \
    0x1.fec9131dbeabbp-4, -0x1.5746b9981b36cp-58, \
    0x1.0d77e7cd08e59p-3, 0x1.9a5dc5e9030acp-57, \
    0x1.1b72ad52f67a0p-3, 0x1.483023472cd74p-58, \
    0x1.29552f81ff523p-3, 0x1.301771c407dbfp-57, \
    0x1.371fc201e8f74p-3, 0x1.de6cb62af18a0p-58, \
    0x1.44d2b6ccb7d1ep-3, 0x1.9f4f6543e1f88p-57, \
    0x1.526e5e3a1b438p-3, -0x1.746ff8a470d3ap-57, \
    0x1.5ff3070a793d4p-3, -0x1.bc60efafc6f6ep-58, \
    0x1.6d60fe719d21dp-3, -0x1.caae268ecd179p-57, \
    0x1.7ab890210d909p-3, 0x1.be36b2d6a0608p-59, \
    0x1.87fa06520c911p-3, -0x1.bf7fdbfa08d9ap-57, \
    0x1.9525a9cf456b4p-3, 0x1.d904c1d4e2e26p-57, \
    0x1.a23bc1fe2b563p-3, 0x1.93711b07a998cp-59, \
    0x1.af3c94e80bff3p-3, -0x1.398cff3641985p-58, \
    0x1.bc286742d8cd6p-3, 0x1.4fce744870f55p-58, \
    0x1.c8ff7c79a9a22p-3, -0x1.4f689f8434012p-57, \
    0x1.d5c216b4fbb91p-3, 0x1.6e443597e4d40p-57, \
    0x1.e27076e2af2e6p-3, -0x1.61578001e0162p-59, \
    0x1.ef0adcbdc5936p-3, 0x1.48637950dc20dp-57, \
    0x1.fb9186d5e3e2bp-3, -0x1.caaae64f21acbp-57, \
    0x1.0402594b4d041p-2, -0x1.28ec217a5022dp-57, \
    0x1.0a324e27390e3p-2, 0x1.7dcfde8061c03p-56, \
    0x1.1058bf9ae4ad5p-2, 0x1.89fa0ab4cb31dp-58, \
    0x1.1675cababa60ep-2, 0x1.ce63eab883717p-61, \
    0x1.1c898c16999fbp-2, -0x1.0e5c62aff1c44p-60, \
    0x1.22941fbcf7966p-2, -0x1.76f5eb09628afp-56, \
    0x1.2895a13de86a3p-2, 0x1.7ad24c13f040ep-56, \
    0x1.2e8e2bae11d31p-2, -0x1.8f4cdb95ebdf9p-56, \
    0x1.347dd9a987d55p-2, -0x1.4dd4c580919f8p-57, \
    0x1.3a64c556945eap-2, -0x1.c68651945f97cp-57, \
    0x1.404308686a7e4p-2, -0x1.0bcfb6082ce6dp-56, \
    0x1.4618bc21c5ec2p-2, 0x1.f42decdeccf1dp-56, \
    0x1.4be5f957778a1p-2, -0x1.259b35b04813dp-57, \
    0x1.51aad872df82dp-2, 0x1.3927ac19f55e3p-59, \
    0x1.5767717455a6cp-2, 0x1.526adb283660cp-56, \
    0x1.5d1bdbf5809cap-2, 0x1.4236383dc7fe1p-56, \
    0x1.62c82f2b9c795p-2, 0x1.7b7af915300e5p-57, \
    0x1.686c81e9b14afp-2, -0x1.ddea0f7f58e3dp-57, \
    0x1.6e08eaa2ba1e4p-2, -0x1.cfb1b39ca3a0fp-56, \
    0x1.739d7f6bbd007p-2, -0x1.8c76ceb014b04p-56, \
    0x1.792a55fdd47a2p-2, 0x1.f057691fe9ed7p-56, \
    0x1.7eaf83b82afc3p-2, 0x1.92ce979ed2950p-56, \
    0x1.842d1da1e8b17p-2, 0x1.24ec519784676p-56, \
    0x1.89a3386c1425bp-2, -0x1.29639dfbbf0fbp-56, \
    0x1.8f11e873662c7p-2, 0x1.f85da755a61a3p-56, \
    0x1.947941c2116fbp-2, -0x1.16cc8bae0bbe4p-56, \
    0x1.99d958117e08bp-2, -0x1.a2b6889dc3e72p-57, \
    0x1.9f323ecbf984cp-2, -0x1.a92e513217f5cp-59, \
    0x1.a484090e5bb0ap-2, 0x1.5fe535b875a75p-57, \
    0x1.a9cec9a9a084ap-2, -0x1.cadec02b436afp-56, \
    0x1.af1293247786bp-2, 0x1.133844a15dc28p-58, \
    0x1.b44f77bcc8f63p-2, -0x1.cd04495459c78p-56, \
    0x1.b9858969310fbp-2, 0x1.663ec53e23bc4p-56, \
    0x1.beb4d9da71b7cp-2, -0x1.0f3c590a887cap-59, \
    0x1.c3dd7a7cdad4dp-2, 0x1.cecf052dea69bp-56, \
    0x1.c8ff7c79a9a22p-2, -0x1.4f689f8434012p-56, \
    0x1.ce1af0b85f3ebp-2, 0x1.edf4af2ab4267p-56, \
    0x1.d32fe7e00ebd5p-2, 0x1.877b232fafa37p-56, \
    0x1.d83e7258a2f3ep-2, 0x1.41456e8bb2511p-56, \
    0x1.dd46a04c1c4a1p-2, -0x1.0467656d8b892p-56, \
    0x1.e24881a7c6c26p-2, 0x1.cbd8f45954a46p-58, \
    0x1.e744261d68788p-2, -0x1.c825c90c344b9p-58, \
    0x1.ec399d2468cc0p-2, 0x1.75cee53f35397p-58, \
    0x1.f128f5faf06edp-2, -0x1.328df13bb38c3p-56, \
    0x1.f6123fa7028acp-2, 0x1.8515b0f2db341p-56, \
    0x1.faf588f78f31fp-2, -0x1.328260d8abca0p-57, \
    0x1.ffd2e0857f498p-2, 0x1.565f40d9321afp-56, \
    0x1.02552a5a5d0ffp-1, -0x1.cb1cb51408c00p-56, \
    0x1.04bdf9da926d2p-1, 0x1.97f304022c9dfp-55, \
    0x1.0723e5c1cdf40p-1, 0x1.395e58e2445bbp-55, \
    0x1.0986f4f573521p-1, -0x1.1b8095ac02f01p-55, \
    0x1.0be72e4252a83p-1, -0x1.259da11330801p-55, \
    0x1.0e44985d1cc8cp-1, -0x1.22a3442d2d384p-58, \
    0x1.109f39e2d4c97p-1, -0x1.0e09b27a4373ap-60, \
    0x1.12f719593efbcp-1, 0x1.4c048c671f435p-55, \
    0x1.154c3d2f4d5eap-1, -0x1.59c33171a6876p-55, \
    0x1.179eabbd899a1p-1, -0x1.00e7c6417e0b4p-55, \
    0x1.19ee6b467c96fp-1, -0x1.9d1a11443f10cp-56, \
    0x1.1c3b81f713c25p-1, -0x1.0dac1c4c810e9p-55, \
    0x1.1e85f5e7040d0p-1, 0x1.ef62cd2f9f1e3p-56, \
    0x1.20cdcd192ab6ep-1, -0x1.b2bf0bc229014p-55, \
    0x1.23130d7bebf43p-1, -0x1.f48725e374d6ep-55, \
    0x1.2555bce98f7cbp-1, 0x1.e021d6d6881e7p-56, \
    0x1.2795e1289b11bp-1, -0x1.487c0c246978ep-57, \
    0x1.29d37fec2b08bp-1, -0x1.bd1949a2d1982p-56, \
    0x1.2c0e9ed448e8cp-1, -0x1.1a158f3917586p-55, \
    0x1.2e47436e40268p-1, 0x1.0150861a4886bp-55, \
    0x1.307d7334f10bep-1, 0x1.fb590a1f566dap-57, \
    0x1.32b1339121d71p-1, 0x1.902ab5b3d916bp-56, \
    0x1.34e289d9ce1d3p-1, 0x1.6eb92d885ce4fp-57, \
    0x1.37117b54747b6p-1, -0x1.d117edbdd9103p-56, \
    0x1.393e0d3562a1ap-1, -0x1.58eef67f2483ap-55, \
    0x1.3b68449fffc23p-1, -0x1.41c484f9e9b26p-55, \
    0x1.3d9026a7156fbp-1, -0x1.6fef670bd4b62p-55, \
    0x1.3fb5b84d16f42p-1, 0x1.6d3a754172aefp-55, \
    0x1.41d8fe84672aep-1, 0x1.9192f30bd1806p-55, \
    0x1.43f9fe2f9ce67p-1, 0x1.e9c9ee6d83b86p-55, \
    0x1.4618bc21c5ec2p-1, 0x1.f42decdeccf1dp-55, \
    0x1.48353d1ea88dfp-1, 0x1.cf57a2ecc07f4p-55, \
    0x1.4a4f85db03ebbp-1, 0x1.13dfa3d3761b6p-60, \
    0x1.4c679afccee3ap-1, -0x1.3a5c4c8b39e41p-55, \
    0x1.4e7d811b75bb1p-1, -0x1.8d3d9ea6e9ea9p-55, \
    0x1.50913cc01686bp-1, 0x1.2f2ce96c2d5b1p-55, \
    0x1.52a2d265bc5abp-1, -0x1.1883750ea4d0ap-57, \
    0x1.54b2467999498p-1, -0x1.5baaf5d2f09f4p-55, \
    0x1.56bf9d5b3f399p-1, 0x1.0471885cd8ff3p-55, \
    0x1.58cadb5cd7989p-1, 0x1.849792ec98458p-56, \
    0x1.5ad404c359f2dp-1, -0x1.35955683f7196p-59, \
    0x1.5cdb1dc6c1765p-1, -0x1.cc2470e8a3df4p-55, \
    0x1.5ee02a9241675p-1, 0x1.c358257f49082p-55, \
    0x1.60e32f44788d9p-1, -0x1.ac1bb52fa589bp-56, \
    0x1.62e42fefa39efp-1, 0x1.abc9e3b39803fp-56, \
}

// 1 / (1 + j/128), j = 0 .. 128, rounded to nearest
#define PDAC_LOG_INVF_TABLE { \
    0x1.0000000000000p+0, \
    0x1.fc07f01fc07f0p-1, \
    0x1.f81f81f81f820p-1, \
    0x1.f44659e4a4271p-1, \
    0x1.f07c1f07c1f08p-1, \
    0x1.ecc07b301ecc0p-1, \
    0x1.e9131abf0b767p-1, \
    0x1.e573ac901e574p-1, \
    0x1.e1e1e1e1e1e1ep-1, \
    0x1.de5d6e3f8868ap-1, \
    0x1.dae6076b981dbp-1, \
    0x1.d77b654b82c34p-1, \
    0x1.d41d41d41d41dp-1, \
    0x1.d0cb58f6ec074p-1, \
    0x1.cd85689039b0bp-1, \
    0x1.ca4b3055ee191p-1, \
    0x1.c71c71c71c71cp-1, \
    0x1.c3f8f01c3f8f0p-1, \
    0x1.c0e070381c0e0p-1, \
    0x1.bdd2b899406f7p-1, \
    0x1.bacf914c1bad0p-1, \
    0x1.b7d6c3dda338bp-1, \
    0x1.b4e81b4e81b4fp-1, \
    0x1.b2036406c80d9p-1, \
    0x1.af286bca1af28p-1, \
    0x1.ac5701ac5701bp-1, \
    0x1.a98ef606a63bep-1, \
    0x1.a6d01a6d01a6dp-1, \
    0x1.a41a41a41a41ap-1, \
    0x1.a16d3f97a4b02p-1, \
    0x1.9ec8e951033d9p-1, \
    0x1.9c2d14ee4a102p-1, \
    0x1.999999999999ap-1, \
    0x1.970e4f80cb872p-1, \
    0x1.948b0fcd6e9e0p-1, \
    0x1.920fb49d0e229p-1, \
    0x1.8f9c18f9c18fap-1, \
    0x1.8d3018d3018d3p-1, \
    0x1.8acb90f6bf3aap-1, \
    0x1.886e5f0abb04ap-1, \
    0x1.8618618618618p-1, \
    0x1.83c977ab2beddp-1, \
    0x1.8181818181818p-1, \
    0x1.7f405fd017f40p-1, \
    0x1.7d05f417d05f4p-1, \
    0x1.7ad2208e0ecc3p-1, \
    0x1.78a4c8178a4c8p-1, \
    0x1.767dce434a9b1p-1, \
    0x1.745d1745d1746p-1, \
    0x1.724287f46debcp-1, \
    0x1.702e05c0b8170p-1, \
    0x1.6e1f76b4337c7p-1, \
    0x1.6c16c16c16c17p-1, \
    0x1.6a13cd1537290p-1, \
    0x1.6816816816817p-1, \
    0x1.661ec6a5122f9p-1, \
    0x1.642c8590b2164p-1, \
    0x1.623fa77016240p-1, \
    0x1.6058160581606p-1, \
    0x1.5e75bb8d015e7p-1, \
    0x1.5c9882b931057p-1, \
    0x1.5ac056b015ac0p-1, \
    0x1.58ed2308158edp-1, \
    0x1.571ed3c506b3ap-1, \
    0x1.5555555555555p-1, \
    0x1.5390948f40febp-1, \
    0x1.51d07eae2f815p-1, \
    0x1.5015015015015p-1, \
    0x1.4e5e0a72f0539p-1, \
    0x1.4cab88725af6ep-1, \
    0x1.4afd6a052bf5bp-1, \
    0x1.49539e3b2d067p-1, \
    0x1.47ae147ae147bp-1, \
    0x1.460cbc7f5cf9ap-1, \
    0x1.446f86562d9fbp-1, \
    0x1.42d6625d51f87p-1, \
    0x1.4141414141414p-1, \
    0x1.3fb013fb013fbp-1, \
    0x1.3e22cbce4a902p-1, \
    0x1.3c995a47babe7p-1, \
    0x1.3b13b13b13b14p-1, \
    0x1.3991c2c187f63p-1, \
    0x1.3813813813814p-1, \
    0x1.3698df3de0748p-1, \
    0x1.3521cfb2b78c1p-1, \
    0x1.33ae45b57bcb2p-1, \
    0x1.323e34a2b10bfp-1, \
    0x1.30d190130d190p-1, \
    0x1.2f684bda12f68p-1, \
    0x1.2e025c04b8097p-1, \
    0x1.2c9fb4d812ca0p-1, \
    0x1.2b404ad012b40p-1, \
    0x1.29e4129e4129ep-1, \
    0x1.288b01288b013p-1, \
    0x1.27350b8812735p-1, \
    0x1.25e22708092f1p-1, \
    0x1.2492492492492p-1, \
    0x1.23456789abcdfp-1, \
    0x1.21fb78121fb78p-1, \
    0x1.20b470c67c0d9p-1, \
    0x1.1f7047dc11f70p-1, \
    0x1.1e2ef3b3fb874p-1, \
    0x1.1cf06ada2811dp-1, \
    0x1.1bb4a4046ed29p-1, \
    0x1.1a7b9611a7b96p-1, \
    0x1.19453808ca29cp-1, \
    0x1.1811811811812p-1, \
    0x1.16e0689427379p-1, \
    0x1.15b1e5f75270dp-1, \
    0x1.1485f0e0acd3bp-1, \
    0x1.135c81135c811p-1, \
    0x1.12358e75d3033p-1, \
    0x1.1111111111111p-1, \
    0x1.0fef010fef011p-1, \
    0x1.0ecf56be69c90p-1, \
    0x1.0db20a88f4696p-1, \
    0x1.0c9714fbcda3bp-1, \
    0x1.0b7e6ec259dc8p-1, \
    0x1.0a6810a6810a7p-1, \
    0x1.0953f39010954p-1, \
    0x1.0842108421084p-1, \
    0x1.073260a47f7c6p-1, \
    0x1.0624dd2f1a9fcp-1, \
    0x1.05197f7d73404p-1, \
    0x1.0410410410410p-1, \
    0x1.03091b51f5e1ap-1, \
    0x1.0204081020408p-1, \
    0x1.0101010101010p-1, \
    0x1.0000000000000p-1, \
}

