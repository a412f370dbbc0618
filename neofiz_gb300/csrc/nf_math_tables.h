/* Generated by gen_nf_math_tables.py; do not edit. */
#ifndef NF_MATH_TABLES_H
#define NF_MATH_TABLES_H

#define NF_LOG_OFF 0x3fe6900000000000ULL
#define NF_EXP_N_OVER_LN2 0x1.71547652b82fep+7   /* 128 / ln 2 */
#define NF_EXP_L_HI 0x1.62e42fefc0000p-8   /* ln 2 / 128, 35 significant bits */
#define NF_EXP_L_LO -0x1.c610ca86c3899p-44

/* invc, -log(invc) hi, lo, 0 */
#define NF_LOG_TABLE \
    0x1.6a13cd1537290p+0, -0x1.630030b3aac48p-2, -0x1.ee0c6728fffccp-56, 0.0, \
    0x1.6816816816817p+0, -0x1.5d5bddf595f31p-2, -0x1.d5f75b9a23ae4p-59, 0.0, \
    0x1.661ec6a5122f9p+0, -0x1.57bf753c8d1fbp-2, 0x1.2908d15f88b63p-57, 0.0, \
    0x1.642c8590b2164p+0, -0x1.522ae0738a3d7p-2, -0x1.3840b263acb43p-56, 0.0, \
    0x1.623fa77016240p+0, -0x1.4c9e09e172c3dp-2, 0x1.123615b147a5fp-58, 0.0, \
    0x1.6058160581606p+0, -0x1.4718dc271c41cp-2, -0x1.d8fb4c14c56eep-56, 0.0, \
    0x1.5e75bb8d015e7p+0, -0x1.419b423d5e8c6p-2, -0x1.5b7648704e721p-58, 0.0, \
    0x1.5c9882b931057p+0, -0x1.3c25277333183p-2, -0x1.152d81af5713ap-56, 0.0, \
    0x1.5ac056b015ac0p+0, -0x1.36b6776be1116p-2, 0x1.324f0e8838590p-58, 0.0, \
    0x1.58ed2308158edp+0, -0x1.314f1e1d35ce3p-2, -0x1.22966f61a3c23p-56, 0.0, \
    0x1.571ed3c506b3ap+0, -0x1.2bef07cdc9355p-2, 0x1.22dad7fd86088p-56, 0.0, \
    0x1.5555555555555p+0, -0x1.269621134db91p-2, -0x1.e0efadd9db02ap-56, 0.0, \
    0x1.5390948f40febp+0, -0x1.214456d0eb8d5p-2, 0x1.50a2dca28b3edp-58, 0.0, \
    0x1.51d07eae2f815p+0, -0x1.1bf99635a6b95p-2, 0x1.e9575c2124912p-56, 0.0, \
    0x1.5015015015015p+0, -0x1.16b5ccbacfb73p-2, -0x1.56fbd28b40935p-56, 0.0, \
    0x1.4e5e0a72f0539p+0, -0x1.1178e8227e47ap-2, -0x1.b8ce2d07f1cb7p-56, 0.0, \
    0x1.4cab88725af6ep+0, -0x1.0c42d676162e2p-2, 0x1.5a74e18a8bb85p-56, 0.0, \
    0x1.4afd6a052bf5bp+0, -0x1.07138604d5864p-2, 0x1.24e912b16ec8bp-60, 0.0, \
    0x1.49539e3b2d067p+0, -0x1.01eae5626c691p-2, -0x1.d9f5bd0b5b348p-57, 0.0, \
    0x1.47ae147ae147bp+0, -0x1.f991c6cb3b37ap-3, -0x1.ecca0cdf30143p-58, 0.0, \
    0x1.460cbc7f5cf9ap+0, -0x1.ef5ade4dcffe5p-3, -0x1.7754d2238f75fp-58, 0.0, \
    0x1.446f86562d9fbp+0, -0x1.e530effe71013p-3, 0x1.f7627ef82f3f0p-57, 0.0, \
    0x1.42d6625d51f87p+0, -0x1.db13db0d48941p-3, 0x1.8af715b0349a4p-57, 0.0, \
    0x1.4141414141414p+0, -0x1.d1037f2655e7bp-3, 0x1.3f3adb7b71cbcp-58, 0.0, \
    0x1.3fb013fb013fbp+0, -0x1.c6ffbc6f00f71p-3, 0x1.ae58b2c57a4a5p-57, 0.0, \
    0x1.3e22cbce4a902p+0, -0x1.bd087383bd8aap-3, 0x1.1165504ad749ep-59, 0.0, \
    0x1.3c995a47babe7p+0, -0x1.b31d8575bce3bp-3, 0x1.0d4eace1aa537p-59, 0.0, \
    0x1.3b13b13b13b14p+0, -0x1.a93ed3c8ad9e5p-3, -0x1.bcafa9de97202p-57, 0.0, \
    0x1.3991c2c187f63p+0, -0x1.9f6c407089663p-3, 0x1.52979a7e86605p-57, 0.0, \
    0x1.3813813813814p+0, -0x1.95a5adcf70182p-3, -0x1.8a16283fdbd1cp-57, 0.0, \
    0x1.3698df3de0748p+0, -0x1.8beafeb38fe8fp-3, 0x1.54aae92cd0b87p-59, 0.0, \
    0x1.3521cfb2b78c1p+0, -0x1.823c16551a3c0p-3, -0x1.6dcd318f4187ep-57, 0.0, \
    0x1.33ae45b57bcb2p+0, -0x1.7898d85444c74p-3, -0x1.be3dbaf3ec804p-60, 0.0, \
    0x1.323e34a2b10bfp+0, -0x1.6f0128b756ab9p-3, 0x1.37967087859b9p-59, 0.0, \
    0x1.30d190130d190p+0, -0x1.6574ebe8c1339p-3, -0x1.c5961e173bc82p-57, 0.0, \
    0x1.2f684bda12f68p+0, -0x1.5bf406b543db0p-3, 0x1.1f5b44c0df7f7p-61, 0.0, \
    0x1.2e025c04b8097p+0, -0x1.527e5e4a1b58dp-3, 0x1.b8d4b411cadffp-60, 0.0, \
    0x1.2c9fb4d812ca0p+0, -0x1.4913d8333b563p-3, 0x1.0d5604930f137p-58, 0.0, \
    0x1.2b404ad012b40p+0, -0x1.3fb45a59928cap-3, 0x1.d87e6a354d057p-57, 0.0, \
    0x1.29e4129e4129ep+0, -0x1.365fcb0159014p-3, -0x1.bea08d2dca256p-57, 0.0, \
    0x1.288b01288b013p+0, -0x1.2d1610c86813dp-3, -0x1.d997036941a6dp-60, 0.0, \
    0x1.27350b8812735p+0, -0x1.23d712a49c201p-3, -0x1.51c7e9efae297p-57, 0.0, \
    0x1.25e22708092f1p+0, -0x1.1aa2b7e23f729p-3, -0x1.6e44389934420p-57, 0.0, \
    0x1.2492492492492p+0, -0x1.1178e8227e47ap-3, 0x1.0e63a5f01c693p-58, 0.0, \
    0x1.23456789abcdfp+0, -0x1.08598b59e3a07p-3, 0x1.fd7009902bf32p-57, 0.0, \
    0x1.21fb78121fb78p+0, -0x1.fe89139dbd565p-4, 0x1.ac9f4215f9394p-58, 0.0, \
    0x1.20b470c67c0d9p+0, -0x1.ec739830a1126p-4, -0x1.eea033743f95bp-58, 0.0, \
    0x1.1f7047dc11f70p+0, -0x1.da7276384469ep-4, -0x1.401fa71733017p-58, 0.0, \
    0x1.1e2ef3b3fb874p+0, -0x1.c885801bc4b20p-4, 0x1.5c734aa6598fcp-58, 0.0, \
    0x1.1cf06ada2811dp+0, -0x1.b6ac88dad5b1dp-4, 0x1.002bf768e52d0p-58, 0.0, \
    0x1.1bb4a4046ed29p+0, -0x1.a4e7640b1bc38p-4, 0x1.9b5ca203e4259p-58, 0.0, \
    0x1.1a7b9611a7b96p+0, -0x1.9335e5d594988p-4, 0x1.478a85704ccb7p-58, 0.0, \
    0x1.19453808ca29cp+0, -0x1.8197e2f40e3f0p-4, 0x1.230690020895fp-59, 0.0, \
    0x1.1811811811812p+0, -0x1.700d30aeac0e8p-4, -0x1.a36a677b4c8b2p-59, 0.0, \
    0x1.16e0689427379p+0, -0x1.5e95a4d9791cdp-4, 0x1.4c78ba3a3baf6p-58, 0.0, \
    0x1.15b1e5f75270dp+0, -0x1.4d3115d207eacp-4, -0x1.da7d0b1e10b2fp-60, 0.0, \
    0x1.1485f0e0acd3bp+0, -0x1.3bdf5a7d1ee5ep-4, -0x1.f52eda76b68acp-60, 0.0, \
    0x1.135c81135c811p+0, -0x1.2aa04a44717a1p-4, -0x1.aea2c72d05c08p-58, 0.0, \
    0x1.12358e75d3033p+0, -0x1.1973bd1465561p-4, 0x1.7aac1b3d35680p-58, 0.0, \
    0x1.1111111111111p+0, -0x1.08598b59e3a06p-4, 0x1.dd7009902bf32p-58, 0.0, \
    0x1.0fef010fef011p+0, -0x1.eea31c006b87cp-5, 0x1.7c9f9276f6cd8p-60, 0.0, \
    0x1.0ecf56be69c90p+0, -0x1.ccb73cdddb2d0p-5, 0x1.e48fb0500efd5p-59, 0.0, \
    0x1.0db20a88f4696p+0, -0x1.aaef2d0fb1108p-5, -0x1.68d4eed0b82aep-59, 0.0, \
    0x1.0c9714fbcda3bp+0, -0x1.894aa149fb34bp-5, 0x1.2ba0b44cfaee5p-59, 0.0, \
    0x1.0b7e6ec259dc8p+0, -0x1.67c94f2d4bb65p-5, -0x1.0413e6505e5f9p-59, 0.0, \
    0x1.0a6810a6810a7p+0, -0x1.466aed42de3f9p-5, 0x1.9badefe942718p-60, 0.0, \
    0x1.0953f39010954p+0, -0x1.252f32f8d1840p-5, -0x1.ae021b67a9ba8p-61, 0.0, \
    0x1.0842108421084p+0, -0x1.0415d89e74440p-5, -0x1.c05cf1d753621p-59, 0.0, \
    0x1.073260a47f7c6p+0, -0x1.c63d2ec14aad7p-6, -0x1.8fe7acbca131dp-63, 0.0, \
    0x1.0624dd2f1a9fcp+0, -0x1.8492528c8cac5p-6, 0x1.d192d0619fa68p-60, 0.0, \
    0x1.05197f7d73404p+0, -0x1.432a925980cbcp-6, 0x1.8cdaf39004193p-60, 0.0, \
    0x1.0410410410410p+0, -0x1.0205658935837p-6, -0x1.27c8e8416e717p-60, 0.0, \
    0x1.03091b51f5e1ap+0, -0x1.82448a388a283p-7, -0x1.04b16137f0970p-62, 0.0, \
    0x1.0204081020408p+0, -0x1.010157588de69p-7, -0x1.46662d417cecep-62, 0.0, \
    0x1.0101010101010p+0, -0x1.0080559588b25p-8, -0x1.f96638cf63675p-62, 0.0, \
    0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0, 0.0, \
    0x1.fc07f01fc07f0p-1, 0x1.fe02a6b106799p-8, -0x1.e44b7e3711e7fp-67, 0.0, \
    0x1.f81f81f81f820p-1, 0x1.fc0a8b0fc03c4p-7, -0x1.83092c5964281p-62, 0.0, \
    0x1.f44659e4a4271p-1, 0x1.7b91b07d5b126p-6, -0x1.6d80ab38e9430p-62, 0.0, \
    0x1.f07c1f07c1f08p-1, 0x1.f829b0e7832f8p-6, 0x1.33e3f04f1ef25p-60, 0.0, \
    0x1.ecc07b301ecc0p-1, 0x1.39e87b9febd68p-5, -0x1.5bfa937f551b7p-59, 0.0, \
    0x1.e9131abf0b767p-1, 0x1.77458f632dcffp-5, 0x1.8d3ca87b92968p-63, 0.0, \
    0x1.e573ac901e574p-1, 0x1.b42dd711971b9p-5, 0x1.0a34531f67db5p-59, 0.0, \
    0x1.e1e1e1e1e1e1ep-1, 0x1.f0a30c01162a8p-5, 0x1.85f325c5bbacdp-59, 0.0, \
    0x1.de5d6e3f8868ap-1, 0x1.16536eea37ae3p-4, 0x1.2189705cf74cap-58, 0.0, \
    0x1.dae6076b981dbp-1, 0x1.341d7961bd1d0p-4, -0x1.3599f227becbbp-58, 0.0, \
    0x1.d77b654b82c34p-1, 0x1.51b073f06183cp-4, -0x1.5b61c65e5741ap-58, 0.0, \
    0x1.d41d41d41d41dp-1, 0x1.6f0d28ae56b4ep-4, -0x1.20db323097324p-59, 0.0, \
    0x1.d0cb58f6ec074p-1, 0x1.8c345d6319b23p-4, -0x1.294d2f5668495p-58, 0.0, \
    0x1.cd85689039b0bp-1, 0x1.a926d3a4ad562p-4, -0x1.d7a16eab1e2adp-59, 0.0, \
    0x1.ca4b3055ee191p-1, 0x1.c5e548f5bc743p-4, 0x1.2eb0bf7c0b0d9p-59, 0.0, \
    0x1.c71c71c71c71cp-1, 0x1.e27076e2af2eap-4, -0x1.61578001e015ap-60, 0.0, \
    0x1.c3f8f01c3f8f0p-1, 0x1.fec9131dbeabcp-4, -0x1.5746b9981b36cp-58, 0.0, \
    0x1.c0e070381c0e0p-1, 0x1.0d77e7cd08e5bp-3, 0x1.9a5dc5e9030adp-57, 0.0, \
    0x1.bdd2b899406f7p-1, 0x1.1b72ad52f67a2p-3, -0x1.fbe7ee5c69946p-57, 0.0, \
    0x1.bacf914c1bad0p-1, 0x1.29552f81ff521p-3, 0x1.301771c407dc0p-57, 0.0, \
    0x1.b7d6c3dda338bp-1, 0x1.371fc201e8f75p-3, 0x1.e6cb62af18a02p-62, 0.0, \
    0x1.b4e81b4e81b4fp-1, 0x1.44d2b6ccb7d1cp-3, 0x1.7d3d950f87e23p-59, 0.0, \
    0x1.b2036406c80d9p-1, 0x1.526e5e3a1b438p-3, -0x1.546ff8a470d3ap-57, 0.0, \
    0x1.af286bca1af28p-1, 0x1.5ff3070a793d6p-3, -0x1.bc60efafc6f6cp-58, 0.0, \
    0x1.ac5701ac5701bp-1, 0x1.6d60fe719d21bp-3, 0x1.d551d97132e87p-57, 0.0, \
    0x1.a98ef606a63bep-1, 0x1.7ab890210d907p-3, -0x1.1072534a57e7dp-57, 0.0, \
    0x1.a6d01a6d01a6dp-1, 0x1.87fa06520c911p-3, -0x1.9f7fdbfa08d9ap-57, 0.0, \
    0x1.a41a41a41a41ap-1, 0x1.9525a9cf456b6p-3, -0x1.26fb3e2b1d1dap-57, 0.0, \
    0x1.a16d3f97a4b02p-1, 0x1.a23bc1fe2b561p-3, 0x1.24dc46c1ea664p-57, 0.0, \
    0x1.9ec8e951033d9p-1, 0x1.af3c94e80bff3p-3, 0x1.a3398064df33ep-57, 0.0, \
    0x1.9c2d14ee4a102p-1, 0x1.bc286742d8cd4p-3, 0x1.cfce744870f57p-58, 0.0, \
    0x1.999999999999ap-1, 0x1.c8ff7c79a9a20p-3, -0x1.4f689f8434011p-57, 0.0, \
    0x1.970e4f80cb872p-1, 0x1.d5c216b4fbb94p-3, -0x1.a37794d03657dp-58, 0.0, \
    0x1.948b0fcd6e9e0p-1, 0x1.e27076e2af2e8p-3, -0x1.61578001e015ep-59, 0.0, \
    0x1.920fb49d0e229p-1, 0x1.ef0adcbdc5935p-3, 0x1.e8637950dc20dp-57, 0.0, \
    0x1.8f9c18f9c18fap-1, 0x1.fb9186d5e3e29p-3, 0x1.355519b0de535p-57, 0.0, \
    0x1.8d3018d3018d3p-1, 0x1.0402594b4d041p-2, -0x1.08ec217a5022dp-57, 0.0, \
    0x1.8acb90f6bf3aap-1, 0x1.0a324e27390e2p-2, 0x1.bdcfde8061c03p-56, 0.0, \
    0x1.886e5f0abb04ap-1, 0x1.1058bf9ae4ad4p-2, 0x1.3f415699663ecp-63, 0.0, \
    0x1.8618618618618p-1, 0x1.1675cababa60fp-2, 0x1.ce63eab883727p-61, 0.0, \
    0x1.83c977ab2beddp-1, 0x1.1c898c16999fbp-2, 0x1.9f1a39d500e3cp-56, 0.0, \
    0x1.8181818181818p-1, 0x1.22941fbcf7966p-2, -0x1.dbd7ac258a2bdp-58, 0.0, \
    0x1.7f405fd017f40p-1, 0x1.2895a13de86a4p-2, 0x1.7ad24c13f040fp-56, 0.0, \
    0x1.7d05f417d05f4p-1, 0x1.2e8e2bae11d31p-2, -0x1.1e99b72bd7bf2p-57, 0.0, \
    0x1.7ad2208e0ecc3p-1, 0x1.347dd9a987d56p-2, -0x1.16ea62c048cfbp-56, 0.0, \
    0x1.78a4c8178a4c8p-1, 0x1.3a64c556945eap-2, 0x1.cbcd735d03424p-60, 0.0, \
    0x1.767dce434a9b1p-1, 0x1.404308686a7e4p-2, -0x1.f79f6c1059cdbp-57, 0.0, \
    0x1.745d1745d1746p-1, 0x1.4618bc21c5ec2p-2, -0x1.7a42642661c62p-61, 0.0, \
    0x1.724287f46debcp-1, 0x1.4be5f957778a1p-2, -0x1.4b366b609027ap-58, 0.0, \
    0x1.702e05c0b8170p-1, 0x1.51aad872df82ep-2, -0x1.d8db0a7cc1543p-56, 0.0, \
    0x1.6e1f76b4337c7p-1, 0x1.5767717455a6cp-2, -0x1.fb2a49af933e8p-57, 0.0, \
    0x1.6c16c16c16c17p-1, 0x1.5d1bdbf5809cap-2, -0x1.7dc9c7c23801fp-56, 0.0, \

/* 2^(j/128) hi, lo */
#define NF_EXP_TABLE \
    0x1.0000000000000p+0, 0x0.0p+0, \
    0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54, \
    0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56, \
    0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54, \
    0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55, \
    0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55, \
    0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57, \
    0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54, \
    0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54, \
    0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54, \
    0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59, \
    0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57, \
    0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54, \
    0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58, \
    0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54, \
    0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55, \
    0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55, \
    0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54, \
    0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55, \
    0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54, \
    0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54, \
    0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54, \
    0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55, \
    0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55, \
    0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54, \
    0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55, \
    0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55, \
    0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54, \
    0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55, \
    0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59, \
    0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54, \
    0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56, \
    0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55, \
    0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55, \
    0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54, \
    0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55, \
    0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54, \
    0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54, \
    0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56, \
    0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54, \
    0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55, \
    0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54, \
    0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58, \
    0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55, \
    0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59, \
    0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54, \
    0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56, \
    0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54, \
    0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56, \
    0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54, \
    0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54, \
    0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55, \
    0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55, \
    0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55, \
    0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54, \
    0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55, \
    0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54, \
    0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60, \
    0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54, \
    0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54, \
    0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54, \
    0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55, \
    0x1.6623882552225p+0, -0x1.bb60987591c34p-54, \
    0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57, \
    0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54, \
    0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56, \
    0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57, \
    0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55, \
    0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55, \
    0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54, \
    0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54, \
    0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54, \
    0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55, \
    0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54, \
    0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56, \
    0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54, \
    0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54, \
    0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55, \
    0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54, \
    0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54, \
    0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54, \
    0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56, \
    0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55, \
    0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54, \
    0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57, \
    0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56, \
    0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54, \
    0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54, \
    0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56, \
    0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56, \
    0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54, \
    0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54, \
    0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54, \
    0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54, \
    0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54, \
    0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55, \
    0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54, \
    0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54, \
    0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57, \
    0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54, \
    0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56, \
    0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54, \
    0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55, \
    0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54, \
    0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55, \
    0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54, \
    0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54, \
    0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56, \
    0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56, \
    0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55, \
    0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54, \
    0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54, \
    0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55, \
    0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54, \
    0x1.da9e603db3285p+0, 0x1.c2300696db532p-54, \
    0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54, \
    0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54, \
    0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54, \
    0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55, \
    0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54, \
    0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54, \
    0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54, \
    0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54, \
    0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54, \
    0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54, \
    0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54, \
    0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55, \
    0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57, \

/* ln 2 in units of 2^-84, and the integer log table: invc 2^53 (lo, hi), then
 * -log(invc) - 1088 ln 2 in those units (lo, mid, hi); padded to 32 bytes */
#define NF_LN2_FIX0 0x9abc9e3bu
#define NF_LN2_FIX1 0x7f7d1cf7u
#define NF_LN2_FIX2 0x000b1721u
#define NF_LOG_BIAS 1088
#define NF_LOG_WORDS \
    0xa2a6e520u, 0x002d4279u, 0x3f7ebecdu, 0x6976389cu, 0xd0d825a1u, 0u, 0u, 0u, \
    0x2d02d02eu, 0x002d02d0u, 0x1ab39689u, 0xb46e8be2u, 0xd0d83c32u, 0u, 0u, 0u, \
    0xd4a245f2u, 0x002cc3d8u, 0xa7a7cbcbu, 0x5752af2fu, 0xd0d852a4u, 0u, 0u, 0u, \
    0xb21642c8u, 0x002c8590u, 0x8adb7a1au, 0xaa76bab8u, 0xd0d868f6u, 0u, 0u, 0u, \
    0xee02c480u, 0x002c47f4u, 0x22a85d97u, 0x04bf189fu, 0xd0d87f2au, 0u, 0u, 0u, \
    0xc0b02c0cu, 0x002c0b02u, 0x40cfd07fu, 0xbba872a7u, 0xd0d8953eu, 0u, 0u, 0u, \
    0x71a02bceu, 0x002bceb7u, 0xd8f1ac1eu, 0x234f697cu, 0xd0d8ab35u, 0u, 0u, 0u, \
    0x572620aeu, 0x002b9310u, 0x8d0cad25u, 0x8e78174du, 0xd0d8c10du, 0u, 0u, 0u, \
    0xd602b580u, 0x002b580au, 0xe328c17au, 0x4e955f68u, 0xd0d8d6c8u, 0u, 0u, 0u, \
    0x6102b1dau, 0x002b1da4u, 0x8c361e4au, 0xb3d00c75u, 0xd0d8ec65u, 0u, 0u, 0u, \
    0x78a0d674u, 0x002ae3dau, 0x308d32c0u, 0x0d0dbed9u, 0xd0d901e6u, 0u, 0u, 0u, \
    0xaaaaaaaau, 0x002aaaaau, 0x00508a62u, 0xa7f7accau, 0xd0d91749u, 0u, 0u, 0u, \
    0x91e81fd6u, 0x002a7212u, 0x23a210b3u, 0xd1013579u, 0xd0d92c90u, 0u, 0u, 0u, \
    0xd5c5f02au, 0x002a3a0fu, 0x3cf4fb02u, 0xd36e48c9u, 0xd0d941bbu, 0u, 0u, 0u, \
    0x2a02a02au, 0x002a02a0u, 0x88efc817u, 0xf959a4d1u, 0xd0d956cau, 0u, 0u, 0u, \
    0x4e5e0a72u, 0x0029cbc1u, 0xc2d2a270u, 0x8bbaea8fu, 0xd0d96bbeu, 0u, 0u, 0u, \
    0x0e4b5edcu, 0x00299571u, 0xf406d359u, 0xd26c8af5u, 0xd0d98096u, 0u, 0u, 0u, \
    0x40a57eb6u, 0x00295fadu, 0x5f846e53u, 0x14318d95u, 0xd0d99554u, 0u, 0u, 0u, \
    0xc765a0ceu, 0x00292a73u, 0x0f8fd758u, 0x96bb320au, 0xd0d9a9f6u, 0u, 0u, 0u, \
    0x8f5c28f6u, 0x0028f5c2u, 0x16ac5d0du, 0x9eae6d3fu, 0xd0d9be7eu, 0u, 0u, 0u, \
    0x8feb9f34u, 0x0028c197u, 0xb88231f7u, 0x6fa943b1u, 0xd0d9d2ecu, 0u, 0u, 0u, \
    0xcac5b3f6u, 0x00288df0u, 0x0e1a9938u, 0x4c4801acu, 0xd0d9e740u, 0u, 0u, 0u, \
    0x4baa3f0eu, 0x00285accu, 0x4ab73deeu, 0x762a5286u, 0xd0d9fb7au, 0u, 0u, 0u, \
    0x28282828u, 0x00282828u, 0x035c70aeu, 0x2df837dfu, 0xd0da0f9bu, 0u, 0u, 0u, \
    0x7f6027f6u, 0x0027f602u, 0x4bd24ad6u, 0xb366e1c0u, 0xd0da23a2u, 0u, 0u, 0u, \
    0x79c95204u, 0x0027c459u, 0x20824fe1u, 0x453d6899u, 0xd0da3791u, 0u, 0u, 0u, \
    0x48f757ceu, 0x0027932bu, 0x007a229au, 0x215969e7u, 0xd0da4b67u, 0u, 0u, 0u, \
    0x27627628u, 0x00276276u, 0xb07a07f1u, 0x84b38871u, 0xd0da5f24u, 0u, 0u, 0u, \
    0x5830fec6u, 0x00273238u, 0x08f44214u, 0xab63d0e2u, 0xd0da72c9u, 0u, 0u, 0u, \
    0x27027028u, 0x00270270u, 0x120ed3feu, 0xd0a6037eu, 0xd0da8656u, 0u, 0u, 0u, \
    0xe7bc0e90u, 0x0026d31bu, 0x8108db12u, 0x2eddc3dcu, 0xd0da99ccu, 0u, 0u, 0u, \
    0xf656f182u, 0x0026a439u, 0x52f11bb4u, 0xff9aaf36u, 0xd0daad29u, 0u, 0u, 0u, \
    0xb6af7964u, 0x002675c8u, 0xdca14785u, 0x7b9c5a1fu, 0xd0dac070u, 0u, 0u, 0u, \
    0x9456217eu, 0x002647c6u, 0x40ceb221u, 0xdad63657u, 0xd0dad39fu, 0u, 0u, 0u, \
    0x0261a320u, 0x00261a32u, 0x3032d44fu, 0x54736147u, 0xd0dae6b8u, 0u, 0u, 0u, \
    0x7b425ed0u, 0x0025ed09u, 0x5eef32e2u, 0x1eda5bf8u, 0xd0daf9bau, 0u, 0u, 0u, \
    0x8097012eu, 0x0025c04bu, 0xc01859f4u, 0x6fb0acfcu, 0xd0db0ca5u, 0u, 0u, 0u, \
    0x9b025940u, 0x002593f6u, 0x0294dd52u, 0x7bde6d02u, 0xd0db1f7au, 0u, 0u, 0u, \
    0x5a025680u, 0x00256809u, 0x2d237892u, 0x7791be95u, 0xd0db3239u, 0u, 0u, 0u, \
    0x53c8253cu, 0x00253c82u, 0xd06a80d7u, 0x964231abu, 0xd0db44e2u, 0u, 0u, 0u, \
    0x25116026u, 0x00251160u, 0xbc85ee3du, 0x0ab41386u, 0xd0db5776u, 0u, 0u, 0u, \
    0x71024e6au, 0x0024e6a1u, 0x33d145f1u, 0x06fbab6eu, 0xd0db69f4u, 0u, 0u, 0u, \
    0xe10125e2u, 0x0024bc44u, 0x32ed637bu, 0xbc8064c9u, 0xd0db7c5cu, 0u, 0u, 0u, \
    0x24924924u, 0x00249249u, 0x229913d8u, 0x5bffe71fu, 0xd0db8eb0u, 0u, 0u, 0u, \
    0xf13579beu, 0x002468acu, 0x8e4b058du, 0x15911c6du, 0xd0dba0efu, 0u, 0u, 0u, \
    0x0243f6f0u, 0x00243f6fu, 0x15120248u, 0x18a72658u, 0xd0dbb319u, 0u, 0u, 0u, \
    0x18cf81b2u, 0x0024168eu, 0xf6a50472u, 0x9414429bu, 0xd0dbc52eu, 0u, 0u, 0u, \
    0xfb823ee0u, 0x0023ee08u, 0x795f06a4u, 0xb60c9f44u, 0xd0dbd72fu, 0u, 0u, 0u, \
    0x767f70e8u, 0x0023c5deu, 0x63d1526bu, 0xac291efcu, 0xd0dbe91cu, 0u, 0u, 0u, \
    0x5b45023au, 0x00239e0du, 0x9260351eu, 0xa36a0dfcu, 0xd0dbfaf5u, 0u, 0u, 0u, \
    0x808dda52u, 0x00237694u, 0xe4ccf7c8u, 0xc839c7eau, 0xd0dc0cbau, 0u, 0u, 0u, \
    0xc234f72cu, 0x00234f72u, 0xe37daf56u, 0x466f4f15u, 0xd0dc1e6cu, 0u, 0u, 0u, \
    0x01194538u, 0x002328a7u, 0x60a59260u, 0x4950d56fu, 0xd0dc300au, 0u, 0u, 0u, \
    0x23023024u, 0x00230230u, 0xdb18b071u, 0xfb96379fu, 0xd0dc4194u, 0u, 0u, 0u, \
    0x1284e6f2u, 0x0022dc0du, 0x93916829u, 0x876b6a91u, 0xd0dc530cu, 0u, 0u, 0u, \
    0xbeea4e1au, 0x0022b63cu, 0x9c850835u, 0x1672dbc3u, 0xd0dc6471u, 0u, 0u, 0u, \
    0x1c159a76u, 0x002290beu, 0x7c6a5666u, 0xd1c7c4c8u, 0xd0dc75c2u, 0u, 0u, 0u, \
    0x226b9022u, 0x00226b90u, 0x47a4fa23u, 0xe2007234u, 0xd0dc8701u, 0u, 0u, 0u, \
    0xceba6066u, 0x002246b1u, 0x544a35adu, 0x6f307e58u, 0xd0dc982eu, 0u, 0u, 0u, \
    0x22222222u, 0x00222222u, 0x05d54566u, 0xa0eb000eu, 0xd0dca948u, 0u, 0u, 0u, \
    0x21fde022u, 0x0021fde0u, 0x7fdc24d2u, 0x9e44adeau, 0xd0dcba50u, 0u, 0u, 0u, \
    0xd7cd3920u, 0x0021d9eau, 0xe228a4a1u, 0x8dd5f617u, 0xd0dccb46u, 0u, 0u, 0u, \
    0x511e8d2cu, 0x0021b641u, 0x1b8ddb62u, 0x95bd0b26u, 0xd0dcdc2au, 0u, 0u, 0u, \
    0x9f79b476u, 0x002192e2u, 0x08b6c6a9u, 0xdb9fe614u, 0xd0dcecfcu, 0u, 0u, 0u, \
    0xd84b3b90u, 0x00216fcdu, 0x34575d73u, 0x84ae3dd3u, 0xd0dcfdbdu, 0u, 0u, 0u, \
    0x14d0214eu, 0x00214d02u, 0x97fb3330u, 0xb5a3748eu, 0xd0dd0e6cu, 0u, 0u, 0u, \
    0x720212a8u, 0x00212a7eu, 0x5d888432u, 0x92c87aecu, 0xd0dd1f0au, 0u, 0u, 0u, \
    0x10842108u, 0x00210842u, 0x5adecb5cu, 0x3ff5a98cu, 0xd0dd2f97u, 0u, 0u, 0u, \
    0x148fef8cu, 0x0020e64cu, 0x022d884au, 0xe0949103u, 0xd0dd4012u, 0u, 0u, 0u, \
    0xa5e353f8u, 0x0020c49bu, 0x4c311810u, 0x97a1c083u, 0xd0dd507du, 0u, 0u, 0u, \
    0xefae6808u, 0x0020a32fu, 0x6fec6034u, 0x87ae837bu, 0xd0dd60d7u, 0u, 0u, 0u, \
    0x20820820u, 0x00208208u, 0x8137bc58u, 0xd2e2964du, 0xd0dd7120u, 0u, 0u, 0u, \
    0x6a3ebc34u, 0x00206123u, 0x581e58e8u, 0x9afdd269u, 0xd0dd8159u, 0u, 0u, 0u, \
    0x02040810u, 0x00204081u, 0x8c0debb5u, 0x0159d1f1u, 0xd0dd9182u, 0u, 0u, 0u, \
    0x20202020u, 0x00202020u, 0x38e12bb2u, 0x26eb8b23u, 0xd0dda19au, 0u, 0u, 0u, \
    0x00000000u, 0x00200000u, 0x5e5f8540u, 0x2c44e3aeu, 0xd0ddb1a2u, 0u, 0u, 0u, \
    0x01fc07f0u, 0x001fc07fu, 0xf75bbca9u, 0x56aff415u, 0xd0ddd182u, 0u, 0u, 0u, \
    0x1f81f820u, 0x001f81f8u, 0xe5fec2f5u, 0x7da6dbb5u, 0xd0ddf123u, 0u, 0u, 0u, \
    0x9e4a4271u, 0x001f4465u, 0xf6042515u, 0x98643a72u, 0xd0de1086u, 0u, 0u, 0u, \
    0xf07c1f08u, 0x001f07c1u, 0x3f936930u, 0x987ec47au, 0xd0de2facu, 0u, 0u, 0u, \
    0xb301ecc0u, 0x001ecc07u, 0x9ba79019u, 0x6a14d999u, 0xd0de4e96u, 0u, 0u, 0u, \
    0xabf0b767u, 0x001e9131u, 0x56912cd5u, 0xf3f67a96u, 0xd0de6d44u, 0u, 0u, 0u, \
    0xc901e574u, 0x001e573au, 0x2873ede6u, 0x17cdaf3cu, 0xd0de8bb9u, 0u, 0u, 0u, \
    0x1e1e1e1eu, 0x001e1e1eu, 0xa16b6b8cu, 0xb2456ec3u, 0xd0dea9f3u, 0u, 0u, 0u, \
    0xe3f8868au, 0x001de5d6u, 0x92e5ab01u, 0x9b2f1b5cu, 0xd0dec7f5u, 0u, 0u, 0u, \
    0x76b981dbu, 0x001dae60u, 0x59891d77u, 0xa5a6a0cbu, 0xd0dee5bfu, 0u, 0u, 0u, \
    0x54b82c34u, 0x001d77b6u, 0x18f1fe27u, 0xa0354532u, 0xd0df0352u, 0u, 0u, 0u, \
    0x1d41d41du, 0x001d41d4u, 0x3c1dcedcu, 0x54f33a63u, 0xd0df20afu, 0u, 0u, 0u, \
    0x8f6ec074u, 0x001d0cb5u, 0x89ba5083u, 0x89a7fd60u, 0xd0df3dd6u, 0u, 0u, 0u, \
    0x89039b0bu, 0x001cd856u, 0x7ab04263u, 0xffe99104u, 0xd0df5ac8u, 0u, 0u, 0u, \
    0x055ee191u, 0x001ca4b3u, 0x90bce6bfu, 0x753aa022u, 0xd0df7787u, 0u, 0u, 0u, \
    0x1c71c71cu, 0x001c71c7u, 0xfcfe2dc0u, 0xa32792dcu, 0xd0df9412u, 0u, 0u, 0u, \
    0x01c3f8f0u, 0x001c3f8fu, 0x19026a5au, 0x3f62a25au, 0xd0dfb06bu, 0u, 0u, 0u, \
    0x0381c0e0u, 0x001c0e07u, 0xcb32736fu, 0xfbdef579u, 0xd0dfcc91u, 0u, 0u, 0u, \
    0x899406f7u, 0x001bdd2bu, 0x8e8045cdu, 0x86ead0a2u, 0xd0dfe887u, 0u, 0u, 0u, \
    0x14c1bad0u, 0x001bacf9u, 0x87e040ceu, 0x8b48e252u, 0xd0e0044cu, 0u, 0u, 0u, \
    0x3dda338bu, 0x001b7d6cu, 0xfed93819u, 0xb048b59cu, 0xd0e01fe1u, 0u, 0u, 0u, \
    0xb4e81b4fu, 0x001b4e81u, 0xe15a006au, 0x99de5351u, 0xd0e03b47u, 0u, 0u, 0u, \
    0x406c80d9u, 0x001b2036u, 0x53bc057bu, 0xe8b91a35u, 0xd0e0567eu, 0u, 0u, 0u, \
    0xbca1af28u, 0x001af286u, 0x176e0181u, 0x3a59d629u, 0xd0e07188u, 0u, 0u, 0u, \
    0x1ac5701bu, 0x001ac570u, 0xcd0a140cu, 0x29281df1u, 0xd0e08c64u, 0u, 0u, 0u, \
    0x606a63beu, 0x001a98efu, 0x35dbf2a6u, 0x4c86fecfu, 0xd0e0a713u, 0u, 0u, 0u, \
    0xa6d01a6du, 0x001a6d01u, 0x71638660u, 0x38e8fcd0u, 0xd0e0c196u, 0u, 0u, 0u, \
    0x1a41a41au, 0x001a41a4u, 0x1527ab4fu, 0x7fe36e85u, 0xd0e0dbedu, 0u, 0u, 0u, \
    0xf97a4b02u, 0x001a16d3u, 0x87866776u, 0xb0413a5au, 0xd0e0f619u, 0u, 0u, 0u, \
    0x951033d9u, 0x0019ec8eu, 0xcb795143u, 0x5614fbacu, 0xd0e1101bu, 0u, 0u, 0u, \
    0x4ee4a102u, 0x0019c2d1u, 0xe59ebf11u, 0xfaca9548u, 0xd0e129f2u, 0u, 0u, 0u, \
    0x9999999au, 0x00199999u, 0x53e44044u, 0x253836f2u, 0xd0e143a1u, 0u, 0u, 0u, \
    0xf80cb872u, 0x001970e4u, 0xd7d1a6edu, 0x59aedb20u, 0xd0e15d26u, 0u, 0u, 0u, \
    0xfcd6e9e0u, 0x001948b0u, 0x5b9cd640u, 0x1a0a420bu, 0xd0e17683u, 0u, 0u, 0u, \
    0x49d0e229u, 0x001920fbu, 0x0da2a10bu, 0xe5c06ed5u, 0xd0e18fb7u, 0u, 0u, 0u, \
    0x8f9c18fau, 0x0018f9c1u, 0x880a2e0eu, 0x39f0ab73u, 0xd0e1a8c5u, 0u, 0u, 0u, \
    0x8d3018d3u, 0x0018d301u, 0x96182434u, 0x917217beu, 0xd0e1c1abu, 0u, 0u, 0u, \
    0x0f6bf3aau, 0x0018acb9u, 0xfa3c8328u, 0x64e1c7e6u, 0xd0e1da6bu, 0u, 0u, 0u, \
    0xf0abb04au, 0x001886e5u, 0x5e876d6bu, 0x2ab07663u, 0xd0e1f305u, 0u, 0u, 0u, \
    0x18618618u, 0x00186186u, 0x1f46b735u, 0x572fcd32u, 0xd0e20b79u, 0u, 0u, 0u, \
    0x7ab2beddu, 0x00183c97u, 0x385128ddu, 0x5c9f4a2du, 0xd0e223c8u, 0u, 0u, 0u, \
    0x18181818u, 0x00181818u, 0xd6f0268fu, 0xab38c207u, 0xd0e23bf2u, 0u, 0u, 0u, \
    0xfd017f40u, 0x0017f405u, 0x760caa01u, 0xb13c8557u, 0xd0e253f8u, 0u, 0u, 0u, \
    0x417d05f4u, 0x0017d05fu, 0x956ab787u, 0xdafd2afau, 0xd0e26bdau, 0u, 0u, 0u, \
    0x08e0ecc3u, 0x0017ad22u, 0xccf0df14u, 0x92eb0303u, 0xd0e28399u, 0u, 0u, 0u, \
    0x8178a4c8u, 0x00178a4cu, 0xe02b52b3u, 0x419f3528u, 0xd0e29b35u, 0u, 0u, 0u, \
    0xe434a9b1u, 0x001767dcu, 0x4ea289dfu, 0x4de68da7u, 0xd0e2b2aeu, 0u, 0u, 0u, \
    0x745d1746u, 0x001745d1u, 0xdda2640eu, 0x1ccbfb5eu, 0xd0e2ca05u, 0u, 0u, 0u, \
    0x7f46debcu, 0x00172428u, 0x9932ab92u, 0x11a2c1d6u, 0xd0e2e13au, 0u, 0u, 0u, \
    0x5c0b8170u, 0x001702e0u, 0xc0d1d498u, 0x8e1061b9u, 0xd0e2f84du, 0u, 0u, 0u, \
    0x6b4337c7u, 0x0016e1f7u, 0x4e8632f3u, 0xf2163a49u, 0xd0e30f3fu, 0u, 0u, 0u, \
    0x16c16c17u, 0x0016c16cu, 0xc682e8c4u, 0x9c1ae620u, 0xd0e32611u, 0u, 0u, 0u, \

#endif /* NF_MATH_TABLES_H */
