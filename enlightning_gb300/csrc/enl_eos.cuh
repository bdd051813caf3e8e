// Equation of state in FP64 (update_state.m4:90-105), shared by the per-patch
// entry point, the batched engine's stage epilogue and its state exchange, so
// that they agree bit for bit.
//
// The FP64 pipe completes 2 operations per SM and clock, so pressure and
// temperature are arranged to need few of them: one seeded reciprocal of rho,
// constant divisors as factors, and the exponential and logarithm below (12
// FP64 operations each), which reduce their argument by a table of 256
// entries and finish with a Taylor polynomial.
#pragma once
#include <cmath>

#include "enl_rcp.cuh"

namespace enl {

// Table of the logarithm: the mantissa range [0.707, 1.414) in 256 steps of the
// high word; c is the double next to the reciprocal of the step's middle
// (exactly 1 on both sides of 1, so that log is accurate where its value is
// small) and the second entry the double next to -log(c).
__device__ const double2 kLogTable64[256] = {
    {0x1.6993f349cc726p+0, -0x1.61965cdb02c1ep-2}, {0x1.68954dd2390bap+0, -0x1.5ec433d5c35aep-2},
    {0x1.67980e0bf08c7p+0, -0x1.5bf406b543db1p-2}, {0x1.669c31075ab40p+0, -0x1.5925d2b112a59p-2},
    {0x1.65a1b3dd13357p+0, -0x1.565995069514cp-2}, {0x1.64a893adcd25fp+0, -0x1.538f4af8f72fcp-2},
    {0x1.63b0cda236e1cp+0, -0x1.50c6f1d11b97bp-2}, {0x1.62ba5eeade65ep+0, -0x1.4e0086dd8baccp-2},
    {0x1.61c544c0161c5p+0, -0x1.4b3c077267e9ap-2}, {0x1.60d17c61da198p+0, -0x1.487970e958771p-2},
    {0x1.5fdf0317b5c6fp+0, -0x1.45b8c0a17df12p-2}, {0x1.5eedd630a9fb3p+0, -0x1.42f9f3ff62641p-2},
    {0x1.5dfdf303137b6p+0, -0x1.403d086cea79bp-2}, {0x1.5d0f56ec91e57p+0, -0x1.3d81fb5946dbcp-2},
    {0x1.5c21ff51ef005p+0, -0x1.3ac8ca38e5c5dp-2}, {0x1.5b35e99f06714p+0, -0x1.3811728564cb2p-2},
    {0x1.5a4b1346add2bp+0, -0x1.355bf1bd82c8bp-2}, {0x1.596179c29d2cep+0, -0x1.32a84565120a9p-2},
    {0x1.58791a9357ccep+0, -0x1.2ff66b04ea9d5p-2}, {0x1.5791f34015792p+0, -0x1.2d46602adccefp-2},
    {0x1.56ac0156ac015p+0, -0x1.2a982269a3dbep-2}, {0x1.55c7426b79286p+0, -0x1.27ebaf58d8c9cp-2},
    {0x1.54e3b4194ce66p+0, -0x1.25410494e56c8p-2}, {0x1.5401540154015p+0, -0x1.22981fbef797ap-2},
    {0x1.53201fcb02fb1p+0, -0x1.1ff0fe7cf47a9p-2}, {0x1.5240152401524p+0, -0x1.1d4b9e796c245p-2},
    {0x1.516131c015161p+0, -0x1.1aa7fd638d33ep-2}, {0x1.508373590ec9cp+0, -0x1.180618ef18adep-2},
    {0x1.4fa6d7aeb597cp+0, -0x1.1565eed455fc2p-2}, {0x1.4ecb5c86b3d24p+0, -0x1.12c77cd00713cp-2},
    {0x1.4df0ffac83c01p+0, -0x1.102ac0a35cc1bp-2}, {0x1.4d17bef15cb4ep+0, -0x1.0d8fb813eb1efp-2},
    {0x1.4c3f982c20723p+0, -0x1.0af660eb9e278p-2}, {0x1.4b68893948d1cp+0, -0x1.085eb8f8ae799p-2},
    {0x1.4a928ffad5b5cp+0, -0x1.05c8be0d9635ap-2}, {0x1.49bdaa583b401p+0, -0x1.03346e0106062p-2},
    {0x1.48e9d63e504d1p+0, -0x1.00a1c6adda472p-2}, {0x1.4817119f3d325p+0, -0x1.fc218be620a5fp-3},
    {0x1.47455a726abf2p+0, -0x1.f702d36777df0p-3}, {0x1.4674aeb4717e9p+0, -0x1.f1e75fadf9bdep-3},
    {0x1.45a50c670938fp+0, -0x1.eccf2c8fe920bp-3}, {0x1.44d67190f8b43p+0, -0x1.e7ba35eb77e2ap-3},
    {0x1.4408dc3e05b22p+0, -0x1.e2a877a6b2c0fp-3}, {0x1.433c4a7ee52b4p+0, -0x1.dd99edaf6d7e9p-3},
    {0x1.4270ba692bc4dp+0, -0x1.d88e93fb2f451p-3}, {0x1.41a62a173e821p+0, -0x1.d38666871f467p-3},
    {0x1.40dc97a843ae8p+0, -0x1.ce816157f1985p-3}, {0x1.4014014014014p+0, -0x1.c97f8079d44ecp-3},
    {0x1.3f4c65072bf74p+0, -0x1.c480c0005cccfp-3}, {0x1.3e85c12a9d651p+0, -0x1.bf851c067555cp-3},
    {0x1.3dc013dc013dcp+0, -0x1.ba8c90ae4ad19p-3}, {0x1.3cfb5b51698ebp+0, -0x1.b5971a213acd9p-3},
    {0x1.3c3795c553afbp+0, -0x1.b0a4b48fc1b44p-3}, {0x1.3b74c1769aa5cp+0, -0x1.abb55c31693aep-3},
    {0x1.3ab2dca869b81p+0, -0x1.a6c90d44b704cp-3}, {0x1.39f1e5a22f36ep+0, -0x1.a1dfc40f1b7f1p-3},
    {0x1.3931daaf8f721p+0, -0x1.9cf97cdce0ec1p-3}, {0x1.3872ba2057e04p+0, -0x1.981634011aa74p-3},
    {0x1.37b4824872744p+0, -0x1.9335e5d594985p-3}, {0x1.36f7317fd9212p+0, -0x1.8e588ebac2dc1p-3},
    {0x1.363ac622898b1p+0, -0x1.897e2b17b19a6p-3}, {0x1.357f3e9078e5bp+0, -0x1.84a6b759f512dp-3},
    {0x1.34c4992d87fd9p+0, -0x1.7fd22ff599d4cp-3}, {0x1.340ad461776d3p+0, -0x1.7b0091651528bp-3},
    {0x1.3351ee97dbfc6p+0, -0x1.7631d82935a84p-3}, {0x1.3299e6401329ap+0, -0x1.716600c914055p-3},
    {0x1.31e2b9cd37dc2p+0, -0x1.6c9d07d203fc4p-3}, {0x1.312c67b6173eep+0, -0x1.67d6e9d785770p-3},
    {0x1.3076ee7525c2cp+0, -0x1.6313a37335d76p-3}, {0x1.2fc24c8874486p+0, -0x1.5e533144c1718p-3},
    {0x1.2f0e8071a5703p+0, -0x1.59958ff1d52f4p-3}, {0x1.2e5b88b5e3104p+0, -0x1.54dabc26105d3p-3},
    {0x1.2da963ddd3cfbp+0, -0x1.5022b292f6a45p-3}, {0x1.2cf8107590e67p+0, -0x1.4b6d6fefe22a5p-3},
    {0x1.2c478d0c9c013p+0, -0x1.46baf0f9f5db8p-3}, {0x1.2b97d835d548ep+0, -0x1.420b32740fdd6p-3},
    {0x1.2ae8f087718d0p+0, -0x1.3d5e3126bc281p-3}, {0x1.2a3ad49af0907p+0, -0x1.38b3e9e027477p-3},
    {0x1.298d830d13780p+0, -0x1.340c59741142dp-3}, {0x1.28e0fa7dd35a3p+0, -0x1.2f677cbbc0a98p-3},
    {0x1.2835399057efdp+0, -0x1.2ac55095f5c5bp-3}, {0x1.278a3eeaee650p+0, -0x1.2625d1e6ddf55p-3},
    {0x1.26e009370049cp+0, -0x1.2188fd9807266p-3}, {0x1.263697210aa18p+0, -0x1.1ceed09853755p-3},
    {0x1.258de75895121p+0, -0x1.185747dbecf34p-3}, {0x1.24e5f89029305p+0, -0x1.13c2605c398bfp-3},
    {0x1.243ec97d49eaep+0, -0x1.0f301717cf0fbp-3}, {0x1.239858d86b11fp+0, -0x1.0aa06912675d5p-3},
    {0x1.22f2a55ce8fc5p+0, -0x1.06135354d4b19p-3}, {0x1.224dadc900489p+0, -0x1.0188d2ecf613ep-3},
    {0x1.21a970ddc5ba7p+0, -0x1.fa01c9db57ce7p-4}, {0x1.2105ed5f1e336p+0, -0x1.f0f70cdd992e4p-4},
    {0x1.20632213b6c6dp+0, -0x1.e7f1691a32d3ap-4}, {0x1.1fc10dc4fce8bp+0, -0x1.def0d8d466dbbp-4},
    {0x1.1f1faf3f16b64p+0, -0x1.d5f55659210e1p-4}, {0x1.1e7f0550db594p+0, -0x1.ccfedbfee13a8p-4},
    {0x1.1ddf0ecbcb841p+0, -0x1.c40d6425a5cb4p-4}, {0x1.1d3fca840a074p+0, -0x1.bb20e936d6976p-4},
    {0x1.1ca13750547fep+0, -0x1.b23965a52ff04p-4}, {0x1.1c035409fc1dfp+0, -0x1.a956d3ecade60p-4},
    {0x1.1b661f8cde833p+0, -0x1.a0792e9277cadp-4}, {0x1.1ac998b75eb90p+0, -0x1.97a07024cbe6ep-4},
    {0x1.1a2dbe6a5e3e4p+0, -0x1.8ecc933aeb6e2p-4}, {0x1.19928f89362b7p+0, -0x1.85fd927506a46p-4},
    {0x1.18f80af9b06dcp+0, -0x1.7d33687c293c8p-4}, {0x1.185e2fa401186p+0, -0x1.746e100226edbp-4},
    {0x1.17c4fc72bfcb9p+0, -0x1.6bad83c1883bap-4}, {0x1.172c7052e1316p+0, -0x1.62f1be7d7774ap-4},
    {0x1.16948a33b08fap+0, -0x1.5a3abb01ade21p-4}, {0x1.15fd4906c96f1p+0, -0x1.5188742261311p-4},
    {0x1.1566abc011567p+0, -0x1.48dae4bc3101dp-4}, {0x1.14d0b155b19aep+0, -0x1.403207b414b79p-4},
    {0x1.143b58c01143bp+0, -0x1.378dd7f74970fp-4}, {0x1.13a6a0f9cf01ep+0, -0x1.2eee507b402ffp-4},
    {0x1.131288ffbb3b6p+0, -0x1.26536c3d8c36cp-4}, {0x1.127f0fd0d2295p+0, -0x1.1dbd2643d1913p-4},
    {0x1.11ec346e36092p+0, -0x1.152b799bb3cd0p-4}, {0x1.1159f5db29606p+0, -0x1.0c9e615ac4e19p-4},
    {0x1.10c8531d0952ep+0, -0x1.0415d89e7444bp-4}, {0x1.10374b3b480aap+0, -0x1.f723b517fc51fp-5},
    {0x1.0fa6dd3f67322p+0, -0x1.e624c4a0b5e15p-5}, {0x1.0f170834f27fap+0, -0x1.d52ed6405d87ap-5},
    {0x1.0e87cb297a51ep+0, -0x1.c441e06f72a93p-5}, {0x1.0df9252c8e5e6p+0, -0x1.b35dd9b58baa8p-5},
    {0x1.0d6b154fb86f9p+0, -0x1.a282b8a936174p-5}, {0x1.0cdd9aa677344p+0, -0x1.91b073efd7314p-5},
    {0x1.0c50b446391f3p+0, -0x1.80e7023d8ccc8p-5}, {0x1.0bc4614657569p+0, -0x1.70265a550e77bp-5},
    {0x1.0b38a0c010b39p+0, -0x1.5f6e73078efc3p-5}, {0x1.0aad71ce84d16p+0, -0x1.4ebf43349e26ap-5},
    {0x1.0a22d38eaf2bfp+0, -0x1.3e18c1ca0ae99p-5}, {0x1.0998c51f624d5p+0, -0x1.2d7ae5c3c5bb7p-5},
    {0x1.090f45a1430aap+0, -0x1.1ce5a62bc3540p-5}, {0x1.08865436c3cf7p+0, -0x1.0c58fa19dfaabp-5},
    {0x1.07fdf0041ff7cp+0, -0x1.f7a9b16782855p-6}, {0x1.0776182f57386p+0, -0x1.d6b272597981fp-6},
    {0x1.06eecbe029155p+0, -0x1.b5cc258b718e7p-6}, {0x1.06680a4010668p+0, -0x1.94f6b99a24473p-6},
    {0x1.05e1d27a3ee9cp+0, -0x1.74321d3d006d2p-6}, {0x1.055c23bb98e2ap+0, -0x1.537e3f45f354ep-6},
    {0x1.04d6fd32b0c7bp+0, -0x1.32db0ea132e10p-6}, {0x1.04525e0fc2fcbp+0, -0x1.12487a5507f68p-6},
    {0x1.03ce4584b19a0p+0, -0x1.e38ce30333100p-7}, {0x1.034ab2c50040dp+0, -0x1.a2a9c6c17044dp-7},
    {0x1.02c7a505cffbfp+0, -0x1.61e77e8b53f9fp-7}, {0x1.02451b7ddb2d2p+0, -0x1.2145e939ef1bcp-7},
    {0x1.01c315657186bp+0, -0x1.c189cbb0e283fp-8}, {0x1.014191f674111p+0, -0x1.40c8a7478788dp-8},
    {0x1.00c0906c513cfp+0, -0x1.809048289860ap-9}, {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.fd04794a10e6ap-1, 0x1.7ee11ebd82ec4p-8},
    {0x1.fb0c610d5e939p-1, 0x1.3e7295d25a7d5p-7}, {0x1.f9182b6813bafp-1, 0x1.bcf712c743853p-7},
    {0x1.f727cce5f530ap-1, 0x1.1d7f7eb9eebf1p-6}, {0x1.f53b3a3fa204ep-1, 0x1.5c45a51b8d393p-6},
    {0x1.f3526859b8cecp-1, 0x1.9ace7551cc515p-6}, {0x1.f16d4c4401f17p-1, 0x1.d91a66c543cbep-6},
    {0x1.ef8bdb389ebadp-1, 0x1.0b94f7c196173p-5}, {0x1.edae0a9b3d3a5p-1, 0x1.2a7ec2214e879p-5},
    {0x1.ebd3cff850b0cp-1, 0x1.494acc34d911dp-5}, {0x1.e9fd21044e799p-1, 0x1.67f94f094bd92p-5},
    {0x1.e829f39aef509p-1, 0x1.868a83083f6d0p-5}, {0x1.e65a3dbe74d6bp-1, 0x1.a4fe9ffa3d233p-5},
    {0x1.e48df596f3394p-1, 0x1.c355dd0921f2fp-5}, {0x1.e2c511719ee16p-1, 0x1.e19070c276010p-5},
    {0x1.e0ff87c01e100p-1, 0x1.ffae9119b92fbp-5}, {0x1.df3d4f17de4dbp-1, 0x1.0ed839b5526fep-4},
    {0x1.dd7e5e316d94cp-1, 0x1.1dcb263db1944p-4}, {0x1.dbc2abe7d71d4p-1, 0x1.2cb0283f5de22p-4},
    {0x1.da0a2f3803b41p-1, 0x1.3b87598b1b6f0p-4}, {0x1.d854df401d855p-1, 0x1.4a50d3aa1b03fp-4},
    {0x1.d6a2b33ef7448p-1, 0x1.590cafdf01c26p-4}, {0x1.d4f3a293769cap-1, 0x1.67bb0726ec0fbp-4},
    {0x1.d347a4bc01d34p-1, 0x1.765bf23a6be17p-4}, {0x1.d19eb155f08a4p-1, 0x1.84ef898e82828p-4},
    {0x1.cff8c01cff8c0p-1, 0x1.9375e55595edfp-4}, {0x1.ce55c8eac7900p-1, 0x1.a1ef1d8061cd8p-4},
    {0x1.ccb5c3b636e3ap-1, 0x1.b05b49bee4403p-4}, {0x1.cb18a8930de60p-1, 0x1.beba818146764p-4},
    {0x1.c97e6fb15e44dp-1, 0x1.cd0cdbf8c13e0p-4}, {0x1.c7e7115d0ce95p-1, 0x1.db5270187d925p-4},
    {0x1.c65285fd56843p-1, 0x1.e98b54967146bp-4}, {0x1.c4c0c61456a8ep-1, 0x1.f7b79fec37de2p-4},
    {0x1.c331ca3e91679p-1, 0x1.02ebb42bf3d4ap-3}, {0x1.c1a58b327f576p-1, 0x1.09f561ee719c4p-3},
    {0x1.c01c01c01c01cp-1, 0x1.10f8e422539b1p-3}, {0x1.be9526d0769fap-1, 0x1.17f6458fca611p-3},
    {0x1.bd10f365451b6p-1, 0x1.1eed90e2dc2c3p-3}, {0x1.bb8f609879493p-1, 0x1.25ded0abc6ad3p-3},
    {0x1.ba10679bd8488p-1, 0x1.2cca0f5f5f252p-3}, {0x1.b89401b89401cp-1, 0x1.33af575770e4dp-3},
    {0x1.b71a284ee6b34p-1, 0x1.3a8eb2d31a375p-3}, {0x1.b5a2d4d5b081fp-1, 0x1.41682bf727bbfp-3},
    {0x1.b42e00da17007p-1, 0x1.483bccce6e3dcp-3}, {0x1.b2bba5ff26a23p-1, 0x1.4f099f4a230b1p-3},
    {0x1.b14bbdfd760e6p-1, 0x1.55d1ad4232d70p-3}, {0x1.afde42a2cb482p-1, 0x1.5c940075972b9p-3},
    {0x1.ae732dd1c2a09p-1, 0x1.6350a28aaa759p-3}, {0x1.ad0a798177693p-1, 0x1.6a079d0f7aad0p-3},
    {0x1.aba41fbd2e5b1p-1, 0x1.70b8f97a1aa74p-3}, {0x1.aa401aa401aa4p-1, 0x1.7764c128f2127p-3},
    {0x1.a8de64688ebabp-1, 0x1.7e0afd630c276p-3}, {0x1.a77ef750a56dap-1, 0x1.84abb75865137p-3},
    {0x1.a621cdb4f8fdfp-1, 0x1.8b46f8223625bp-3}, {0x1.a4c6e200d2637p-1, 0x1.91dcc8c340bdfp-3},
    {0x1.a36e2eb1c432dp-1, 0x1.986d3228180c8p-3}, {0x1.a217ae575ff2fp-1, 0x1.9ef83d2769a34p-3},
    {0x1.a0c35b92ecdf1p-1, 0x1.a57df28244dcbp-3}, {0x1.9f713117200d0p-1, 0x1.abfe5ae46124ap-3},
    {0x1.9e2129a7d5f0ap-1, 0x1.b2797ee46320cp-3}, {0x1.9cd34019cd340p-1, 0x1.b8ef670420c3bp-3},
    {0x1.9b876f5262dd1p-1, 0x1.bf601bb0e44e0p-3}, {0x1.9a3db2474fb98p-1, 0x1.c5cba543ae424p-3},
    {0x1.98f603fe670a0p-1, 0x1.cc320c0176501p-3}, {0x1.97b05f8d56652p-1, 0x1.d293581b6b3e7p-3},
    {0x1.966cc01966cc0p-1, 0x1.d8ef91af31d5ep-3}, {0x1.952b20d73ee97p-1, 0x1.df46c0c722d30p-3},
    {0x1.93eb7d0aa6759p-1, 0x1.e598ed5a87e2ep-3}, {0x1.92add0064ab74p-1, 0x1.ebe61f4dd7b0bp-3},
    {0x1.9172152b841ddp-1, 0x1.f22e5e72f105cp-3}, {0x1.903847ea1cec1p-1, 0x1.f871b28955045p-3},
    {0x1.8f0063c018f00p-1, 0x1.feb0233e607cep-3}, {0x1.8dca64397e408p-1, 0x1.0274dc16c232fp-2},
    {0x1.8c9644f01efbcp-1, 0x1.058f3c703ebc5p-2}, {0x1.8b64018b64019p-1, 0x1.08a73667c57aep-2},
    {0x1.8a3395c018a34p-1, 0x1.0bbccdb0d24bcp-2}, {0x1.8904fd503744bp-1, 0x1.0ed005f657da5p-2},
    {0x1.87d8340ab6e97p-1, 0x1.11e0e2dad9cb6p-2}, {0x1.86ad35cb59a84p-1, 0x1.14ef67f88685ap-2},
    {0x1.8583fe7a7c018p-1, 0x1.17fb98e15095ep-2}, {0x1.845c8a0ce5129p-1, 0x1.1b05791f07b4ap-2},
    {0x1.8336d48397a24p-1, 0x1.1e0d0c33716bdp-2}, {0x1.8212d9eba4018p-1, 0x1.211255986160cp-2},
    {0x1.80f0965dfabcbp-1, 0x1.241558bfd1405p-2}, {0x1.7fd005ff40180p-1, 0x1.27161913f853dp-2},
    {0x1.7eb124ffa053bp-1, 0x1.2a1499f762bcap-2}, {0x1.7d93ef9aa4b46p-1, 0x1.2d10dec508582p-2},
    {0x1.7c7862170949fp-1, 0x1.300aead06350cp-2}, {0x1.7b5e78c693733p-1, 0x1.3302c1658658ap-2},
    {0x1.7a463005e918cp-1, 0x1.35f865c93293ep-2}, {0x1.792f843c689c3p-1, 0x1.38ebdb38ed320p-2},
    {0x1.781a71dc01782p-1, 0x1.3bdd24eb14b69p-2}, {0x1.7706f5610d8d0p-1, 0x1.3ecc460ef5f50p-2},
    {0x1.75f50b522b17cp-1, 0x1.41b941cce0beep-2}, {0x1.74e4b040174e5p-1, 0x1.44a41b463c47bp-2},
    {0x1.73d5e0c5899f7p-1, 0x1.478cd5959b3d8p-2}, {0x1.72c899870f91fp-1, 0x1.4a7373cecf997p-2},
    {0x1.71bcd732e940ap-1, 0x1.4d57f8fefe27fp-2}, {0x1.70b29680e66fap-1, 0x1.503a682cb1cb3p-2},
    {0x1.6fa9d43244380p-1, 0x1.531ac457ee77fp-2}, {0x1.6ea28d118b474p-1, 0x1.55f9107a43ee2p-2},
    {0x1.6d9cbdf26eaefp-1, 0x1.58d54f86e02f3p-2}, {0x1.6c9863b1ab429p-1, 0x1.5baf846aa1b1ap-2},
    {0x1.6b957b34e7803p-1, 0x1.5e87b20c2954ap-2}, {0x1.6a94016a94017p-1, 0x1.615ddb4bec13cp-2},
};
// 2^(i / 256), and what its rounding left out, relative to it.
__device__ const double2 kExpTable64[256] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.00b1afa5abcbfp+0, -0x1.4e82fc61851acp-55},
    {0x1.0163da9fb3335p+0, 0x1.b3b4f1a88bf6ep-54}, {0x1.02168143b0281p+0, -0x1.2985dd8521d32p-55},
    {0x1.02c9a3e778061p+0, -0x1.160139cd8dc5dp-56}, {0x1.037d42e11bbccp+0, 0x1.51e617061bfbdp-57},
    {0x1.04315e86e7f85p+0, -0x1.05e7a108766d1p-54}, {0x1.04e5f72f654b1p+0, 0x1.45fad437fa426p-55},
    {0x1.059b0d3158574p+0, 0x1.cd2523567f613p-55}, {0x1.0650a0e3c1f89p+0, -0x1.54529642b232fp-54},
    {0x1.0706b29ddf6dep+0, -0x1.bce8023f98efap-55}, {0x1.07bd42b72a836p+0, 0x1.293708ef5c32ep-55},
    {0x1.0874518759bc8p+0, 0x1.0f74e61e6c861p-57}, {0x1.092bdf66607e0p+0, -0x1.5b9280905b2a4p-54},
    {0x1.09e3ecac6f383p+0, 0x1.0a3e45b33d399p-54}, {0x1.0a9c79b1f3919p+0, 0x1.4f31f32c4b7e7p-55},
    {0x1.0b5586cf9890fp+0, 0x1.79aa65d837b6dp-54}, {0x1.0c0f145e46c85p+0, 0x1.407fb30d06420p-54},
    {0x1.0cc922b7247f7p+0, 0x1.eb51a92fdeffcp-55}, {0x1.0d83b23395decp+0, -0x1.a5d04b3b9911bp-54},
    {0x1.0e3ec32d3d1a2p+0, 0x1.ebe3d702f9cd1p-60}, {0x1.0efa55fdfa9c5p+0, -0x1.37a01f0739546p-54},
    {0x1.0fb66affed31bp+0, -0x1.a033489906e0bp-57}, {0x1.1073028d7233ep+0, 0x1.b8268b04ef0a5p-55},
    {0x1.11301d0125b51p+0, -0x1.556522a2fbd0ep-54}, {0x1.11edbab5e2ab6p+0, -0x1.ac46e44a2ebccp-54},
    {0x1.12abdc06c31ccp+0, -0x1.080ef8c4eea55p-58}, {0x1.136a814f204abp+0, -0x1.5704e90c9f860p-57},
    {0x1.1429aaea92de0p+0, -0x1.1c923b9d5f416p-54}, {0x1.14e95934f312ep+0, -0x1.97cea57e46280p-55},
    {0x1.15a98c8a58e51p+0, 0x1.0d3e3e95c55afp-55}, {0x1.166a45471c3c2p+0, 0x1.6f01429e2b9d2p-58},
    {0x1.172b83c7d517bp+0, -0x1.01b15eaa59348p-55}, {0x1.17ed48695bbc0p+0, 0x1.e653b2459034bp-57},
    {0x1.18af9388c8deap+0, -0x1.f1ff055de323dp-55}, {0x1.1972658375d2fp+0, 0x1.2cc7ea345b7dcp-54},
    {0x1.1a35beb6fcb75p+0, 0x1.b898c3f1353bfp-55}, {0x1.1af99f8138a1cp+0, 0x1.57bfb2876ea9ep-54},
    {0x1.1bbe084045cd4p+0, -0x1.6d99c7611eb26p-54}, {0x1.1c82f95281c6bp+0, 0x1.cdc1873af2155p-55},
    {0x1.1d4873168b9aap+0, 0x1.aecf73e3a2f60p-54}, {0x1.1e0e75eb44027p+0, -0x1.493684653a131p-54},
    {0x1.1ed5022fcd91dp+0, -0x1.fe782cb86389dp-55}, {0x1.1f9c18438ce4dp+0, -0x1.8e2899077520ap-54},
    {0x1.2063b88628cd6p+0, 0x1.a6f4144a6c38dp-55}, {0x1.212be3578a819p+0, 0x1.120fcd4f59273p-54},
    {0x1.21f49917ddc96p+0, 0x1.07a05b0e4047dp-55}, {0x1.22bdda27912d1p+0, 0x1.9b788c188c9b8p-55},
    {0x1.2387a6e756238p+0, 0x1.68efde3a8a894p-54}, {0x1.2451ffb82140ap+0, 0x1.77afbca90ef84p-55},
    {0x1.251ce4fb2a63fp+0, 0x1.75e18f274487dp-55}, {0x1.25e85711ece75p+0, 0x1.1512f082876eep-54},
    {0x1.26b4565e27cddp+0, 0x1.0472b981fe7f2p-55}, {0x1.2780e341ddf29p+0, 0x1.a02f0c7d75ec6p-54},
    {0x1.284dfe1f56381p+0, -0x1.6b87b3f71085ep-54}, {0x1.291ba7591bb70p+0, -0x1.03297e78260bfp-55},
    {0x1.29e9df51fdee1p+0, 0x1.2f7e16d09ab31p-55}, {0x1.2ab8a66d10f13p+0, -0x1.5b77e5ccd9fbfp-54},
    {0x1.2b87fd0dad990p+0, -0x1.d219b1a6fbffap-60}, {0x1.2c57e39771b2fp+0, -0x1.1e75c40b4251ep-54},
    {0x1.2d285a6e4030bp+0, 0x1.b3782720c0ab4p-55}, {0x1.2df961f641589p+0, 0x1.8a911f1f7785ap-54},
    {0x1.2ecafa93e2f56p+0, 0x1.e149289cecb8fp-57}, {0x1.2f9d24abd886bp+0, -0x1.1e7c998db7dbbp-57},
    {0x1.306fe0a31b715p+0, 0x1.34d754db0abb6p-55}, {0x1.31432edeeb2fdp+0, 0x1.5425c11faadf4p-55},
    {0x1.32170fc4cd831p+0, 0x1.64201e2ac744cp-55}, {0x1.32eb83ba8ea32p+0, -0x1.79517a03e2847p-54},
    {0x1.33c08b26416ffp+0, 0x1.fdd395dd3f84ap-55}, {0x1.3496266e3fa2dp+0, -0x1.00e2a46da4beep-55},
    {0x1.356c55f929ff1p+0, -0x1.6a3803b8e5b04p-55}, {0x1.36431a2de883bp+0, -0x1.7430803972b34p-55},
    {0x1.371a7373aa9cbp+0, -0x1.24aedcc4b5068p-54}, {0x1.37f26231e754ap+0, -0x1.54de30ae02d94p-54},
    {0x1.38cae6d05d866p+0, -0x1.907f81b512d8ep-54}, {0x1.39a401b7140efp+0, -0x1.4f2487e1c03ecp-54},
    {0x1.3a7db34e59ff7p+0, -0x1.1d1e83e9436d2p-56}, {0x1.3b57fbfec6cf4p+0, 0x1.14a5432fcb2f4p-54},
    {0x1.3c32dc313a8e5p+0, -0x1.91919b3ce1b15p-54}, {0x1.3d0e544ede173p+0, 0x1.9c3bba5562a2fp-56},
    {0x1.3dea64c123422p+0, 0x1.59f48a72a4c6dp-55}, {0x1.3ec70df1c5175p+0, -0x1.5a71612e21658p-55},
    {0x1.3fa4504ac801cp+0, -0x1.312607a28698ap-54}, {0x1.40822c367a024p+0, 0x1.6421f6f1d24d6p-55},
    {0x1.4160a21f72e2ap+0, -0x1.8a78f4817895bp-58}, {0x1.423fb2709468ap+0, -0x1.348a6815fce65p-54},
    {0x1.431f5d950a897p+0, -0x1.c2c9b67499a1bp-56}, {0x1.43ffa3f84b9d4p+0, 0x1.35c43984d9871p-55},
    {0x1.44e086061892dp+0, 0x1.363ed60c2ac11p-59}, {0x1.45c2042a7d232p+0, -0x1.32afc8d9473a0p-57},
    {0x1.46a41ed1d0057p+0, 0x1.666093b0664efp-54}, {0x1.4786d668b3237p+0, -0x1.5fc5e44de020ep-54},
    {0x1.486a2b5c13cd0p+0, 0x1.ecce1daa10379p-57}, {0x1.494e1e192aed2p+0, -0x1.ea0148327c42fp-56},
    {0x1.4a32af0d7d3dep+0, 0x1.3ff8e3f0f1230p-54}, {0x1.4b17dea6db7d7p+0, -0x1.a843ad1a88022p-56},
    {0x1.4bfdad5362a27p+0, 0x1.690cebb7aafb0p-56}, {0x1.4ce41b817c114p+0, 0x1.92ca3bf144e63p-55},
    {0x1.4dcb299fddd0dp+0, 0x1.31dbdeb54e077p-54}, {0x1.4eb2d81d8abffp+0, -0x1.02c99b04aa8b0p-54},
    {0x1.4f9b2769d2ca7p+0, -0x1.f94340071a38ep-55}, {0x1.508417f4531eep+0, 0x1.3e34f67e67118p-56},
    {0x1.516daa2cf6642p+0, -0x1.7deccdc93a349p-55}, {0x1.5257de83f4eefp+0, -0x1.5a3b1197ba0f0p-56},
    {0x1.5342b569d4f82p+0, -0x1.8dec6bd0f385fp-56}, {0x1.542e2f4f6ad27p+0, 0x1.1bd2888075068p-55},
    {0x1.551a4ca5d920fp+0, -0x1.61246ec7b5cf6p-55}, {0x1.56070dde910d2p+0, -0x1.96be8ae89ef8fp-55},
    {0x1.56f4736b527dap+0, 0x1.3350518fdd78ep-54}, {0x1.57e27dbe2c4cfp+0, -0x1.8e6ac90348602p-55},
    {0x1.58d12d497c7fdp+0, 0x1.b98b72f8a9b05p-56}, {0x1.59c0827ff07ccp+0, -0x1.1af7f1365c3acp-54},
    {0x1.5ab07dd485429p+0, 0x1.063e1e21c5409p-54}, {0x1.5ba11fba87a03p+0, -0x1.43a3540d1898ap-54},
    {0x1.5c9268a5946b7p+0, 0x1.4c7855019c6eap-60}, {0x1.5d84590998b93p+0, -0x1.51f58ddaa8090p-54},
    {0x1.5e76f15ad2148p+0, 0x1.432e62b64c035p-54}, {0x1.5f6a320dceb71p+0, -0x1.2e1648e50a17cp-55},
    {0x1.605e1b976dc09p+0, -0x1.ce44a6199769fp-55}, {0x1.6152ae6cdf6f4p+0, 0x1.5f30eda98a575p-54},
    {0x1.6247eb03a5585p+0, -0x1.c33c53bef4da8p-55}, {0x1.633dd1d1929fdp+0, 0x1.17ecda8a72159p-54},
    {0x1.6434634ccc320p+0, -0x1.45378892be9aep-55}, {0x1.652b9febc8fb7p+0, -0x1.345f3cee1ae6ep-54},
    {0x1.6623882552225p+0, -0x1.3cedd78565858p-54}, {0x1.671c1c70833f6p+0, -0x1.5c33fdf910406p-55},
    {0x1.68155d44ca973p+0, 0x1.710aa807e1964p-58}, {0x1.690f4b19e9538p+0, 0x1.1079ab5789604p-55},
    {0x1.6a09e667f3bcdp+0, -0x1.3b3efbf5e2228p-54}, {0x1.6b052fa75173ep+0, 0x1.27df161cd7778p-56},
    {0x1.6c012750bdabfp+0, -0x1.a12ad8734b982p-57}, {0x1.6cfdcddd47645p+0, 0x1.3f9924a05b767p-54},
    {0x1.6dfb23c651a2fp+0, -0x1.367efb86da9eep-57}, {0x1.6ef9298593ae5p+0, -0x1.7557939a8b5efp-55},
    {0x1.6ff7df9519484p+0, -0x1.0dc3d54e08851p-55}, {0x1.70f7466f42e87p+0, 0x1.1ed2f56fa9d1ap-58},
    {0x1.71f75e8ec5f74p+0, -0x1.81f647e5a3ecfp-56}, {0x1.72f8286ead08ap+0, -0x1.8e67a9006c909p-55},
    {0x1.73f9a48a58174p+0, -0x1.6ee4ac08b7db0p-55}, {0x1.74fbd35d7cbfdp+0, 0x1.6597566977ac8p-55},
    {0x1.75feb564267c9p+0, -0x1.619321e55e68ap-55}, {0x1.77024b1ab6e09p+0, 0x1.2c0b7028a5c3ap-54},
    {0x1.780694fde5d3fp+0, 0x1.09ccb5e09d4d3p-54}, {0x1.790b938ac1cf6p+0, 0x1.a30faf49cc78cp-55},
    {0x1.7a11473eb0187p+0, -0x1.b32dcb94da51dp-56}, {0x1.7b17b0976cfdbp+0, -0x1.2dad3519d7b5bp-54},
    {0x1.7c1ed0130c132p+0, 0x1.4ecfd5467c06bp-54}, {0x1.7d26a62ff86f0p+0, 0x1.7d51410fd15c2p-55},
    {0x1.7e2f336cf4e62p+0, 0x1.5ebe1abd66c55p-57}, {0x1.7f3878491c491p+0, -0x1.60a3629969871p-56},
    {0x1.80427543e1a12p+0, -0x1.8a1c52fb3cf42p-55}, {0x1.814d2add106d9p+0, 0x1.b18c6e3fdef5dp-55},
    {0x1.82589994cce13p+0, -0x1.369b6f13b3734p-54}, {0x1.8364c1eb941f7p+0, 0x1.0ec1ddcb1390ap-54},
    {0x1.8471a4623c7adp+0, -0x1.05e843a19ff1ep-55}, {0x1.857f4179f5b21p+0, -0x1.22cea4f3afa1ep-58},
    {0x1.868d99b4492edp+0, -0x1.4d450d872576ep-54}, {0x1.879cad931a436p+0, 0x1.c88549b958471p-56},
    {0x1.88ac7d98a6699p+0, 0x1.0ad675b0e8a00p-54}, {0x1.89bd0a478580fp+0, 0x1.31143962f7877p-54},
    {0x1.8ace5422aa0dbp+0, 0x1.db72fc1f0eab4p-55}, {0x1.8be05bad61778p+0, 0x1.3e9e96f112479p-54},
    {0x1.8cf3216b5448cp+0, -0x1.5b6609cc5e7ffp-57}, {0x1.8e06a5e0866d9p+0, -0x1.dac42a4a38df0p-55},
    {0x1.8f1ae99157736p+0, 0x1.bf68359f35f44p-56}, {0x1.902fed0282c8ap+0, 0x1.b99dd98b1ed84p-55},
    {0x1.9145b0b91ffc6p+0, -0x1.3091fa71e3d83p-54}, {0x1.925c353aa2fe2p+0, -0x1.885ad50cbb750p-56},
    {0x1.93737b0cdc5e5p+0, -0x1.da9b88b6c1e29p-58}, {0x1.948b82b5f98e5p+0, -0x1.2d5e85f3e0301p-55},
    {0x1.95a44cbc8520fp+0, -0x1.c23f97c90b959p-57}, {0x1.96bdd9a7670b3p+0, -0x1.1669428996971p-58},
    {0x1.97d829fde4e50p+0, -0x1.2434322f4f9aap-54}, {0x1.98f33e47a22a2p+0, 0x1.1f2b2c1c4c014p-56},
    {0x1.9a0f170ca07bap+0, -0x1.5ca6cd7668e4bp-55}, {0x1.9b2bb4d53fe0dp+0, -0x1.294f304f166b6p-54},
    {0x1.9c49182a3f090p+0, 0x1.1affc2b91ce27p-56}, {0x1.9d674194bb8d5p+0, -0x1.a1e58414c07d3p-55},
    {0x1.9e86319e32323p+0, 0x1.dd235e10a73bbp-57}, {0x1.9fa5e8d07f29ep+0, -0x1.9740b58a20091p-56},
    {0x1.a0c667b5de565p+0, -0x1.7c50422622263p-55}, {0x1.a1e7aed8eb8bbp+0, 0x1.165830a2b96c2p-54},
    {0x1.a309bec4a2d33p+0, 0x1.b1c86e3e231d5p-55}, {0x1.a42c980460ad8p+0, -0x1.03d5cbe27874bp-54},
    {0x1.a5503b23e255dp+0, -0x1.1bbd1d3bcbb15p-54}, {0x1.a674a8af46052p+0, 0x1.986178980fce0p-58},
    {0x1.a799e1330b358p+0, 0x1.0cc319cee31d2p-54}, {0x1.a8bfe53c12e59p+0, -0x1.9472975b1f2a5p-55},
    {0x1.a9e6b5579fdbfp+0, 0x1.469846e735ab3p-55}, {0x1.ab0e521356ebap+0, 0x1.d8157a34b7e7fp-56},
    {0x1.ac36bbfd3f37ap+0, -0x1.2dfcd978e9db4p-55}, {0x1.ad5ff3a3c2774p+0, 0x1.c8a4e231ebb7dp-55},
    {0x1.ae89f995ad3adp+0, 0x1.c1a7792cb3387p-55}, {0x1.afb4ce622f2ffp+0, -0x1.88c8d11a142e5p-55},
    {0x1.b0e07298db666p+0, -0x1.07b8f4ad1d9fap-54}, {0x1.b20ce6c9a8952p+0, 0x1.89c2ea41433c7p-55},
    {0x1.b33a2b84f15fbp+0, -0x1.5c3d956dcaebap-58}, {0x1.b468415b749b1p+0, -0x1.274aedac8ff80p-56},
    {0x1.b59728de5593ap+0, -0x1.0a40e3da6f640p-54}, {0x1.b6c6e29f1c52ap+0, 0x1.5c620ce76df06p-55},
    {0x1.b7f76f2fb5e47p+0, -0x1.8d6f438ad9334p-57}, {0x1.b928cf22749e4p+0, -0x1.fda52e1b51e41p-55},
    {0x1.ba5b030a1064ap+0, -0x1.1eee26b588a35p-54}, {0x1.bb8e0b79a6f1fp+0, -0x1.2141a7b3e2cd8p-60},
    {0x1.bcc1e904bc1d2p+0, 0x1.4ffd70a5fddcdp-56}, {0x1.bdf69c3f3a207p+0, -0x1.02899507554e5p-60},
    {0x1.bf2c25bd71e09p+0, -0x1.1bdfbfa9298acp-54}, {0x1.c06286141b33dp+0, -0x1.0dda2d4c0010cp-55},
    {0x1.c199bdd85529cp+0, 0x1.36eae30af0cb3p-56}, {0x1.c2d1cd9fa652cp+0, -0x1.a007daadf8d68p-55},
    {0x1.c40ab5fffd07ap+0, 0x1.ee3325c9ffd94p-55}, {0x1.c544778fafb22p+0, 0x1.36909391181d3p-55},
    {0x1.c67f12e57d14bp+0, 0x1.4e08fd10959acp-55}, {0x1.c7ba88988c933p+0, -0x1.11cd7dbdf9547p-55},
    {0x1.c8f6d9406e7b5p+0, 0x1.3cdaf384e1a67p-57}, {0x1.ca3405751c4dbp+0, -0x1.ac28b7bef6621p-56},
    {0x1.cb720dcef9069p+0, 0x1.76b2c6c921968p-57}, {0x1.ccb0f2e6d1675p+0, -0x1.030587207b9e1p-56},
    {0x1.cdf0b555dc3fap+0, -0x1.08a1883ccb5d2p-55}, {0x1.cf3155b5bab74p+0, -0x1.cc734592af7fcp-55},
    {0x1.d072d4a07897cp+0, -0x1.fad5d3ffffa6fp-55}, {0x1.d1b532b08c968p+0, 0x1.7752a44f587e8p-55},
    {0x1.d2f87080d89f2p+0, -0x1.00dae3875a949p-54}, {0x1.d43c8eacaa1d6p+0, 0x1.5b66fefeef52ep-55},
    {0x1.d5818dcfba487p+0, 0x1.4a385a63d07a7p-56}, {0x1.d6c76e862e6d3p+0, 0x1.159d9d908a96ep-58},
    {0x1.d80e316c98398p+0, -0x1.2919e2040220fp-55}, {0x1.d955d71ff6075p+0, 0x1.c254d16117a68p-55},
    {0x1.da9e603db3285p+0, 0x1.e5a50d5c192acp-55}, {0x1.dbe7cd63a8315p+0, -0x1.d8c329fbd0e03p-55},
    {0x1.dd321f301b460p+0, 0x1.43a59ac016b4bp-55}, {0x1.de7d5641c0658p+0, -0x1.ea6e6fbd5f2a6p-55},
    {0x1.dfc97337b9b5fp+0, -0x1.2d52107b43e1fp-55}, {0x1.e11676b197d17p+0, -0x1.3e8e3eab2cbb4p-57},
    {0x1.e264614f5a129p+0, -0x1.92ab93b470dc9p-55}, {0x1.e3b333b16ee12p+0, -0x1.b7966cd0d2cd9p-55},
    {0x1.e502ee78b3ff6p+0, 0x1.4b604603a88d3p-56}, {0x1.e653924676d76p+0, -0x1.76caa4c2ff1cfp-56},
    {0x1.e7a51fbc74c83p+0, 0x1.3c5ec519d7271p-55}, {0x1.e8f7977cdb740p+0, -0x1.1d5fc525d9940p-55},
    {0x1.ea4afa2a490dap+0, -0x1.ff7128fd391f0p-55}, {0x1.eb9f4867cca6ep+0, 0x1.55cd8aaea3d21p-55},
    {0x1.ecf482d8e67f1p+0, -0x1.dae98e223747dp-55}, {0x1.ee4aaa2188510p+0, 0x1.269947c2bed4ap-55},
    {0x1.efa1bee615a27p+0, 0x1.ec3bc41aa2008p-55}, {0x1.f0f9c1cb6412ap+0, -0x1.3b6137e9afe9ep-55},
    {0x1.f252b376bba97p+0, 0x1.42b94c3a9eb32p-55}, {0x1.f3ac948dd7274p+0, -0x1.9fa74878ba7c7p-57},
    {0x1.f50765b6e4540p+0, 0x1.a64a931d185eep-55}, {0x1.f6632798844f8p+0, 0x1.01f3a75ee0efep-54},
    {0x1.f7bfdad9cbe14p+0, -0x1.e37bae43be3edp-55}, {0x1.f91d802243c89p+0, -0x1.16a9ce6ed84fap-58},
    {0x1.fa7c1819e90d8p+0, 0x1.7893b4d91cd9dp-56}, {0x1.fbdba3692d514p+0, -0x1.99c7db2effc76p-57},
    {0x1.fd3c22b8f71f1p+0, 0x1.305c14160cc89p-58}, {0x1.fe9d96b2a23d9p+0, 0x1.4b458677f9840p-57},
};

// log(x + e) for positive normal x and e its rounding error (|e| at most half a
// unit of x).  x = 2^k m, r = m c - 1 with |r| < 2^-8, and log(1 + r) by its
// Taylor series to r^7 (the next term is below 2^-67); absolute error below
// 2^-53 max(1, |k|), relative error below 2^-52 near 1.
__device__ __forceinline__ double log64(double x, double e) {
  const int hi = __double2hiint(x);
  const int k = (hi - 0x3fe6a000) >> 20;
  const int hm = hi - (k << 20);
  const double2 t = kLogTable64[(hm - 0x3fe6a000) >> 12];
  double r = __fma_rn(__hiloint2double(hm, __double2loint(x)), t.x, -1.0);
  if (k == 0) r = __fma_rn(e, t.x, r);
  double p = __fma_rn(r, 1.0 / 7.0, -1.0 / 6.0);
  p = __fma_rn(p, r, 0.2);
  p = __fma_rn(p, r, -0.25);
  p = __fma_rn(p, r, 1.0 / 3.0);
  p = __fma_rn(p, r, -0.5);
  double y = __fma_rn(p, __dmul_rn(r, r), r);
  y = __dadd_rn(t.y, y);
  return k == 0 ? y : __fma_rn((double)k, 0x1.62e42fefa39efp-1, y);
}

// exp(a) for |a| < 700: a = (256 k + i) ln2 / 256 + r with |r| < 0.00136, and
// 2^k 2^(i/256) (1 + r + ... + r^5/120) (the next term is below 2^-66).
// Relative error below 1 unit in the last place.
__device__ __forceinline__ double exp64(double a) {
  constexpr double kMagic = 0x1.8p52;
  const double t = __fma_rn(a, 0x1.71547652b82fep+8, kMagic);
  const int n = __double2loint(t);
  const double d = __dadd_rn(t, -kMagic);
  double r = __fma_rn(d, -0x1.62e42fee00000p-9, a);
  r = __fma_rn(d, -0x1.a39ef35793c76p-41, r);
  const double2 s = kExpTable64[n & 255];
  r = __dadd_rn(r, s.y);
  double p = __fma_rn(r, 1.0 / 120.0, 1.0 / 24.0);
  p = __fma_rn(p, r, 1.0 / 6.0);
  p = __fma_rn(p, r, 0.5);
  p = __fma_rn(p, __dmul_rn(r, r), r);
  const double y = __fma_rn(s.x, p, s.x);
  return __hiloint2double(__double2hiint(y) + ((n >> 8) << 20), __double2loint(y));
}

struct EosConst64 {
  double rho0, c, c_lr, gm1_over_2rho0, inv_c_p, p0, T0, c_v, R, inv_c_v, inv_rho0, R_over_c_v;
  double a0;  // R / c_v times the relative rounding error of 1/rho0
};
inline EosConst64 make_eos_const64(double rho0, double c, double c_lr, double gamma1, double c_p, double p0, double T0,
                                   double c_v, double R) {
  return EosConst64{rho0, c, c_lr, (gamma1 - 1.0) / (2.0 * rho0), 1.0 / c_p, p0, T0, c_v, R, 1.0 / c_v, 1.0 / rho0,
                    R / c_v,
                    (R / c_v) * std::fma(-rho0, 1.0 / rho0, 1.0)};
}

// Any density and entropy (zero, negative, non-finite, far from ambient): .x the
// temperature; .y the pressure's term rho / c_p (rho s / rho) where it is not
// finite (a zero or infinite density, an entropy per mass beyond the range),
// which the sum of eos64 without that quotient has to take on, else 0.
static __device__ __noinline__ double2 state_general64(const EosConst64& E, double w0, double w3) {
  const double s = w3 / w0, q = w0 * E.inv_c_p * s;
  return double2{E.T0 * exp((s - E.R * log(E.rho0 / w0)) / E.c_v), isfinite(q) ? 0.0 : q};
}

// p and T of a cell; height = centre height of the cell row.  Every operation
// is explicitly rounded: no contraction differences between call sites.
//   p = cc^2 (d + (gamma-1)/(2 rho0) d^2 + rho s / c_p) + p0, d = rho - rho0
//   T = T0 exp((s + R log(rho / rho0)) / c_v)
// Against 128-bit arithmetic (1e6 states around ambient, 30 % density and 10
// J/(kg K) entropy noise) T is off by 0.67 units of 2^-53 RMS, 3.1 at most
// (divisions and library functions: 0.69, 3.3), p by 0.46 and 4.6 (0.50, 5.9).
__device__ __forceinline__ double row_height64(double ylo, double dy, int j) {
  return __dadd_rn(ylo, __dmul_rn(dy, (double)j + 0.5));
}
__device__ __forceinline__ void eos64(const EosConst64& E, double w0, double w3, double height, double& p, double& T) {
  const double cc = E.c_lr == 0.0 ? E.c : __dadd_rn(E.c, __dmul_rn(E.c_lr, height));
  const double d = __dsub_rn(w0, E.rho0);
  const double in = __fma_rn(w3, E.inv_c_p, __fma_rn(__dmul_rn(E.gm1_over_2rho0, d), d, d));
  p = __fma_rn(__dmul_rn(cc, cc), in, E.p0);
  const double s = __dmul_rn(w3, rcp64(w0));
  const double x = __dmul_rn(w0, E.inv_rho0);
  // x positive and normal; the factored argument's error (4 roundings of s
  // in place of 3) stays below that of the exponential while |a| < 1, which
  // is T from 108 to 797 K at T0 = 293 K
  if ((unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u) {
    const double l = log64(x, __fma_rn(w0, E.inv_rho0, -x));
    const double a = __fma_rn(E.R_over_c_v, l, __fma_rn(s, E.inv_c_v, E.a0));
    if (fabs(a) < 1.0) {
      T = __dmul_rn(E.T0, exp64(a));
      return;
    }
  }
  const double2 g = state_general64(E, w0, w3);
  T = g.x;
  p = __dadd_rn(p, g.y);
}

}  // namespace enl
