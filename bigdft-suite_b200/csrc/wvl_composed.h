/* Generated by gen_composed.py from wvl_filters.h; do not edit. */
#pragma once

/* FP64 taps gs(-14..16) of magic filter . synthesis (index m+14) */
#define WVL_B64_S_INIT { \
    -0x1.3cf8170a61665p-27, \
    0x1.7584b6cc19e93p-23, \
    -0x1.a22c6343059f0p-20, \
    0x1.471debc153f6fp-17, \
    -0x1.ddd29203e5663p-16, \
    -0x1.1e94462b95551p-15, \
    0x1.1ef2c23018650p-11, \
    -0x1.c4c398dcb32cdp-9, \
    -0x1.1bc55662ee569p-8, \
    0x1.04cbb3ef0ec5cp-5, \
    0x1.7fc9f48d6f805p-6, \
    -0x1.1bb2e0a9a5730p-3, \
    -0x1.c3809e3d806e8p-4, \
    0x1.aa0d73796e5eap-2, \
    0x1.8f98841cfeab2p-1, \
    0x1.b4363198b08a4p-2, \
    -0x1.e31eafacb9d6cp-7, \
    -0x1.0083e7af55d06p-5, \
    0x1.66c14317b1ac9p-5, \
    0x1.06d40edb1ea38p-7, \
    -0x1.b604881365b68p-7, \
    -0x1.c130041cc65f2p-10, \
    0x1.97932616fdfcap-10, \
    0x1.f70fad0a1f57cp-13, \
    0x1.a464244c351c1p-16, \
    -0x1.dab650f294f59p-17, \
    0x1.1693f55adeacfp-19, \
    -0x1.addbe063f7c7dp-22, \
    0x1.50f93b4d1f949p-23, \
    -0x1.a76bd1c38b185p-26, \
    0x1.b61f026a675b6p-30}
/* FP64 taps gw(-14..16) of magic filter . synthesis (index m+14) */
#define WVL_B64_W_INIT { \
    -0x1.6237bd7ff8f51p-28, \
    0x1.a16995d0003bap-24, \
    -0x1.d75a530edcdd1p-21, \
    0x1.771306e07e87dp-18, \
    -0x1.200fe236e67c0p-16, \
    -0x1.7e9a65da33101p-17, \
    0x1.2aa115c26921ep-12, \
    -0x1.02346668ffa4cp-9, \
    -0x1.00edddb2e1ff6p-9, \
    0x1.f4c0df6d3111ap-7, \
    0x1.ddae6439c39ebp-8, \
    -0x1.4706682a2d563p-5, \
    -0x1.b1a673043891cp-5, \
    0x1.937044210da41p-5, \
    0x1.9d2682def80a0p-2, \
    -0x1.8fecf4024f12fp-1, \
    0x1.c09e9f4467508p-2, \
    0x1.3ee826419ced0p-4, \
    -0x1.e97fe3d587ba9p-4, \
    -0x1.76800c229e604p-6, \
    0x1.ce22501c27cbcp-6, \
    0x1.eab07e046e98cp-9, \
    -0x1.64b09b40252dbp-9, \
    -0x1.e7117f4074346p-12, \
    -0x1.552657c781ed5p-15, \
    0x1.9ad26625a3f10p-16, \
    -0x1.bd6a98e5a698ap-19, \
    0x1.5e1a753ab4e97p-21, \
    -0x1.2911ba5f482c4p-22, \
    0x1.7ae531030df92p-25, \
    -0x1.880ca76eac140p-29}
/* FP32 taps gs(-14..16) of magic filter . synthesis, times 0.9752083272817533 (index m+14) */
#define WVL_B32_S_INIT { \
    -0x1.35067c0000000p-27f, \
    0x1.6c406a0000000p-23f, \
    -0x1.97ce9c0000000p-20f, \
    0x1.3f01c80000000p-17f, \
    -0x1.d1f9f80000000p-16f, \
    -0x1.1779360000000p-15f, \
    0x1.17d5980000000p-11f, \
    -0x1.b98a080000000p-9f, \
    -0x1.14bc540000000p-8f, \
    0x1.fca9080000000p-6f, \
    0x1.76462a0000000p-6f, \
    -0x1.14aa560000000p-3f, \
    -0x1.b84f160000000p-4f, \
    0x1.9f7d700000000p-2f, \
    0x1.85b06a0000000p-1f, \
    0x1.a965b40000000p-2f, \
    -0x1.d7247a0000000p-7f, \
    -0x1.f44fc60000000p-6f, \
    0x1.5ddc5e0000000p-5f, \
    0x1.0050000000000p-7f, \
    -0x1.ab28960000000p-7f, \
    -0x1.b60d2c0000000p-10f, \
    0x1.8d78660000000p-10f, \
    0x1.ea96e20000000p-13f, \
    0x1.99f7aa0000000p-16f, \
    -0x1.cef1980000000p-17f, \
    0x1.0fabf60000000p-19f, \
    -0x1.a332ea0000000p-22f, \
    0x1.48a0880000000p-23f, \
    -0x1.9cc9080000000p-26f, \
    0x1.ab8dae0000000p-30f}
/* FP32 taps gw(-14..16) of magic filter . synthesis, times 0.9752083272817533 (index m+14) */
#define WVL_B32_W_INIT { \
    -0x1.58f1340000000p-28f, \
    0x1.9715a80000000p-24f, \
    -0x1.cbabc40000000p-21f, \
    0x1.6dc6940000000p-18f, \
    -0x1.18eba60000000p-16f, \
    -0x1.751e0c0000000p-17f, \
    0x1.2339cc0000000p-12f, \
    -0x1.f79b5a0000000p-10f, \
    -0x1.f51e6a0000000p-10f, \
    0x1.e856c40000000p-7f, \
    0x1.d1d6b80000000p-8f, \
    -0x1.3eeae20000000p-5f, \
    -0x1.a6e6380000000p-5f, \
    0x1.896fc60000000p-5f, \
    0x1.92e8620000000p-2f, \
    -0x1.8602c20000000p-1f, \
    0x1.b57f620000000p-2f, \
    0x1.3700280000000p-4f, \
    -0x1.dd5d320000000p-4f, \
    -0x1.6d373a0000000p-6f, \
    0x1.c2ad4e0000000p-6f, \
    0x1.de86400000000p-9f, \
    -0x1.5bd8d20000000p-9f, \
    -0x1.dafe0c0000000p-12f, \
    -0x1.4cb10e0000000p-15f, \
    0x1.90a3320000000p-16f, \
    -0x1.b25f9e0000000p-19f, \
    0x1.556bd80000000p-21f, \
    -0x1.21b4a20000000p-22f, \
    0x1.718bfe0000000p-25f, \
    -0x1.7f4b980000000p-29f}
/* that factor's -6th power */
#define WVL_B32_INV6 0x1.299d91ffff928p+0
/* FP64 taps a(0..14) of analysis . kinetic . synthesis */
#define WVL_T64_A_INIT { \
    -0x1.c6df63929cbc6p+1, \
    0x1.1c0cfedee564dp+1, \
    -0x1.3b31c704d5a7cp-1, \
    0x1.e5bd9c1ae926bp-3, \
    -0x1.50f692972eaedp-4, \
    0x1.69998376f173bp-6, \
    -0x1.0c8b4658f56fap-8, \
    0x1.d99eb6795ef2ep-12, \
    -0x1.925b217cd373ap-16, \
    0x1.18926785388d8p-19, \
    -0x1.8fc3246778128p-22, \
    -0x1.6bb8d9c92ea58p-27, \
    -0x1.ff64ebd74464ap-35, \
    0x1.30e1578b337e4p-42, \
    0x0.0p+0}
/* FP64 taps c(-14..14) of analysis . kinetic . synthesis (index l+14) */
#define WVL_T64_C_INIT { \
    0x0.0p+0, \
    0x1.54b5f0ae59996p-43, \
    -0x1.1bcda68fe9ddap-35, \
    -0x1.99c0098fe4b7bp-28, \
    -0x1.d113af7c23d26p-23, \
    0x1.d848a400104a4p-21, \
    -0x1.7c5330f6b7d95p-17, \
    0x1.c74ef21ac362dp-13, \
    -0x1.17ebd3009653cp-9, \
    0x1.d3c542e7740dcp-8, \
    -0x1.d2723a0ac45ffp-6, \
    0x1.256c77f0a4f52p-3, \
    -0x1.b32e1735e41f7p-2, \
    0x1.5066554a2523fp-1, \
    -0x1.aeea88d1ec73ap-2, \
    -0x1.bcbeff8673da3p-3, \
    0x1.44e667bf88ca4p-1, \
    -0x1.10e30c511a2b7p-1, \
    0x1.dea0ad8c63400p-3, \
    -0x1.cf7b581657694p-5, \
    0x1.09006013021ffp-7, \
    -0x1.e9cf108a9bb0ap-11, \
    0x1.a9ca254ac1755p-15, \
    -0x1.366b75cd07305p-18, \
    0x1.5729c80321a62p-21, \
    0x1.42d35b090d4eep-26, \
    0x1.ccba493c1cf33p-34, \
    -0x1.10d7b7f7fe198p-41, \
    0x0.0p+0}
/* FP64 taps e(0..14) of analysis . kinetic . synthesis */
#define WVL_T64_E_INIT { \
    -0x1.8e0377204924fp+4, \
    -0x1.c9384674485a3p+2, \
    -0x1.5c4cb92590702p-5, \
    -0x1.147036d893417p-2, \
    0x1.502d650670453p-4, \
    -0x1.69a6019014afbp-6, \
    0x1.0c8b445990809p-8, \
    -0x1.d99eb6795f3abp-12, \
    0x1.925b217cd3652p-16, \
    -0x1.189267853c2dfp-19, \
    0x1.8fc3246774392p-22, \
    0x1.6bb8d9c5727b3p-27, \
    0x1.ff64eec400352p-35, \
    -0x1.30e69e4e8bbc9p-42, \
    0x0.0p+0}
/* FP32 taps a(0..14) of analysis . kinetic . synthesis, times 1.9474363232066856 */
#define WVL_T32_A_INIT { \
    -0x1.baeaf00000000p+2f, \
    0x1.1495dc0000000p+2f, \
    -0x1.32e91a0000000p+0f, \
    0x1.d8f9780000000p-2f, \
    -0x1.481b6e0000000p-3f, \
    0x1.60189e0000000p-5f, \
    -0x1.057c740000000p-7f, \
    0x1.cd2bec0000000p-11f, \
    -0x1.87c76e0000000p-15f, \
    0x1.1131820000000p-18f, \
    -0x1.852e040000000p-21f, \
    -0x1.65f3ea0000000p-26f, \
    0x0.0p+0f, \
    0x0.0p+0f, \
    0x0.0p+0f}
/* FP32 taps c(-14..14) of analysis . kinetic . synthesis, times 1.9474363232066856 (index l+14) */
#define WVL_T32_C_INIT { \
    0x0.0p+0f, \
    0x0.0p+0f, \
    0x0.0p+0f, \
    -0x1.91ab880000000p-27f, \
    -0x1.c4fc820000000p-22f, \
    0x1.cbd9aa0000000p-20f, \
    -0x1.7254d60000000p-16f, \
    0x1.bb578a0000000p-12f, \
    -0x1.10907a0000000p-8f, \
    0x1.c77a080000000p-7f, \
    -0x1.c62fe80000000p-5f, \
    0x1.1db6460000000p-2f, \
    -0x1.a7be220000000p-1f, \
    0x1.478efc0000000p+0f, \
    -0x1.a397440000000p-1f, \
    -0x1.b10eae0000000p-2f, \
    0x1.3c5c6e0000000p+0f, \
    -0x1.09b7060000000p+0f, \
    0x1.d20c660000000p-2f, \
    -0x1.c34cf80000000p-4f, \
    0x1.0209680000000p-6f, \
    -0x1.dcef900000000p-10f, \
    0x1.9e993c0000000p-14f, \
    -0x1.2e43940000000p-17f, \
    0x1.4e1c720000000p-20f, \
    0x1.39ab400000000p-25f, \
    0x0.0p+0f, \
    0x0.0p+0f, \
    0x0.0p+0f}
/* FP32 taps e(0..14) of analysis . kinetic . synthesis, times 1.9474363232066856 */
#define WVL_T32_E_INIT { \
    -0x1.838d920000000p+5f, \
    -0x1.bd34080000000p+3f, \
    -0x1.5325500000000p-4f, \
    -0x1.0d2c4c0000000p-1f, \
    0x1.47578a0000000p-3f, \
    -0x1.6024c80000000p-5f, \
    0x1.057c760000000p-7f, \
    -0x1.cd2c220000000p-11f, \
    0x1.87c85a0000000p-15f, \
    -0x1.1133400000000p-18f, \
    0x1.8556d60000000p-21f, \
    0x1.6195cc0000000p-26f, \
    0x0.0p+0f, \
    0x0.0p+0f, \
    0x0.0p+0f}
/* that factor */
#define WVL_T32_NORM 1.9474363232066856
