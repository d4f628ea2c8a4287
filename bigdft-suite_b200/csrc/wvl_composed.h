/* Generated by gen_composed.py from wvl_filters.h; do not edit. */
#pragma once

/* taps gs(-14..16) of magic filter . synthesis (index m+14) */
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
/* taps gw(-14..16) of magic filter . synthesis (index m+14) */
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
