// FP64 logarithm and reciprocal from one table look-up (table-driven
// logarithm: P. T. P. Tang, ACM Trans. Math. Softw. 16, 1990).  Entry i serves the
// mantissas whose high word lies in [0x3fe6a09e + i 2^13, + 2^13), that is m in
// [sqrt(1/2), sqrt(2)): y near 1/m (1 for the intervals next to m = 1, so that
// logarithms near 0 keep their relative accuracy) and -log(y), each the double
// nearest to its 50-digit value.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

static __device__ const double2 kLogTab[128] = {
    {0x1.690aa14c2f61dp+0, -0x1.60112dbc1b0f3p-2},
    {0x1.67103c7e0340fp+0, -0x1.5a70f9db56263p-2},
    {0x1.651b5c793d42dp+0, -0x1.54d8a47c798cap-2},
    {0x1.632bea459c7d5p+0, -0x1.4f4817ba7b025p-2},
    {0x1.6141cf69a8eb0p+0, -0x1.49bf3e0b3292bp-2},
    {0x1.5f5cf5e74d59dp+0, -0x1.443e023d66468p-2},
    {0x1.5d7d48388d303p+0, -0x1.3ec44f76e3358p-2},
    {0x1.5ba2b14c5500dp+0, -0x1.39521132a38c0p-2},
    {0x1.59cd1c8364ef7p+0, -0x1.33e7333f011a4p-2},
    {0x1.57fc75ad53f2dp+0, -0x1.2e83a1bbf4072p-2},
    {0x1.5630a905ab0cbp+0, -0x1.292749195d46ap-2},
    {0x1.5469a3311797cp+0, -0x1.23d216155c74cp-2},
    {0x1.52a7513ab3d5ep+0, -0x1.1e83f5bab0b9bp-2},
    {0x1.50e9a09164f25p+0, -0x1.193cd55f2461dp-2},
    {0x1.4f307f054db28p+0, -0x1.13fca2a202d36p-2},
    {0x1.4d7bdac555190p+0, -0x1.0ec34b6a98910p-2},
    {0x1.4bcba25cc0461p+0, -0x1.0990bde6bcfb5p-2},
    {0x1.4a1fc4b0dee7cp+0, -0x1.0464e88965862p-2},
    {0x1.487830fec992fp+0, -0x1.fe7f7412842e7p-3},
    {0x1.46d4d6d931650p+0, -0x1.f44242bec490ap-3},
    {0x1.4535a62640555p+0, -0x1.ea121b8bc696dp-3},
    {0x1.439a8f1d89a16p+0, -0x1.dfeedd6d4c53ep-3},
    {0x1.4203824609c7ap+0, -0x1.d5d867d41c4d1p-3},
    {0x1.407070743586ep+0, -0x1.cbce9aab8dfb4p-3},
    {0x1.3ee14ac81760ap+0, -0x1.c1d15657259d5p-3},
    {0x1.3d5602ab7b200p+0, -0x1.b7e07bb03ee5bp-3},
    {0x1.3bce89d026ebfp+0, -0x1.adfbec03c6142p-3},
    {0x1.3a4ad22e2170ap+0, -0x1.a423890fff12bp-3},
    {0x1.38cace0204b00p+0, -0x1.9a5735025a2e8p-3},
    {0x1.374e6fcb5d0dep+0, -0x1.9096d27556098p-3},
    {0x1.35d5aa4b142f9p+0, -0x1.86e2446e6e629p-3},
    {0x1.34607081e74c0p+0, -0x1.7d396e5c175b4p-3},
    {0x1.32eeb5aee88b9p+0, -0x1.739c3413c4dc1p-3},
    {0x1.31806d4e0b1bap+0, -0x1.6a0a79cffdc2dp-3},
    {0x1.30158b16b99d3p+0, -0x1.6084242e7a89dp-3},
    {0x1.2eae02fa7697cp+0, -0x1.5709182e4f0dfp-3},
    {0x1.2d49c923869f9p+0, -0x1.4d993b2e1f306p-3},
    {0x1.2be8d1f3a3de1p+0, -0x1.443472ea5dfcap-3},
    {0x1.2a8b1202bab0cp+0, -0x1.3adaa57b970e9p-3},
    {0x1.29307e1daf14dp+0, -0x1.318bb954c1f1fp-3},
    {0x1.27d90b452a980p+0, -0x1.284795419f347p-3},
    {0x1.2684aeac72899p+0, -0x1.1f0e20651ee2ap-3},
    {0x1.25335db8462a9p+0, -0x1.15df4237d0395p-3},
    {0x1.23e50dfdc49c4p+0, -0x1.0cbae2865a420p-3},
    {0x1.2299b5415a4fdp+0, -0x1.03a0e96ffd233p-3},
    {0x1.21514975b5bbfp+0, -0x1.f5227eca37d08p-4},
    {0x1.200bc0bac31edp+0, -0x1.e3179a4b9d0d7p-4},
    {0x1.1ec9115caf152p+0, -0x1.d120f780f7d10p-4},
    {0x1.1d8931d2efd1bp+0, -0x1.bf3e6920f797fp-4},
    {0x1.1c4c18bf54c08p+0, -0x1.ad6fc2798073fp-4},
    {0x1.1b11bced1c64fp+0, -0x1.9bb4d76d0cd1ap-4},
    {0x1.19da15501042dp+0, -0x1.8a0d7c701db33p-4},
    {0x1.18a51903a6a35p+0, -0x1.78798686b8f7dp-4},
    {0x1.1772bf4a2a09ap+0, -0x1.66f8cb41f55b0p-4},
    {0x1.1642ff8be62bcp+0, -0x1.558b20bd93cfep-4},
    {0x1.1515d1565a45fp+0, -0x1.44305d9da5e3fp-4},
    {0x1.13eb2c5b70a01p+0, -0x1.32e8590c40d16p-4},
    {0x1.12c30870bb1dfp+0, -0x1.21b2eab73ceefp-4},
    {0x1.119d5d8eb4b51p+0, -0x1.108feace01313p-4},
    {0x1.107a23d007a34p+0, -0x1.fefe63feb4df0p-5},
    {0x1.0f595370d842ap+0, -0x1.dd0132eebc3afp-5},
    {0x1.0e3ae4ce14593p+0, -0x1.bb27f5bab0694p-5},
    {0x1.0d1ed064c6c2fp+0, -0x1.997260a3880fap-5},
    {0x1.0c050ed16f565p+0, -0x1.77e028d89f6c3p-5},
    {0x1.0aed98cf5ee48p+0, -0x1.56710473d4017p-5},
    {0x1.09d867381737ap+0, -0x1.3524aa75b4843p-5},
    {0x1.08c57302aef1cp+0, -0x1.13fad2c1c486ap-5},
    {0x1.07b4b54339310p+0, -0x1.e5e66c35a6e01p-6},
    {0x1.06a6272a30dd5p+0, -0x1.a41b1c3ecc79ap-6},
    {0x1.0599c203e7862p+0, -0x1.62932a8c6745dp-6},
    {0x1.048f7f37f7b66p+0, -0x1.214e0db564450p-6},
    {0x1.03875848baa63p+0, -0x1.c0967be6de52dp-7},
    {0x1.028146d2c1326p+0, -0x1.3f146a38a7295p-7},
    {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.0000000000000p+0, 0x0.0p+0},
    {0x1.f9fe7fcf63b4fp-1, 0x1.82a5ba13a4d27p-7},
    {0x1.f61e0b5e77662p-1, 0x1.3f561d03f17fep-6},
    {0x1.f24cae8520b85p-1, 0x1.bc6324ae6b1f1p-6},
    {0x1.ee8a11cc60d64p-1, 0x1.1c3ed779036bep-5},
    {0x1.ead5e05c04446p-1, 0x1.59d4b09716fb8p-5},
    {0x1.e72fc7e1b406dp-1, 0x1.96f4e5eebd371p-5},
    {0x1.e3977879215f4p-1, 0x1.d3a1359a16dcep-5},
    {0x1.e00ca4953da63p-1, 0x1.07eda9ee351dfp-4},
    {0x1.dc8f00ea70998p-1, 0x1.25d275b5d6021p-4},
    {0x1.d91e4459c0442p-1, 0x1.437fcedbaf10dp-4},
    {0x1.d5ba27dcde604p-1, 0x1.60f6819671036p-4},
    {0x1.d26266730fc58p-1, 0x1.7e3755bcad2f4p-4},
    {0x1.cf16bd0ee3195p-1, 0x1.9b430ee49b643p-4},
    {0x1.cbd6ea84ac94fp-1, 0x1.b81a6c82c162bp-4},
    {0x1.c8a2af79bd42cp-1, 0x1.d4be2a0787fd6p-4},
    {0x1.c579ce544c9f1p-1, 0x1.f12efefbc94c5p-4},
    {0x1.c25c0b2c0c07fp-1, 0x1.06b6cf8e31687p-3},
    {0x1.bf492bbb5bdeap-1, 0x1.14bd5d3a6af52p-3},
    {0x1.bc40f7511aae8p-1, 0x1.22ab7ebc803bdp-3},
    {0x1.b94336c307176p-1, 0x1.3081888efb85bp-3},
    {0x1.b64fb460ad9c1p-1, 0x1.3e3fcd7904d22p-3},
    {0x1.b3663be6dbd40p-1, 0x1.4be69e99fdbacp-3},
    {0x1.b0869a7392d58p-1, 0x1.59764b74baf4dp-3},
    {0x1.adb09e7a73033p-1, 0x1.66ef21fa5f4bdp-3},
    {0x1.aae417b99bb29p-1, 0x1.74516e94dbcf7p-3},
    {0x1.a820d72ef96cap-1, 0x1.819d7c3118bcdp-3},
    {0x1.a566af0dfdce8p-1, 0x1.8ed39448ca815p-3},
    {0x1.a2b572b5bc4fap-1, 0x1.9bf3feebf6168p-3},
    {0x1.a00cf6a767735p-1, 0x1.a8ff02ca27c4bp-3},
    {0x1.9d6d107d2a21fp-1, 0x1.b5f4e53b5f46bp-3},
    {0x1.9ad596e1591fep-1, 0x1.c2d5ea48b4181p-3},
    {0x1.98466185f8c9dp-1, 0x1.cfa254b4b4a4bp-3},
    {0x1.95bf491c936fap-1, 0x1.dc5a660382e9cp-3},
    {0x1.9340274e5cd4dp-1, 0x1.e8fe5e82b101dp-3},
    {0x1.90c8d6b49f894p-1, 0x1.f58e7d50dff4ep-3},
    {0x1.8e5932d170f5bp-1, 0x1.0105803291889p-2},
    {0x1.8bf11808a91e9p-1, 0x1.073a124b14fa7p-2},
    {0x1.899063991b448p-1, 0x1.0d6512d099adep-2},
    {0x1.8736f3960cacep-1, 0x1.13869f1865554p-2},
    {0x1.84e4a6e0e6fd0p-1, 0x1.199ed3f1a910bp-2},
    {0x1.82995d2323b23p-1, 0x1.1fadcda8adc47p-2},
    {0x1.8054f6c86e5f2p-1, 0x1.25b3a809e88abp-2},
    {0x1.7e1754f8fb71bp-1, 0x1.2bb07e64f817dp-2},
    {0x1.7be05994115fap-1, 0x1.31a46b8f8be09p-2},
    {0x1.79afe72ac2320p-1, 0x1.378f89e835c4ap-2},
    {0x1.7785e0fad37e4p-1, 0x1.3d71f35926fe0p-2},
    {0x1.75622ae9d2f2ep-1, 0x1.434bc15ad90a1p-2},
    {0x1.7344a98055b3ap-1, 0x1.491d0cf6a33a5p-2},
    {0x1.712d41e560d4ap-1, 0x1.4ee5eec93d95bp-2},
    {0x1.6f1bd9d9f957ep-1, 0x1.54a67f0531ab8p-2},
    {0x1.6d1057b4da225p-1, 0x1.5a5ed57539f35p-2},
    {0x1.6b0aa25e4e709p-1, 0x1.600f097e904c4p-2},
};

// 1 / x and ln x of a positive normal x = 2^k m, m in [sqrt(1/2), sqrt(2)):
// with the table's y near 1 / m and r = m y - 1 (|r| < 2^-6.9, exact up to
// rounding), ln x = k ln 2 - ln y + ln(1 + r) by the series to r^8, and 1 / m
// = y (1 - r)(1 + r^2) corrected by one Newton step.  Both within 1.3 units in
// the last place on 2e4 arguments against 50 digits.  Anything else (0,
// negative, subnormal, infinite, NaN) takes the library's functions.
__device__ __forceinline__ void rcp_log(double x, const double2* __restrict__ tab, double& inv, double& lg) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  if (h - 0x00100000u >= 0x7fe00000u) {
    inv = 1.0 / x;
    lg = log(x);
    return;
  }
  const uint32_t hx = h + (0x3ff00000u - 0x3fe6a09eu);
  const int k = (int)(hx >> 20) - 0x3ff;
  const uint32_t hm = (hx & 0xfffffu) + 0x3fe6a09eu;
  const double m = __hiloint2double((int)hm, __double2loint(x));
  const double2 t = tab[(hm - 0x3fe6a09eu) >> 13];
  const double r = fma(m, t.x, -1.0), r2 = r * r;
  double y = fma(-r, t.x, t.x);
  y = fma(y, r2, y);
  y = fma(y, fma(-m, y, 1.0), y);
  // y 2^-k by its exponent (1 / x is subnormal only where x is not below 2^1022)
  inv = k < 1020 && k > -1020 ? __hiloint2double(__double2hiint(y) - (k << 20), __double2loint(y)) : 1.0 / x;
  const double kd = __hiloint2double(0x43300000, (int)((uint32_t)k ^ 0x80000000u)) - 4503601774854144.0;  // k
  double q = fma(r2, -0.125, fma(r, 1.0 / 7, -1.0 / 6));
  q = fma(r2, q, fma(r, 0.2, -0.25));
  q = fma(r2, q, fma(r, 1.0 / 3, -0.5));
  lg = fma(kd, 0.69314718055994530942, t.y) + fma(r2, q, r);
}
