// tdy_pow.h -- powers of positive numbers in integer arithmetic.
//
// On GB300 a warp's FP64 instruction occupies its quarter of the FP64 pipe for
// 57 cycles, so pow() takes 6,150 cycles a warp and a division 600 (measured,
// one warp, chained).  The constitutive relations need several powers of the
// same two bases.  Here a base's binary logarithm is formed once, as an
// integer plus a 62-bit fixed-point fraction, exponents are scaled and added
// in that form, and each power costs one exp2 of 64-bit fixed-point
// arithmetic on the integer pipes (about 70 instructions of 2 cycles).
//
// Method: table-driven logarithm and exponential (P. T. P. Tang, ACM TOMS 15
// (1989) 144 and 16 (1990) 378), with tables of 128 entries and Taylor
// polynomials of the reduced arguments:
//   log2 x = e - log2 c + log2(1 + r),  r = f c - 1 exact, |r| < 2^-7.6, c a
//   10-bit approximation of 1/f from the leading 7 fraction bits of x = f 2^e;
//   2^t = 2^k 2^(i/128) e^s,  s = (the rest of t) ln 2 < 2^-7.5.
// Measured against 200-bit arithmetic: the logarithm's absolute error is below
// 2^-61.4 (x in 2^-300..2^300 and beside 1); x^y as exp2_fx(fx_scale(y,
// log2_fx(x))) is within 0.51 ulp for y up to 4, 0.60 up to 32 and 0.68 up to
// 64 (x in 2^-10..2^10 and beside 1).
#pragma once

#include <cuda_runtime.h>

namespace tdy {

struct __align__(16) LogEntry {
  long long l;  // -log2(c / 1024), 62 fraction bits
  long long c;
};
#define TDY_POW_TABLE __device__ const
static TDY_POW_TABLE LogEntry kLogTable[128] = {
    {0x005c836701aa0d7bLL, 1020}, {0x0116a21e20a0a451LL, 1012}, {0x01d23afc49139f8aLL, 1004}, {0x02779bb373e01e67LL, 997},
    {0x03360a071b0812abLL, 989}, {0x03ddef24a116d3acLL, 982}, {0x048707bd57c1b081LL, 975}, {0x0549c69e188a83daLL, 967},
    {0x05f58125b3eed31aLL, 960}, {0x06a27d69b726b2fbLL, 953}, {0x0750c0289493505eLL, 946}, {0x07e725770744593aLL, 940},
    {0x0897d37aa87c4aecLL, 933}, {0x0949d61ee0d33433LL, 926}, {0x09e37db2866f2851LL, 920}, {0x0a9806bcb6f99ccfLL, 913},
    {0x0b33e041385c8284LL, 907}, {0x0bd0c294b1ac92d3LL, 901}, {0x0c6eb1410a025485LL, 895}, {0x0d0dafe2705a326eLL, 889},
    {0x0dadc227da59f78bLL, 883}, {0x0e4eebd38768affcLL, 877}, {0x0ef130bb884681b9LL, 871}, {0x0f9494ca4b544456LL, 865},
    {0x10391bff2dbcf338LL, 859}, {0x10c318aedff3c076LL, 854}, {0x1169c05363f15872LL, 848}, {0x11f588973c874718LL, 843},
    {0x128225bb5e64a3e9LL, 838}, {0x132bfee370ee6866LL, 832}, {0x13ba7963fc1f8ef0LL, 827}, {0x1449d115ef7d876cLL, 822},
    {0x14da08ac46495a4aLL, 817}, {0x156b22e6b578e49dLL, 812}, {0x15fd2291fc33cef6LL, 807}, {0x16900a8836d0d507LL, 802},
    {0x1723ddb1346b6515LL, 797}, {0x17b89f02cf2aad32LL, 792}, {0x184e5181475448f9LL, 787}, {0x18c6c335d8b965b2LL, 783},
    {0x195e2f9b51f04e2fLL, 778}, {0x19f695efbbd0ee9fLL, 773}, {0x1a713787ad97a4b8LL, 769}, {0x1b0b67f4f4680ff5LL, 764},
    {0x1b877c57b1b06ff0LL, 760}, {0x1c2381c08baf4e9eLL, 755}, {0x1ca111cb2aa5c544LL, 751}, {0x1d1f4d7febf867feLL, 747},
    {0x1d9e36b6b825b0a4LL, 743}, {0x1e3dd1156507ddd9LL, 738}, {0x1ebe47960e3c0880LL, 734}, {0x1f3f71cc1b629b83LL, 730},
    {0x1fc151b11b36401cLL, 726}, {0x2043e946fd97f5dcLL, 722}, {0x20c73a98433abf2fLL, 718}, {0x214b47b82ea431acLL, 714},
    {0x21d012c2f68d67f2LL, 710}, {0x223428f74e8ca777LL, 707}, {0x22ba458ca455b0f6LL, 703}, {0x2341260a447795faLL, 699},
    {0x23c8ccafd2fb087bLL, 695}, {0x242f0d16186fcf55LL, 692}, {0x24b81408c77d5f5cLL, 688}, {0x2541e78680e0b71eLL, 684},
    {0x25a9cdd122c8ce9dLL, 681}, {0x26350d0eb6705c56LL, 677}, {0x269e06fad8bf6473LL, 674}, {0x272ab98c4a3c8e55LL, 670},
    {0x2794ccdfa924feb8LL, 667}, {0x27ff5a9ce9e3abcdLL, 664}, {0x288e2d458104c41cLL, 660}, {0x28f9dcfaea92e2b1LL, 657},
    {0x29660adb732b4797LL, 654}, {0x29f70e4bd6b75269LL, 650}, {0x2a64671b21d8e3c4LL, 647}, {0x2ad24203b3694c82LL, 644},
    {0x2b40a03c917a88cdLL, 641}, {0x2baf830122b03c6bLL, 638}, {0x2c1eeb9143600e3dLL, 635}, {0x2c8edb315b321326LL, 632},
    {0x2cff532a7344f069LL, 629}, {0x2d7054ca4cd97c9dLL, 626}, {0x2de1e1637889c727LL, 623}, {0x2e53fa4d6e0f8fadLL, 620},
    {0x2ec6a0e4a49e5a42LL, 617}, {0x2f39d68aabd5715bLL, 614}, {0x2fad9ca6454e4c9eLL, 611}, {0x3021f4a37ecbfaeeLL, 608},
    {0x3096dff3cd105705LL, 605}, {0x30e524bb196cd583LL, 603}, {0x315b08d9e6d3481cLL, 600}, {0x31d184403cfbecceLL, 597},
    {0x3248987450350b4aLL, 594}, {0x329850e92589b608LL, 592}, {0x3310673cb9f7159aLL, 589}, {0x33891a8be56a4a25LL, 586},
    {0x33d9ea17e87e2681LL, 584}, {0x3453a6a249c24501LL, 581}, {0x34a52885aa8c11f0LL, 579}, {0x351ff2e30214bc30LL, 576},
    {0x35722a37c2d1badcLL, 574}, {0x35ee071e9f68aed8LL, 571}, {0x3640f713a7783bb0LL, 569}, {0x36bdeb5a7c2ce039LL, 566},
    {0x37119734556a4251LL, 564}, {0x378fa7d29bdb897bLL, 561}, {0x37e412ec386bc7c2LL, 559}, {0x3838cb7b6a079d0bLL, 557},
    {0x38b872c7291f496dLL, 554}, {0x390def6fd4951167LL, 552}, {0x3963bb8832dedb05LL, 550}, {0x39e503e2be17ce3aLL, 547},
    {0x3a3b991e25055e81LL, 545}, {0x3a927fd6fd0ac35eLL, 543}, {0x3ae9b8a73bc9e97fLL, 541}, {0x3b6d29207b2970deLL, 538},
    {0x3bc531d817581953LL, 536}, {0x3c1d8ecf99b58c0cLL, 534}, {0x3c7640a8deaa9421LL, 532}, {0x3ccf480796d5cd74LL, 530},
    {0x3d5574da88e6550dLL, 527}, {0x3daf54df46b1e14fLL, 525}, {0x3e098cb530796a64LL, 523}, {0x3e641d088b6533dbLL, 521},
    {0x3ebf0687997a2d6dLL, 519}, {0x3f1a49e2a175d53aLL, 517}, {0x3f75e7cbf6d11790LL, 515}, {0x3fd1e0f801eb1536LL, 513},
};
static TDY_POW_TABLE unsigned long long kExpTable[128] = {
    0x8000000000000000ULL, 0x80b1ed4fd999ab6cULL, 0x8164d1f3bc030773ULL, 0x8218af4373fc25ecULL,
    0x82cd8698ac2ba1d7ULL, 0x8383594eefb6ee37ULL, 0x843a28c3acde4046ULL, 0x84f1f656379c1a29ULL,
    0x85aac367cc487b15ULL, 0x8664915b923fba04ULL, 0x871f61969e8d1010ULL, 0x87db357ff698d792ULL,
    0x88980e8092da8527ULL, 0x8955ee03618e5fddULL, 0x8a14d575496efd9aULL, 0x8ad4c6452c728924ULL,
    0x8b95c1e3ea8bd6e7ULL, 0x8c57c9c4646f4ddeULL, 0x8d1adf5b7e5ba9e6ULL, 0x8ddf042022e69cd6ULL,
    0x8ea4398b45cd53c0ULL, 0x8f6a8117e6c8e5c4ULL, 0x9031dc431466b1dcULL, 0x90fa4c8beee4b12bULL,
    0x91c3d373ab11c336ULL, 0x928e727d9531f9acULL, 0x935a2b2f13e6e92cULL, 0x9426ff0fab1c04b6ULL,
    0x94f4efa8fef70961ULL, 0x95c3fe86d6cc7fefULL, 0x96942d3720185a00ULL, 0x97657d49f17ab08eULL,
    0x9837f0518db8a96fULL, 0x990b87e266c189aaULL, 0x99e0459320b7fa65ULL, 0x9ab62afc94ff864aULL,
    0x9b8d39b9d54e5539ULL, 0x9c6573682ec32c2dULL, 0x9d3ed9a72cffb751ULL, 0x9e196e189d472420ULL,
    0x9ef5326091a111aeULL, 0x9fd228256400dd06ULL, 0xa0b0510fb9714fc2ULL, 0xa18faeca8544b6e4ULL,
    0xa27043030c496819ULL, 0xa3520f68e802bb93ULL, 0xa43515ae09e6809eULL, 0xa5195786be9ef339ULL,
    0xa5fed6a9b15138eaULL, 0xa6e594cfeee86b1eULL, 0xa7cd93b4e965356aULL, 0xa8b6d5167b320e09ULL,
    0xa9a15ab4ea7c0ef8ULL, 0xaa8d2652ec907629ULL, 0xab7a39b5a93ed337ULL, 0xac6896a4be3fe929ULL,
    0xad583eea42a14ac6ULL, 0xae493452ca35b80eULL, 0xaf3b78ad690a4375ULL, 0xb02f0dcbb6e04584ULL,
    0xb123f581d2ac2590ULL, 0xb21a31a66618fe3bULL, 0xb311c412a9112489ULL, 0xb40aaea2654b9841ULL,
    0xb504f333f9de6484ULL, 0xb60093a85ed5f76cULL, 0xb6fd91e328d17791ULL, 0xb7fbefca8ca41e7cULL,
    0xb8fbaf4762fb9ee9ULL, 0xb9fcd2452c0b9debULL, 0xbaff5ab2133e45fbULL, 0xbc034a7ef2e9fb0dULL,
    0xbd08a39f580c36bfULL, 0xbe0f6809860993e2ULL, 0xbf1799b67a731083ULL, 0xc0213aa1f0d08db0ULL,
    0xc12c4cca66709456ULL, 0xc238d2311e3d6673ULL, 0xc346ccda24976407ULL, 0xc4563ecc5334cb33ULL,
    0xc5672a115506daddULL, 0xc67990b5aa245f79ULL, 0xc78d74c8abb9b15dULL, 0xc8a2d85c8ffe2c45ULL,
    0xc9b9bd866e2f27a3ULL, 0xcad2265e4290774eULL, 0xcbec14fef2727c5dULL, 0xcd078b86503dcdd2ULL,
    0xce248c151f8480e4ULL, 0xcf4318cf191918c1ULL, 0xd06333daef2b2595ULL, 0xd184df6251699ac6ULL,
    0xd2a81d91f12ae45aULL, 0xd3ccf099859ac379ULL, 0xd4f35aabcfedfa1fULL, 0xd61b5dfe9f9bce07ULL,
    0xd744fccad69d6af4ULL, 0xd870394c6db32c84ULL, 0xd99d15c278afd7b6ULL, 0xdacb946f2ac9cc72ULL,
    0xdbfbb797daf23755ULL, 0xdd2d818508324c20ULL, 0xde60f4825e0e9124ULL, 0xdf9612deb8f04420ULL,
    0xe0ccdeec2a94e111ULL, 0xe2055afffe83d369ULL, 0xe33f8972be8a5a51ULL, 0xe47b6ca0373da88dULL,
    0xe5b906e77c8348a8ULL, 0xe6f85aaaee1fce22ULL, 0xe8396a503c4bdc68ULL, 0xe97c38406c4f8c57ULL,
    0xeac0c6e7dd24392fULL, 0xec0718b64c1cbddcULL, 0xed4f301ed9942b84ULL, 0xee990f980da3025bULL,
    0xefe4b99bdcdaf5cbULL, 0xf13230a7ad094509ULL, 0xf281773c59ffb13aULL, 0xf3d28fde3a641a5bULL,
    0xf5257d152486cc2cULL, 0xf67a416c733f846eULL, 0xf7d0df730ad13bb9ULL, 0xf92959bb5dd4ba74ULL,
    0xfa83b2db722a033aULL, 0xfbdfed6ce5f09c49ULL, 0xfd3e0c0cf486c175ULL, 0xfe9e115c7b8f884cULL,
};

__device__ __forceinline__ long long fx_mulhi(long long a, long long b) { return __mul64hi(a, b); }
__device__ __forceinline__ unsigned long long fx_umulhi(unsigned long long a, unsigned long long b) {
  return __umul64hi(a, b);
}

// k + f / 2^62; f may lie outside [0, 2^62) until exp2_fx
struct fx {
  int k;
  long long f;
};
__device__ __forceinline__ fx fx_add(fx a, fx b) { return fx{a.k + b.k, a.f + b.f}; }
__device__ __forceinline__ fx fx_neg(fx a) { return fx{-a.k, -a.f}; }
__device__ __forceinline__ fx fx_half(fx a) { return fx{a.k >> 1, (a.f >> 1) + ((long long)(a.k & 1) << 61)}; }

// log2 of a normal positive x
__device__ __forceinline__ fx log2_fx(double x) {
  const long long b = __double_as_longlong(x);
  const int i = (int)(b >> 45) & 127;
  const LogEntry t = kLogTable[i];
  const long long f = (b & 0xfffffffffffffLL) | (1LL << 52);
  const long long r = (f * t.c - (1LL << 62)) << 2;  // 64 fraction bits, exact
  // log(1 + r) = r - r^2 (1/2 - r (1/3 - r (1/4 - r (1/5 - r (1/6 - r/7)))))
  const int r32 = (int)(r >> 32), r38 = (int)(r >> 26);
  const int h = 0x33333333 - __mulhi(r32, 0x2aaaaaab - __mulhi(r32, 0x24924925));           // 32 fraction bits
  const long long g4 = 0x4000000000000000LL - (((long long)r38 * h) >> 6);                  // 64, as all below
  const long long g3 = 0x5555555555555555LL - (((long long)r38 * (int)(g4 >> 32)) >> 6);
  // (1/2 has no positive 64-bit form: half of it, doubled in the product)
  const long long g2 = 0x4000000000000000LL - (fx_mulhi(r, g3) >> 1);
  const long long p = r - (fx_mulhi(r, fx_mulhi(r, g2)) << 1);
  return fx{(int)((b >> 52) & 0x7ff) - 1023, t.l + fx_mulhi(p, 0x5c551d94ae0bf85eLL)};
}

// y a, for positive y with an exponent in [-8, 6] and |a| < 512
__device__ __forceinline__ fx fx_scale(double y, fx a) {
  const long long b = __double_as_longlong(y);
  const int s = 52 - ((int)((b >> 52) & 0x7ff) - 1023);  // y = m 2^-s, 46 <= s <= 60
  const long long m = (b & 0xfffffffffffffLL) | (1LL << 52);
  const long long w = m * a.k;
  fx t = {(int)(w >> s), (w & ((1LL << s) - 1)) << (62 - s)};
  const long long h = fx_mulhi(a.f, m << 10);  // y a.f / 2^62 with 8 + s fraction bits
  if (s > 54) {
    t.f += h >> (s - 54);
  } else {
    t.k += (int)(h >> (8 + s));
    t.f += (h & ((1LL << (8 + s)) - 1)) << (54 - s);
  }
  return t;
}

// 2^(fraction of a) with 63 fraction bits, in [1, 2); *k: the integer part
__device__ __forceinline__ unsigned long long exp2_fraction(fx a, int *k) {
  *k = a.k + (int)(a.f >> 62);
  const unsigned long long f = (unsigned long long)a.f & 0x3fffffffffffffffULL;
  const unsigned long long T = kExpTable[(int)(f >> 55)];
  const unsigned long long s = fx_umulhi((f & 0x7fffffffffffffULL) << 2, 0xb17217f7d1cf79acULL);  // 64 fraction bits
  // e^s - 1 = s + s^2 (1/2 + s (1/6 + s (1/24 + s (1/120 + s/720))))
  const unsigned s32 = (unsigned)(s >> 32), s39 = (unsigned)(s >> 25);
  const unsigned q = 0x0aaaaaabu + __umulhi(s32, 0x02222222u + __umulhi(s32, 0x005b05b0u));  // 32 fraction bits
  const unsigned long long g3 = 0x2aaaaaaaaaaaaaabULL + (((unsigned long long)s39 * q) >> 7);
  const unsigned long long g2 = 0x8000000000000000ULL + fx_umulhi(s, g3);
  const unsigned long long p = s + fx_umulhi(s, fx_umulhi(s, g2));
  return T + fx_umulhi(T, p);
}

// 2^a, |a| < 1000
__device__ __forceinline__ double exp2_fx(fx a) {
  int k;
  const unsigned long long v = exp2_fraction(a, &k);
  // round to 53 bits; a carry moves into the exponent
  return __longlong_as_double(((long long)(k + 1022) << 52) + (long long)((v >> 11) + ((v >> 10) & 1)));
}

// 1 - 2^a, -1000 < a < -2^-50, to 2^-62: the difference is formed before the
// rounding to 53 bits
__device__ __forceinline__ double one_minus_exp2_fx(fx a) {
  int k;
  const unsigned long long v = exp2_fraction(a, &k);
  if (k < -60) return 1.0;
  const unsigned long long u = 0ULL - (v >> (-1 - k));  // 64 fraction bits
  const int lz = __clzll((long long)u);
  const unsigned long long m = u << lz;
  return __longlong_as_double(((long long)(1021 - lz) << 52) + (long long)((m >> 11) + ((m >> 10) & 1)));
}

}  // namespace tdy
