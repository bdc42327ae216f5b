// x^y in double precision by fixed-point logarithm and exponential on the
// integer pipe.
//
// CUDA's pow is a chain of some 150 dependent FP64 operations, and one costs
// 64 cycles on GB300 (the FP64 pipe is shared by the SM): about 10,000 cycles,
// which set the pace of every kernel that takes a power per boundary face (the
// far-field state takes three, one after the other).  Integer multiplies
// return in 5 cycles (64-bit high products in 43), so the same value is
// cheaper in fixed point (an explicit Euler step of 32,768 cells with far-field
// boundaries 75.8 -> 54.6 us, an RK3 step of 1,980 cells 229 -> 198 us, four
// viscous RK2 steps of 44,849 cells with Sutherland's law 4.43 -> 3.80 ms):
//
//   x = 2^E m, 1 <= m < 2: r_j = R_j / 2^11 close to 1 / m from the leading 7
//   bits of m, z = m r_j - 1 exactly (|z| < 2^-7.8), log2 x = E - log2 r_j +
//   log2(1 + z) with -log2 r_j from a table and eight terms of the
//   logarithm's power series (truncation below 2^-73);
//   w = y log2 x = I + F, I an integer, 0 <= F < 1 with 64 bits;
//   2^F = 2^(i/128) 2^g, the first factor from a table, seven terms of the
//   exponential series for the second (g < 2^-7, truncation below 2^-75);
//
// and the 64-bit significand is rounded to 53 bits once.  The absolute error
// of log2 x is below 2^-62.5, so for |y| <= 8 the result is off by less than
// 0.51 units in the last place, and for |y| <= 64 (the largest taken here)
// less than 0.56; CUDA states 2 for its pow.  Operands outside the positive
// normal range, larger |y| and results outside the normal range call pow.
// The method is the textbook table-driven one (J.-M. Muller, Elementary
// Functions, 3rd ed., chapters 4 and 6).
#pragma once

#include "mcfd_arith.cuh"

#if defined(__CUDACC__)
#define MCFD_IA_FN __host__ __device__ __forceinline__
#define MCFD_IA_SLOW static __host__ __device__ __noinline__
#else
#define MCFD_IA_FN static inline
#define MCFD_IA_SLOW static
#endif

namespace mcfd {
namespace ia {

// R_j = nearest integer to 2^11 / (1 + (j + 1/2) / 128)
#define MCFD_POW_R \
  2040, 2024, 2009, 1993, 1978, 1964, 1949, 1935, 1920, 1907, 1893, 1879, 1866, 1853, 1840, 1827, \
  1814, 1802, 1789, 1777, 1765, 1753, 1742, 1730, 1719, 1708, 1697, 1686, 1675, 1664, 1654, 1644, \
  1633, 1623, 1613, 1603, 1594, 1584, 1574, 1565, 1556, 1547, 1538, 1529, 1520, 1511, 1502, 1494, \
  1485, 1477, 1469, 1460, 1452, 1444, 1436, 1429, 1421, 1413, 1406, 1398, 1391, 1383, 1376, 1369, \
  1362, 1355, 1348, 1341, 1334, 1327, 1321, 1314, 1307, 1301, 1295, 1288, 1282, 1276, 1269, 1263, \
  1257, 1251, 1245, 1239, 1234, 1228, 1222, 1216, 1211, 1205, 1200, 1194, 1189, 1183, 1178, 1173, \
  1168, 1163, 1157, 1152, 1147, 1142, 1137, 1132, 1128, 1123, 1118, 1113, 1108, 1104, 1099, 1095, \
  1090, 1085, 1081, 1077, 1072, 1068, 1063, 1059, 1055, 1051, 1046, 1042, 1038, 1034, 1030, 1026
// nearest integer to -log2(R_j / 2^11) 2^64
#define MCFD_POW_L \
  0x01720d9c06a835eaull, 0x045a887882829143ull, 0x0719d8f48ac1503bull, 0x0a0ddc77bfca54e0ull, \
  0x0cd8281c6c204aacull, 0x0f77bc92845b4eb1ull, 0x124c9ea888454579ull, 0x14f63a7ff1da4237ull, \
  0x17d60496cfbb4c67ull, 0x1a585dec4cb04136ull, 0x1d110afcb2a116abull, 0x1fcee3f8285bc67eull, \
  0x225f4deaa1f12bb1ull, 0x24f44eacff708f80ull, 0x278df6ca19bca143ull, 0x2a2c5726de368333ull, \
  0x2ccf8104e1720a11ull, 0x2f430a52c6b24b4cull, 0x31ef9acf37fb7a82ull, 0x346bf0a50acf78ffull, \
  0x36ec9648b252f002ull, 0x39719ac9b247a99dull, 0x3bc4c2ee211a06e3ull, 0x3e5253292d51115aull, \
  0x40ad6b5fd9f33095ull, 0x430c62bb7fcf01daull, 0x456f460aefa5d74dull, 0x47d6225cf21d1c62ull, \
  0x4a410501f4840d5aull, 0x4caffb8dc3b9a197ull, 0x4ee9e58ff07e3bbfull, 0x51274457bdf61db2ull, \
  0x53a204345cce98fdull, 0x55e6c862f3511e5cull, 0x582f237685f5fec9ull, 0x5a7b20dcf138ce42ull, \
  0x5c8f76c4d1ad9455ull, 0x5ee27c0b3caab4c8ull, 0x613946051d5123e2ull, 0x635771f9fef7c67bull, \
  0x6578be6d47c138bdull, 0x679d34a87a20efe7ull, 0x69c4de1eb65e92e0ull, 0x6befc46db4b211eaull, \
  0x6e1df15ec6c1bfc0ull, 0x704f6ee7e0c5c4acull, 0x7284472caa971510ull, 0x747d35ffafe19ff6ull, \
  0x76b880a20c66012full, 0x78b73b3cd41685a4ull, 0x7ab8bbf152f8ab13ull, 0x7cfdc7306d8a6e0bull, \
  0x7f0546c46cd9006eull, 0x810fa51bf65fd771ull, 0x831cea610ceafcbcull, 0x84eaeef20e6371e6ull, \
  0x86fdbbb0555df73full, 0x8913879ad1e83304ull, 0x8ae916329156c3d9ull, 0x8d04982911de57e9ull, \
  0x8edf33c41ba28147ull, 0x91008b663ca5262aull, 0x92e050231df57d70ull, 0x94c287492c4db040ull, \
  0x96a737448b233a76ull, 0x988e669ac8561d32ull, 0x9a781beb62fd91ccull, 0x9c645df055b7143full, \
  0x9e53337ea493fae2ull, 0xa044a386eec2db2aull, 0xa1f11b5b53afb96eull, 0xa3e773ebaa4b8ac5ull, \
  0xa5e07b676fd2e1f6ull, 0xa79385917af226dfull, 0xa948928ae13310f4ull, 0xab49080ecda53209ull, \
  0xad0280f245ea2333ull, 0xaebe0c048ac0f1adull, 0xb0c6285d5dfbfa03ull, 0xb2864167d5f8bb2cull, \
  0xb4487cb37dbc0804ull, 0xb60cdf7a88ad3ea4ull, 0xb7d36f0a7749fb9dull, 0xb99c30c476a13392ull, \
  0xbb1a83929279690aull, 0xbce75a2aaf55c56cull, 0xbeb6729915393279ull, 0xc087d28dfb2febb9ull, \
  0xc20d646de139a220ull, 0xc3e3013cd2032abbull, 0xc56c23679b4d206eull, 0xc7461100f3efb33aull, \
  0xc8d2d44ee235b447ull, 0xcab1273106eda7faull, 0xcc419cf2e7dc5668ull, 0xcdd3c6c489412f20ull, \
  0xcf67a85fa1f89a04ull, 0xd0fd458a2f1d6dadull, 0xd2e6510626665965ull, 0xd47fcb8c0852f0c1ull, \
  0xd61b0e0982d342cfull, 0xd7b81c7a7da2bb61ull, 0xd956fae84d7ca6d6ull, 0xdaf7ad69f0b380e5ull, \
  0xdc465cd155a90943ull, 0xddea645805b79275ull, 0xdf904bb0e1af1f06ull, 0xe138172913693ef6ull, \
  0xe2e1cb1ca47d25b3ull, 0xe437bdbf5254459cull, 0xe5e4ec24490fa711ull, 0xe73dacf671b3e66cull, \
  0xe8ee647894157a03ull, 0xeaa1194b37b8a383ull, 0xebfe4f049faa5e1eull, 0xed5cd0271114751cull, \
  0xef14c7605d60654cull, 0xf0763b3e66d6302full, 0xf231e9d66a7ab75cull, 0xf3965d3deaea945cull, \
  0xf4fc29f8202df4deull, 0xf66352a4ab03c266ull, 0xf82632d4c1e5a98eull, 0xf99074222d94cf6bull, \
  0xfafc1a1e65e8b5b3ull, 0xfc69278a85d754e9ull, 0xfdd79f2fdb445e41ull, 0xff4783e007ac54daull
// nearest integer to 2^(j / 128) 2^63
#define MCFD_POW_T \
  0x8000000000000000ull, 0x80b1ed4fd999ab6cull, 0x8164d1f3bc030773ull, 0x8218af4373fc25ecull, \
  0x82cd8698ac2ba1d7ull, 0x8383594eefb6ee37ull, 0x843a28c3acde4046ull, 0x84f1f656379c1a29ull, \
  0x85aac367cc487b15ull, 0x8664915b923fba04ull, 0x871f61969e8d1010ull, 0x87db357ff698d792ull, \
  0x88980e8092da8527ull, 0x8955ee03618e5fddull, 0x8a14d575496efd9aull, 0x8ad4c6452c728924ull, \
  0x8b95c1e3ea8bd6e7ull, 0x8c57c9c4646f4ddeull, 0x8d1adf5b7e5ba9e6ull, 0x8ddf042022e69cd6ull, \
  0x8ea4398b45cd53c0ull, 0x8f6a8117e6c8e5c4ull, 0x9031dc431466b1dcull, 0x90fa4c8beee4b12bull, \
  0x91c3d373ab11c336ull, 0x928e727d9531f9acull, 0x935a2b2f13e6e92cull, 0x9426ff0fab1c04b6ull, \
  0x94f4efa8fef70961ull, 0x95c3fe86d6cc7fefull, 0x96942d3720185a00ull, 0x97657d49f17ab08eull, \
  0x9837f0518db8a96full, 0x990b87e266c189aaull, 0x99e0459320b7fa65ull, 0x9ab62afc94ff864aull, \
  0x9b8d39b9d54e5539ull, 0x9c6573682ec32c2dull, 0x9d3ed9a72cffb751ull, 0x9e196e189d472420ull, \
  0x9ef5326091a111aeull, 0x9fd228256400dd06ull, 0xa0b0510fb9714fc2ull, 0xa18faeca8544b6e4ull, \
  0xa27043030c496819ull, 0xa3520f68e802bb93ull, 0xa43515ae09e6809eull, 0xa5195786be9ef339ull, \
  0xa5fed6a9b15138eaull, 0xa6e594cfeee86b1eull, 0xa7cd93b4e965356aull, 0xa8b6d5167b320e09ull, \
  0xa9a15ab4ea7c0ef8ull, 0xaa8d2652ec907629ull, 0xab7a39b5a93ed337ull, 0xac6896a4be3fe929ull, \
  0xad583eea42a14ac6ull, 0xae493452ca35b80eull, 0xaf3b78ad690a4375ull, 0xb02f0dcbb6e04584ull, \
  0xb123f581d2ac2590ull, 0xb21a31a66618fe3bull, 0xb311c412a9112489ull, 0xb40aaea2654b9841ull, \
  0xb504f333f9de6484ull, 0xb60093a85ed5f76cull, 0xb6fd91e328d17791ull, 0xb7fbefca8ca41e7cull, \
  0xb8fbaf4762fb9ee9ull, 0xb9fcd2452c0b9debull, 0xbaff5ab2133e45fbull, 0xbc034a7ef2e9fb0dull, \
  0xbd08a39f580c36bfull, 0xbe0f6809860993e2ull, 0xbf1799b67a731083ull, 0xc0213aa1f0d08db0ull, \
  0xc12c4cca66709456ull, 0xc238d2311e3d6673ull, 0xc346ccda24976407ull, 0xc4563ecc5334cb33ull, \
  0xc5672a115506daddull, 0xc67990b5aa245f79ull, 0xc78d74c8abb9b15dull, 0xc8a2d85c8ffe2c45ull, \
  0xc9b9bd866e2f27a3ull, 0xcad2265e4290774eull, 0xcbec14fef2727c5dull, 0xcd078b86503dcdd2ull, \
  0xce248c151f8480e4ull, 0xcf4318cf191918c1ull, 0xd06333daef2b2595ull, 0xd184df6251699ac6ull, \
  0xd2a81d91f12ae45aull, 0xd3ccf099859ac379ull, 0xd4f35aabcfedfa1full, 0xd61b5dfe9f9bce07ull, \
  0xd744fccad69d6af4ull, 0xd870394c6db32c84ull, 0xd99d15c278afd7b6ull, 0xdacb946f2ac9cc72ull, \
  0xdbfbb797daf23755ull, 0xdd2d818508324c20ull, 0xde60f4825e0e9124ull, 0xdf9612deb8f04420ull, \
  0xe0ccdeec2a94e111ull, 0xe2055afffe83d369ull, 0xe33f8972be8a5a51ull, 0xe47b6ca0373da88dull, \
  0xe5b906e77c8348a8ull, 0xe6f85aaaee1fce22ull, 0xe8396a503c4bdc68ull, 0xe97c38406c4f8c57ull, \
  0xeac0c6e7dd24392full, 0xec0718b64c1cbddcull, 0xed4f301ed9942b84ull, 0xee990f980da3025bull, \
  0xefe4b99bdcdaf5cbull, 0xf13230a7ad094509ull, 0xf281773c59ffb13aull, 0xf3d28fde3a641a5bull, \
  0xf5257d152486cc2cull, 0xf67a416c733f846eull, 0xf7d0df730ad13bb9ull, 0xf92959bb5dd4ba74ull, \
  0xfa83b2db722a033aull, 0xfbdfed6ce5f09c49ull, 0xfd3e0c0cf486c175ull, 0xfe9e115c7b8f884cull

#if defined(__CUDACC__)
static __device__ const unsigned short kPowR_dev[128] = {MCFD_POW_R};
static __device__ const u64 kPowL_dev[128] = {MCFD_POW_L};
static __device__ const u64 kPowT_dev[128] = {MCFD_POW_T};
#endif
#if !defined(__CUDA_ARCH__)
static const unsigned short kPowR_host[128] = {MCFD_POW_R};
static const u64 kPowL_host[128] = {MCFD_POW_L};
static const u64 kPowT_host[128] = {MCFD_POW_T};
#define MCFD_POW_TABLE(name) name##_host
#else
#define MCFD_POW_TABLE(name) name##_dev
#endif
#undef MCFD_POW_R
#undef MCFD_POW_L
#undef MCFD_POW_T

MCFD_IA_SLOW double pow_fp64(double x, double y) { return pow(x, y); }

// high 64 bits of a signed product
MCFD_IA_FN long long mulhi_signed(long long a, long long b) {
#if defined(__CUDA_ARCH__)
  return __mul64hi(a, b);
#else
  return (long long)(((__int128)a * b) >> 64);
#endif
}

MCFD_IA_SLOW double pow_rn(double x, double y) {
  const u64 ix = bits(x), iy = bits(y);
  const unsigned ex = (unsigned)(ix >> 52), ey = (unsigned)(iy >> 52) & 0x7ffu;  // ex with the sign: 1..2046 positive normal
  const int sh = 1075 - (int)ey;  // y = significand 2^-sh
  // |y| in [2^-40, 64]
  if (ex - 1u >= 0x7feu || sh < 46 || sh > 92 || (sh == 46 && (iy & kMant) != 0ull)) return pow_fp64(x, y);
  const u64 mx = (ix & kMant) | kImpl, my = (iy & kMant) | kImpl;
  // ---- log2 x = E + frac, frac in units of 2^-64
  const int j = (int)(mx >> 45) & 127;
  const long long z = (long long)(mx * (u64)MCFD_POW_TABLE(kPowR)[j] - 0x8000000000000000ull);  // z 2^63, exact
  const long long zz = (long long)((u64)z << 7);  // z 2^70
  // log2(1 + z) = z (a1 + a2 z + ... + a8 z^7), coefficients and partial sums
  // times 2^62: a product with zz is its value times 2^68, hence the shifts
#define MCFD_TIMES_Z(q) (mulhi_signed((q), zz) >> 6)
  const long long a1 = 0x5c551d94ae0bf85ell, a2 = -0x2e2a8eca5705fc2fll, a3 = 0x1ec709dc3a03fd75ll, a4 = -0x171547652b82fe17ll,
                  a5 = 0x12776c50ef9bfe79ll, a6 = -0xf6384ee1d01feball, a7 = 0xd30bb153d6f6ca0ll, a8 = -0xb8aa3b295c17f0cll;
  const long long z2 = mulhi_signed(zz, zz);  // z^2 2^76
  const long long p12 = a1 + MCFD_TIMES_Z(a2), p34 = a3 + MCFD_TIMES_Z(a4), p56 = a5 + MCFD_TIMES_Z(a6),
                  p78 = a7 + MCFD_TIMES_Z(a8);
#undef MCFD_TIMES_Z
  const long long z4 = mulhi_signed(z2, z2);  // z^4 2^88
  const long long lo4 = p12 + (mulhi_signed(p34, z2) >> 12), hi4 = p56 + (mulhi_signed(p78, z2) >> 12);
  const long long series = lo4 + (mulhi_signed(hi4, z4) >> 24);
  const long long lg = mulhi_signed(series, zz);  // log2(1 + z) 2^68
  const u64 tab = MCFD_POW_TABLE(kPowL)[j];
  // 128-bit sum: E 2^64 + table + lg / 16
  const u64 add = (u64)(lg >> 4);
  const u64 f = tab + add;
  long long hi = (long long)(int)ex - 1023 + (lg >> 63) + (f < tab ? 1 : 0);
  // ---- w = |y| |log2 x|, then its sign
  const bool neg_log = hi < 0;
  u64 t0 = f, t1 = (u64)hi;
  if (neg_log) {
    t0 = 0ull - f;
    t1 = ~(u64)hi + (f == 0ull ? 1ull : 0ull);
  }
  const u64 w0 = t0 * my;                        // 128-bit product, t1 < 2^11
  const u64 w1 = mulhi(t0, my) + t1 * my;
  u64 F, I;  // (w1 : w0) >> sh, 46 <= sh <= 92
  if (sh < 64) {
    F = (w0 >> sh) | (w1 << (64 - sh));
    I = w1 >> sh;
  } else {
    F = sh == 64 ? w1 : w1 >> (sh - 64);
    I = 0ull;
  }
  long long n = (long long)I;
  if (neg_log != ((iy >> 63) != 0ull)) {
    F = 0ull - F;
    n = -n - (F != 0ull ? 1 : 0);
  }
  // ---- 2^F
  const int i = (int)(F >> 57);
  const u64 g = F << 7;  // the remaining fraction times 2^71
  const u64 b1 = 0xb17217f7d1cf79acull, b2 = 0x3d7f7bff058b1d51ull, b3 = 0xe35846b82505fc6ull, b4 = 0x276556df749cee5ull,
            b5 = 0x5761ff9e299cc4ull, b6 = 0xa184897c363c4ull, b7 = 0xffe5fe2c4586ull;
  // partial sums times 2^64; a product with g is its value times 2^71
  const u64 g2 = mulhi(g, g);  // g^2 2^78
  const u64 q12 = b1 + (mulhi(b2, g) >> 7), q34 = b3 + (mulhi(b4, g) >> 7), q56 = b5 + (mulhi(b6, g) >> 7);
  const u64 g4 = mulhi(g2, g2);  // g^4 2^92
  const u64 q14 = q12 + (mulhi(q34, g2) >> 14), q57 = q56 + (mulhi(b7, g2) >> 14);
  const u64 q = q14 + (mulhi(q57, g4) >> 28);
  const u64 em1 = mulhi(q, g);  // (2^g - 1) 2^71
  const u64 base = MCFD_POW_TABLE(kPowT)[i];
  u64 m = base + (mulhi(base, em1) >> 7);
  if (m < base) m = ~0ull;  // rounded past 2: the rounding below gives 2
  // ---- round to 53 bits
  const u64 up = m + 1024ull;
  const bool carry = up < m;
  const u64 sig = carry ? 0ull : (up >> 11) & kMant;
  const long long e = n + 1023 + (carry ? 1 : 0);
  if (e < 1 || e > 2046) return pow_fp64(x, y);
  return from_bits(((u64)e << 52) | sig);
}

}  // namespace ia

using ia::pow_rn;

}  // namespace mcfd

#undef MCFD_POW_TABLE
#undef MCFD_IA_FN
#undef MCFD_IA_SLOW
