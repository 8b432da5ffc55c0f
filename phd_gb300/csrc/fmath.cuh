// FP64 elementary functions off the FP64 pipe.
//
// The GB300 SM starts two FP64 operations a clock (measured 1.96) and 128
// 32-bit ones, and the division, reciprocal, exponential and logarithm of
// the CUDA library are chains of FP64 operations: measured in slots of that
// pipe, 1/x takes 5.4, a/x 9, exp 19, log 36 and pow 100.  The reciprocal and
// the quotient here take a seed from the special-function unit and as few
// FP64 operations as reach the rounding of the format, by published methods
// named at each, from which their bounds follow; exp, log and x^y are
// evaluated in 64-bit fixed point on the integer pipes (about 75, 100 and 170
// instructions, no FP64 operation), within 0.53 ulp (exp, |x| < 16), 0.52 (log,
// |log x| >= 1/2) and 0.55 (x^y) where the library's bounds are 1 and 2.
//
// Fixed-point method: table-driven reduction (P. T. P. Tang, ACM TOMS 15, 1989
// and 16, 1990) with 128 table entries.  exp: x log2(e) = k + j/128 + r, the
// value 2^k T_j 2^r with T_j = 2^(j/128).  log2: x = 2^e m, m c_j = 1 + r with
// c_j just above 1 / (1 + j/128), the value e - log2(c_j) + log2(1 + r).  The
// polynomials in rho = 128 r interpolate at the Chebyshev nodes of [0, 1]
// (errors 7e-20 and 2e-19); all coefficients are in units of 2^-64.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

// T_j = 2^(j/128) in units of 2^-63
#define FM_EXP_TAB \
    0x8000000000000000ULL, 0x80b1ed4fd999ab6cULL, 0x8164d1f3bc030773ULL, 0x8218af4373fc25ecULL, \
    0x82cd8698ac2ba1d7ULL, 0x8383594eefb6ee37ULL, 0x843a28c3acde4046ULL, 0x84f1f656379c1a29ULL, \
    0x85aac367cc487b15ULL, 0x8664915b923fba04ULL, 0x871f61969e8d1010ULL, 0x87db357ff698d792ULL, \
    0x88980e8092da8527ULL, 0x8955ee03618e5fddULL, 0x8a14d575496efd9aULL, 0x8ad4c6452c728924ULL, \
    0x8b95c1e3ea8bd6e7ULL, 0x8c57c9c4646f4ddeULL, 0x8d1adf5b7e5ba9e6ULL, 0x8ddf042022e69cd6ULL, \
    0x8ea4398b45cd53c0ULL, 0x8f6a8117e6c8e5c4ULL, 0x9031dc431466b1dcULL, 0x90fa4c8beee4b12bULL, \
    0x91c3d373ab11c336ULL, 0x928e727d9531f9acULL, 0x935a2b2f13e6e92cULL, 0x9426ff0fab1c04b6ULL, \
    0x94f4efa8fef70961ULL, 0x95c3fe86d6cc7fefULL, 0x96942d3720185a00ULL, 0x97657d49f17ab08eULL, \
    0x9837f0518db8a96fULL, 0x990b87e266c189aaULL, 0x99e0459320b7fa65ULL, 0x9ab62afc94ff864aULL, \
    0x9b8d39b9d54e5539ULL, 0x9c6573682ec32c2dULL, 0x9d3ed9a72cffb751ULL, 0x9e196e189d472420ULL, \
    0x9ef5326091a111aeULL, 0x9fd228256400dd06ULL, 0xa0b0510fb9714fc2ULL, 0xa18faeca8544b6e4ULL, \
    0xa27043030c496819ULL, 0xa3520f68e802bb93ULL, 0xa43515ae09e6809eULL, 0xa5195786be9ef339ULL, \
    0xa5fed6a9b15138eaULL, 0xa6e594cfeee86b1eULL, 0xa7cd93b4e965356aULL, 0xa8b6d5167b320e09ULL, \
    0xa9a15ab4ea7c0ef8ULL, 0xaa8d2652ec907629ULL, 0xab7a39b5a93ed337ULL, 0xac6896a4be3fe929ULL, \
    0xad583eea42a14ac6ULL, 0xae493452ca35b80eULL, 0xaf3b78ad690a4375ULL, 0xb02f0dcbb6e04584ULL, \
    0xb123f581d2ac2590ULL, 0xb21a31a66618fe3bULL, 0xb311c412a9112489ULL, 0xb40aaea2654b9841ULL, \
    0xb504f333f9de6484ULL, 0xb60093a85ed5f76cULL, 0xb6fd91e328d17791ULL, 0xb7fbefca8ca41e7cULL, \
    0xb8fbaf4762fb9ee9ULL, 0xb9fcd2452c0b9debULL, 0xbaff5ab2133e45fbULL, 0xbc034a7ef2e9fb0dULL, \
    0xbd08a39f580c36bfULL, 0xbe0f6809860993e2ULL, 0xbf1799b67a731083ULL, 0xc0213aa1f0d08db0ULL, \
    0xc12c4cca66709456ULL, 0xc238d2311e3d6673ULL, 0xc346ccda24976407ULL, 0xc4563ecc5334cb33ULL, \
    0xc5672a115506daddULL, 0xc67990b5aa245f79ULL, 0xc78d74c8abb9b15dULL, 0xc8a2d85c8ffe2c45ULL, \
    0xc9b9bd866e2f27a3ULL, 0xcad2265e4290774eULL, 0xcbec14fef2727c5dULL, 0xcd078b86503dcdd2ULL, \
    0xce248c151f8480e4ULL, 0xcf4318cf191918c1ULL, 0xd06333daef2b2595ULL, 0xd184df6251699ac6ULL, \
    0xd2a81d91f12ae45aULL, 0xd3ccf099859ac379ULL, 0xd4f35aabcfedfa1fULL, 0xd61b5dfe9f9bce07ULL, \
    0xd744fccad69d6af4ULL, 0xd870394c6db32c84ULL, 0xd99d15c278afd7b6ULL, 0xdacb946f2ac9cc72ULL, \
    0xdbfbb797daf23755ULL, 0xdd2d818508324c20ULL, 0xde60f4825e0e9124ULL, 0xdf9612deb8f04420ULL, \
    0xe0ccdeec2a94e111ULL, 0xe2055afffe83d369ULL, 0xe33f8972be8a5a51ULL, 0xe47b6ca0373da88dULL, \
    0xe5b906e77c8348a8ULL, 0xe6f85aaaee1fce22ULL, 0xe8396a503c4bdc68ULL, 0xe97c38406c4f8c57ULL, \
    0xeac0c6e7dd24392fULL, 0xec0718b64c1cbddcULL, 0xed4f301ed9942b84ULL, 0xee990f980da3025bULL, \
    0xefe4b99bdcdaf5cbULL, 0xf13230a7ad094509ULL, 0xf281773c59ffb13aULL, 0xf3d28fde3a641a5bULL, \
    0xf5257d152486cc2cULL, 0xf67a416c733f846eULL, 0xf7d0df730ad13bb9ULL, 0xf92959bb5dd4ba74ULL, \
    0xfa83b2db722a033aULL, 0xfbdfed6ce5f09c49ULL, 0xfd3e0c0cf486c175ULL, 0xfe9e115c7b8f884cULL
// c_j = ceil(2^63 / (1 + j/128)), -log2(c_j 2^-63) in units of 2^-64
#define FM_LOG_TAB \
    {0x8000000000000000ULL, 0x0000000000000000ULL}, {0x7f01fc07f01fc080ULL, 0x02dfca16dde10a2dULL}, \
    {0x7e07e07e07e07e08ULL, 0x05b9e5a170b48a62ULL}, {0x7d1196792909c560ULL, 0x088e68ea899a0976ULL}, \
    {0x7c1f07c1f07c1f08ULL, 0x0b5d69bac77ec398ULL}, {0x7b301ecc07b301edULL, 0x0e26fd5c8555af7aULL}, \
    {0x7a44c6afc2dd9ca9ULL, 0x10eb389fa29f9ab1ULL}, {0x795ceb240795ceb3ULL, 0x13aa2fdd27f1c2d6ULL}, \
    {0x7878787878787879ULL, 0x1663f6fac913167bULL}, {0x77975b8fe21a291dULL, 0x1918a16e46335aabULL}, \
    {0x76b981dae6076b99ULL, 0x1bc84240adabba61ULL}, {0x75ded952e0b0ce46ULL, 0x1e72ec117fa5b21dULL}, \
    {0x7507507507507508ULL, 0x2118b119b4f3c72aULL}, {0x7432d63dbb01d0ccULL, 0x23b9a32eaa56f6bbULL}, \
    {0x73615a240e6c2b45ULL, 0x2655d3c4f15c343dULL}, {0x7292cc157b864408ULL, 0x28ed53f307ee9a60ULL}, \
    {0x71c71c71c71c71c8ULL, 0x2b803473f7ad0f3cULL}, {0x70fe3c070fe3c071ULL, 0x2e0e85a9de04fe53ULL}, \
    {0x70381c0e070381c1ULL, 0x309857a05e0765fbULL}, {0x6f74ae26501bdd2cULL, 0x331dba0efce1be04ULL}, \
    {0x6eb3e45306eb3e46ULL, 0x359ebc5b69d927ddULL}, {0x6df5b0f768ce2cacULL, 0x381b6d9bb29bdc81ULL}, \
    {0x6d3a06d3a06d3a07ULL, 0x3a93dc9864b2df91ULL}, {0x6c80d901b2036407ULL, 0x3d0817ce9cd4998fULL}, \
    {0x6bca1af286bca1b0ULL, 0x3f782d7204d01444ULL}, {0x6b15c06b15c06b16ULL, 0x41e42b6ec0c025bbULL}, \
    {0x6a63bd81a98ef607ULL, 0x444c1f6b4c2dd72bULL}, {0x69b4069b4069b407ULL, 0x46b016ca47c1c149ULL}, \
    {0x6906906906906907ULL, 0x49101eac381ce608ULL}, {0x685b4fe5e92c0686ULL, 0x4b6c43f1366abdbbULL}, \
    {0x67b23a5440cf6475ULL, 0x4dc4933a9337b365ULL}, {0x670b453b92840671ULL, 0x501918ec6c1125d6ULL}, \
    {0x6666666666666667ULL, 0x5269e12f346e2bf7ULL}, {0x65c393e032e1c9f1ULL, 0x54b6f7f1325acdf4ULL}, \
    {0x6522c3f35ba78195ULL, 0x570068e7ef5a1e7dULL}, {0x6483ed274388a357ULL, 0x59463f919dee9b92ULL}, \
    {0x63e7063e7063e707ULL, 0x5b8887367433795bULL}, {0x634c0634c0634c07ULL, 0x5dc74ae9fbecef8fULL}, \
    {0x62b2e43dafcea68eULL, 0x6002958c587150caULL}, {0x621b97c2aec12653ULL, 0x623a71cb82c89692ULL}, \
    {0x6186186186186187ULL, 0x646eea247c5c22cfULL}, {0x60f25deacafb74a4ULL, 0x66a008e4788cbcd1ULL}, \
    {0x6060606060606061ULL, 0x68cdd829fd814274ULL}, {0x5fd017f405fd0180ULL, 0x6af861e5fc7d2384ULL}, \
    {0x5f417d05f417d060ULL, 0x6d1fafdce20a828dULL}, {0x5eb4882383b30d52ULL, 0x6f43cba79e40c2abULL}, \
    {0x5e293205e293205fULL, 0x7164beb4a56d59f7ULL}, {0x5d9f7390d2a6c406ULL, 0x73829248e961f325ULL}, \
    {0x5d1745d1745d1746ULL, 0x759d4f80cba83bf8ULL}, {0x5c90a1fd1b7af018ULL, 0x77b4ff5108d93137ULL}, \
    {0x5c0b81702e05c0b9ULL, 0x79c9aa879d53482eULL}, {0x5b87ddad0cdf1b2dULL, 0x7bdb59cca38881f2ULL}, \
    {0x5b05b05b05b05b06ULL, 0x7dea15a32c1b3b37ULL}, {0x5a84f3454dca4110ULL, 0x7ff5e66a0ffe6ae5ULL}, \
    {0x5a05a05a05a05a06ULL, 0x81fed45cbccbf99bULL}, {0x5987b1a9448be406ULL, 0x8404e793fb81ea91ULL}, \
    {0x590b21642c8590b3ULL, 0x86082806b1d532c0ULL}, {0x588fe9dc0588fe9eULL, 0x88089d8a9e4753d8ULL}, \
    {0x5816058160581606ULL, 0x8a064fd50f2a1cefULL}, {0x579d6ee340579d6fULL, 0x8c01467b94bb5275ULL}, \
    {0x572620ae4c415c99ULL, 0x8df988f4ae806f1cULL}, {0x56b015ac056b015bULL, 0x8fef1e9874093211ULL}, \
    {0x563b48c20563b48dULL, 0x91e20ea1393e403dULL}, {0x55c7b4f141ace689ULL, 0x93d2602c2e5fc02bULL}, \
    {0x5555555555555556ULL, 0x95c01a39fbd6879dULL}, {0x54e42523d03fab1cULL, 0x97ab43af59f930a1ULL}, \
    {0x54741fab8be05475ULL, 0x9993e355a4e53640ULL}, {0x5405405405405406ULL, 0x9b79ffdb6c8b11ffULL}, \
    {0x5397829cbc14e5e1ULL, 0x9d5d9fd5010b3665ULL}, {0x532ae21c96bdb9d4ULL, 0x9f3ec9bcfb80b356ULL}, \
    {0x52bf5a814afd6a06ULL, 0xa11d83f4c3554b35ULL}, {0x5254e78ecb419ba9ULL, 0xa2f9d4c51039c525ULL}, \
    {0x51eb851eb851eb86ULL, 0xa4d3c25e68dc57eeULL}, {0x51832f1fd73e6871ULL, 0xa6ab52d99e76224fULL}, \
    {0x511be1958b67ebbaULL, 0xa8808c384547c6ebULL}, {0x50b59897547e1bbfULL, 0xaa5374652a1c6d8bULL}, \
    {0x5050505050505051ULL, 0xac241134c4e99e19ULL}, {0x4fec04fec04fec05ULL, 0xadf26865a8a1a557ULL}, \
    {0x4f88b2f392a409f2ULL, 0xafbe7fa0f04d75c2ULL}, {0x4f265691eeaf9d11ULL, 0xb1885c7aa98241ffULL}, \
    {0x4ec4ec4ec4ec4ec5ULL, 0xb35004723c465e69ULL}, {0x4e6470b061fd8cddULL, 0xb5157cf2d078503eULL}, \
    {0x4e04e04e04e04e05ULL, 0xb6d8cb53b0ca4ecbULL}, {0x4da637cf781d1e55ULL, 0xb899f4d8ab63df28ULL}, \
    {0x4d4873ecade304d5ULL, 0xba58feb2703a9e35ULL}, {0x4ceb916d5ef2c784ULL, 0xbc15edfeed32bbd9ULL}, \
    {0x4c8f8d28ac42fd9cULL, 0xbdd0c7c9a817204dULL}, {0x4c346404c346404dULL, 0xbf89910c1678ae86ULL}, \
    {0x4bda12f684bda130ULL, 0xc1404eadf38396dcULL}, {0x4b8097012e025c05ULL, 0xc2f5058593d93083ULL}, \
    {0x4b27ed3604b27ed4ULL, 0xc4a7ba58377c5a00ULL}, {0x4ad012b404ad012cULL, 0xc65871da59dded98ULL}, \
    {0x4a7904a7904a7905ULL, 0xc80730b0001667f0ULL}, {0x4a22c04a22c04a23ULL, 0xc9b3fb6d055974e5ULL}, \
    {0x49cd42e2049cd42fULL, 0xcb5ed69565afaf7bULL}, {0x497889c2024bc44fULL, 0xcd07c69d87027ef0ULL}, \
    {0x4924924924924925ULL, 0xceaecfea80859b31ULL}, {0x48d159e26af37c05ULL, 0xd053f6d26089672fULL}, \
    {0x487ede0487ede049ULL, 0xd1f73f9c70c0f681ULL}, {0x482d1c319f03621eULL, 0xd398ae8179063de7ULL}, \
    {0x47dc11f7047dc120ULL, 0xd53847ac00a69be4ULL}, {0x478bbcecfee1d10dULL, 0xd6d60f388e419687ULL}, \
    {0x473c1ab68a0473c2ULL, 0xd8720935e6435ebcULL}, {0x46ed29011bb4a405ULL, 0xda0c39a548045ec9ULL}, \
    {0x469ee58469ee5847ULL, 0xdba4a47aa996d258ULL}, {0x46514e02328a7012ULL, 0xdd3b4d9cf24b2076ULL}, \
    {0x4604604604604605ULL, 0xded038e633f36da5ULL}, {0x45b81a2509cde3aeULL, 0xe0636a23e2ee9b13ULL}, \
    {0x456c797dd49c3412ULL, 0xe1f4e5170d02a998ULL}, {0x45217c382b34eda4ULL, 0xe384ad748f0e3b01ULL}, \
    {0x44d72044d72044d8ULL, 0xe512c6e54998b1abULL}, {0x448d639d74c0cda9ULL, 0xe69f35065448360eULL}, \
    {0x4444444444444445ULL, 0xe829fb693044b395ULL}, {0x43fbc043fbc043fcULL, 0xe9b31d93f98ea94aULL}, \
    {0x43b3d5af9a723f79ULL, 0xeb3a9f01975077f0ULL}, {0x436c82a23d1a5664ULL, 0xecc08321eb30a619ULL}, \
    {0x4325c53ef368eb05ULL, 0xee44cd59ffab62efULL}, {0x42df9bb096771e4eULL, 0xefc781043579625cULL}, \
    {0x429a0429a0429a05ULL, 0xf148a170700a00f9ULL}, {0x4254fce404254fcfULL, 0xf2c831e4411672adULL}, \
    {0x4210842108421085ULL, 0xf446359b1353954cULL}, {0x41cc98291fdf19b4ULL, 0xf5c2afc65447d86aULL}, \
    {0x4189374bc6a7ef9eULL, 0xf73da38d9d4a83eaULL}, {0x41465fdf5cd01052ULL, 0xf8b7140edbb181d7ULL}, \
    {0x4104104104104105ULL, 0xfa2f045e7832aa6dULL}, {0x40c246d47d78693cULL, 0xfba577877d7d6ebbULL}, \
    {0x4081020408102041ULL, 0xfd1a708bbe119b12ULL}, {0x4040404040404041ULL, 0xfe8df263f957ca11ULL}

static __device__ const unsigned long long fm_exp_tab_dev[128] = {FM_EXP_TAB};
static __device__ const ulonglong2 fm_log_tab_dev[128] = {FM_LOG_TAB};
static const unsigned long long fm_exp_tab_host[128] = {FM_EXP_TAB};
static const ulonglong2 fm_log_tab_host[128] = {FM_LOG_TAB};

#define FM_HD __host__ __device__ __forceinline__

FM_HD unsigned long long fm_bits(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
FM_HD double fm_from_bits(unsigned long long u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
FM_HD unsigned long long fm_mulhi(unsigned long long a, unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (unsigned long long)(((unsigned __int128)a * b) >> 64);
#endif
}
FM_HD unsigned fm_mulhi32(unsigned a, unsigned b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (unsigned)(((unsigned long long)a * b) >> 32);
#endif
}
FM_HD int fm_clz(unsigned long long a) {   // a != 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)a);
#else
  return __builtin_clzll(a);
#endif
}

// 2^(k + f 2^-64) for |k| < 1000
FM_HD double fm_exp2_fix(int k, unsigned long long f) {
  const int j = (int)(f >> 57);
#ifdef __CUDA_ARCH__
  const unsigned long long t = __ldg(fm_exp_tab_dev + j);
#else
  const unsigned long long t = fm_exp_tab_host[j];
#endif
  const unsigned long long rho = f << 7;
  const unsigned r32 = (unsigned)(rho >> 32);
  const unsigned q4 = 0x27655158u + fm_mulhi32(0xaf291u, r32);
  const unsigned long long q3 = 0x71ac235e0cULL + fm_mulhi32(q4, r32);
  const unsigned long long q2 = 0xf5fdeffc15edULL + fm_mulhi(q3, rho);
  const unsigned long long q1 = 0x162e42fefa39ef5ULL + fm_mulhi(q2, rho);
  unsigned long long s = t + fm_mulhi(t, fm_mulhi(q1, rho));
  s = s < t ? ~0ULL : s;   // just below 2
  return fm_from_bits(((unsigned long long)(unsigned)(k + 1022) << 52) + (s >> 11) + ((s >> 10) & 1));
}

// log2(x) of a positive normal x: the integer part and the fraction in
// units of 2^-64 (error below 2^-61)
FM_HD unsigned long long fm_log2_fix(unsigned long long bits, int& e) {
  e = (int)(bits >> 52) - 1023;
  const unsigned long long m = (bits << 11) | (1ULL << 63);   // units of 2^-63
  const int j = (int)((m >> 56) & 127);
#ifdef __CUDA_ARCH__
  const ulonglong2 c = __ldg(fm_log_tab_dev + j);
#else
  const ulonglong2 c = fm_log_tab_host[j];
#endif
  const unsigned long long rho = fm_mulhi(m, c.x) << 9;   // 128 (m c - 1), units of 2^-64
  const unsigned r32 = (unsigned)(rho >> 32);
  const unsigned q5 = 0x93b5e9eu - fm_mulhi32(0xf1562u, r32);
  const unsigned long long q4 = 0x5c551abfdULL - fm_mulhi32(q5, r32);
  const unsigned long long q3 = 0x3d8e13b7ca5ULL - fm_mulhi(q4, rho);
  const unsigned long long q2 = 0x2e2a8eca56f77ULL - fm_mulhi(q3, rho);
  const unsigned long long q1 = 0x2e2a8eca5705fc0ULL - fm_mulhi(q2, rho);
  const unsigned long long p = fm_mulhi(q1, rho), f = c.y + p;
  return f < p ? ~0ULL : f;   // just below 1
}

// exp(x).  |x| < 128 in fixed point; beyond, 0 and infinity where the result
// is certain to under- or overflow, else the library's.
FM_HD double fm_exp(double x) {
  const unsigned long long u = fm_bits(x);
  const unsigned long long a = u & 0x7fffffffffffffffULL;
  if (a >= 0x4060000000000000ULL) {   // |x| >= 128, infinity or NaN
    if (u > 0xc088000000000000ULL && a <= 0x7ff0000000000000ULL) return 0.0;   // x < -768
    return exp(x);
  }
  const unsigned long long m = (u << 11) | (1ULL << 63);
  const unsigned long long p = fm_mulhi(m, 0xb8aa3b295c17f0bcULL);   // |x| log2(e) in units of 2^-sh
  const int sh = 1085 - (int)(a >> 52);                              // 56 or more
  unsigned long long f = 0;
  int k = 0;
  if (sh < 64) {
    f = p << (64 - sh);
    k = (int)(p >> sh);
  } else if (sh < 128) {
    f = p >> (sh - 64);
  }
  if (u >> 63) {
    k = -k - (f != 0 ? 1 : 0);
    f = 0 - f;
  }
  return fm_exp2_fix(k, f);
}

// log(x) of a positive normal x; others go to the library.  So does 1 - 2^-6 <=
// x < 1 + 2^-6: the fixed-point error is absolute (2^-61), and nearer to 1 it
// would be more than a quarter of the result's last place (at 2^-6 the result
// is above 2^-7), without limit as x goes to 1.  The learned chemistry takes
// the logarithm of pressures near 1 atm.
FM_HD double fm_log(double x) {
  const unsigned long long u = fm_bits(x);
  if (u - 0x0010000000000000ULL >= 0x7fe0000000000000ULL || u - 0x3fef800000000000ULL < 0x0000c00000000000ULL)
    return log(x);
  int e;
  unsigned long long f = fm_log2_fix(u, e);
  const unsigned long long neg = (unsigned long long)(unsigned)(e >> 31) >> 31;   // 1 for x < 1
  // |log2 x| = h + f
  unsigned h = (unsigned)e;
  if (neg) {
    h = (unsigned)(-e) - (f != 0 ? 1u : 0u);
    f = 0 - f;
  }
  // times ln 2
  const unsigned long long ln2 = 0xb17217f7d1cf79acULL;
  unsigned long long lo = (unsigned long long)h * ln2, hi = fm_mulhi((unsigned long long)h, ln2);
  const unsigned long long fl = fm_mulhi(f, ln2);
  lo += fl;
  hi += lo < fl ? 1 : 0;
  if ((hi | lo) == 0) return 0.0;
  int z, ex;
  unsigned long long s;
  if (hi) {
    z = fm_clz(hi);   // 54 or more
    s = (hi << z) | (lo >> (64 - z));
    ex = 63 - z;
  } else {
    z = fm_clz(lo);
    s = lo << z;
    ex = -1 - z;
  }
  return fm_from_bits(((neg << 63) | ((unsigned long long)(unsigned)(ex + 1022) << 52)) + (s >> 11) + ((s >> 10) & 1));
}

// x^y for y in (0, 1] (a root's exponent): 2^(y log2 x), the product kept in
// fixed point; other arguments go to the library
FM_HD double fm_root(double x, double y) {
  const unsigned long long u = fm_bits(x), v = fm_bits(y);
  // y in [2^-10, 1], x positive and normal
  if (u - 0x0010000000000000ULL >= 0x7fe0000000000000ULL || v - 0x3f50000000000000ULL > 0x00a0000000000000ULL)
    return pow(x, y);
  int e;
  unsigned long long f = fm_log2_fix(u, e);
  const bool neg = e < 0;
  unsigned h = (unsigned)e;
  if (neg) {
    h = (unsigned)(-e) - (f != 0 ? 1u : 0u);
    f = 0 - f;
  }
  const unsigned long long m = (v << 11) | (1ULL << 63);   // y in units of 2^-sh
  const int sh = 1086 - (int)(v >> 52);                    // 63 .. 73
  // (h + f) y in units of 2^-sh (hi:lo, hi < 2^11)
  unsigned long long lo = (unsigned long long)h * m, hi = fm_mulhi((unsigned long long)h, m);
  const unsigned long long fl = fm_mulhi(f, m);
  lo += fl;
  hi += lo < fl ? 1 : 0;
  // to units of 2^-64
  int k;
  unsigned long long g;
  if (sh == 63) {
    g = lo << 1;
    k = (int)((hi << 1) | (lo >> 63));
  } else if (sh == 64) {
    g = lo;
    k = (int)hi;
  } else {
    g = (lo >> (sh - 64)) | (hi << (128 - sh));
    k = (int)(hi >> (sh - 64));
  }
  if (neg) {
    k = -k - (g != 0 ? 1 : 0);
    g = 0 - g;
  }
  if (k <= -1000 || k >= 1000) return pow(x, y);
  return fm_exp2_fix(k, g);
}

#ifdef __CUDACC__
// true when |x| is in [2^-900, 2^900): the seed, its square and the products
// below then neither overflow nor lose bits to underflow
__device__ __forceinline__ bool fm_mid(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  return e - 123u < 1800u;
}

// The seed of both: PTX rcp.approx.ftz.f64, which the special-function unit
// forms from the upper 32 bits of x.  e = 1 - x y is below 2^-19.9 in magnitude
// (measured over every upper word of a binade, the lower word at both its ends).
__device__ __forceinline__ double fm_rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// the library's forms for the arguments outside the seed's range, out of line
static __device__ __noinline__ double fm_div_general(double a, double x) { return a / x; }

// 1 / x.  With a seed y and e = 1 - x y, 1 / x = y / (1 - e) = y (1 + e + e^2 +
// ...): the geometric series of functional iteration (M. J. Flynn, On division
// by functional iteration, IEEE Trans. Comput. C-19, 1970), here cut after e^2.
// Left out: |e|^3 / (1 - e) < 2^-59.6.  Roundings: of e and of e + e^2, 2^-72 of
// the result each; of the last operation.  Together below 0.6 units of the last
// place.  3 slots against 5.4 of 1.0 / x.
__device__ __forceinline__ double fm_rcp(double x) {
  if (!fm_mid(x)) return fm_div_general(1.0, x);
  const double y = fm_rcp_seed(x);
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// a / x.  The series above cut after e gives y to e^2 < 2^-39.8; then the
// quotient q = a y and its remainder a - x q, one fused operation, folded back as
// q + (a - x q) y (P. W. Markstein, Computation of elementary functions on the
// IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  q is off by less
// than 2^-39 of itself and y by 2^-39: the correction leaves 2^-78, and its
// remainder's rounding 2^-92, beside the rounding of the last operation: below
// 0.51 units of the last place.  5 slots against 9 of a / x.
__device__ __forceinline__ double fm_div(double a, double x) {
  const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu;
  const unsigned ex = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  // the quotient and the remainder stay normal (a = 0 takes the general form)
  if (!(ex - 523u < 1000u) || !(ea - 523u < 1000u)) return fm_div_general(a, x);
  double y = fm_rcp_seed(x);
  y = fma(y, fma(-x, y, 1.0), y);
  const double q = a * y;
  return fma(fma(-x, q, a), y, q);
}

// 1 / (a b) and what the roundings of the product and of the reciprocal leave
// over; fm_over takes x / (a b) from it with one rounding beyond those of x.
// Mole fractions X_k = (rho Y_k / W_k) / (rho W_i) of many species share it: rms
// error 0.60 units of 2^-53 (two roundings), 0.74 as one quotient a species
// (three), 0.85 as plain products with a reciprocal (four).
struct fm_pair {
  double hi, lo;
};
__device__ __forceinline__ fm_pair fm_rcp_prod(double a, double b) {
  const double p = a * b;
  fm_pair r;
  r.hi = fm_rcp(p);
  r.lo = fma(-fma(a, b, -p), r.hi, fma(-p, r.hi, 1.0)) * r.hi;
  return r;
}
__device__ __forceinline__ double fm_over(double x, const fm_pair& r) { return fma(x, r.hi, x * r.lo); }
#endif  // __CUDACC__
