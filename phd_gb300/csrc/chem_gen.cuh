// Generated by phd_gb300/mechgen.py from phd_gb300/data/h2_sandiego12.inp -- do not edit.
// The constant-volume reactor right-hand side of this mechanism (9 species,
// 12 reactions): the expressions and operation order of fun_tpart / fun_cpart
// in chem.cu, the composition part straight-line code with the mechanism's numbers
// as literals, the Arrhenius and NASA terms loops over constant tables.
#pragma once

namespace chem_gen {

constexpr int KK = 9;

// temperature terms of one right-hand side; the finite-difference Jacobian's
// species columns reuse them (rc_drive)
struct FunT {
  double T;
  double cvk[9], u[9];
  double k[20];   // forward rate constants, then
                 // reverse: k[12] of reaction 0, k[13] of reaction 1, k[14] of reaction 2, k[15] of reaction 5, k[16] of reaction 7, k[17] of reaction 8
                 // low- over high-pressure: k[18] of reaction 3, k[19] of reaction 11
  double lnfc[2], trc[2], trn[2];   // reactions 3, 11
};

HD __forceinline__ void cell_set(double rho, Cell<9>& c) {
  c.rho = rho;
  c.rho_i = c_rcp(rho);
  c.rw[0] = rho * 0x1.fbf39e8ab06bdp-1;
  c.rw[1] = rho * 0x1.fbf39e8ab06bdp-2;
  c.rw[2] = rho * 0x1.000275060987dp-4;
  c.rw[3] = rho * 0x1.000275060987dp-5;
  c.rw[4] = rho * 0x1.e1ac6c774b6a9p-5;
  c.rw[5] = rho * 0x1.c6b93cc1512cbp-5;
  c.rw[6] = rho * 0x1.f0620d016f133p-6;
  c.rw[7] = rho * 0x1.e1ac6c774b6a9p-6;
  c.rw[8] = rho * 0x1.246e76057aa8cp-5;
}

// A, b, E/R of the Arrhenius expressions; c_v (5) and internal energy (6)
// polynomials of the species below and above their middle temperature: in
// constant memory, so that the loops over them stay small code
#define CHEM_GEN_ARR {0x1.f438daa060000p+54, (-0x1.6666666666666p-1), 0x1.0c6f4493ef159p+13}, \
  {0x1.8b50000000000p+15, 0x1.55c28f5c28f5cp+1, 0x1.8bb78dad5b973p+11}, \
  {0x1.16f3220000000p+30, 0x1.4cccccccccccdp+0, 0x1.c94c533be761cp+10}, \
  {0x1.0eaa664900000p+42, 0x1.c28f5c28f5c29p-2, 0.0}, \
  {0x1.0191a36680000p+46, 0.0, 0x1.27e432c1d6dbcp+7}, \
  {0x1.e31fa34e00000p+43, 0.0, 0x1.9da4e3b0f0481p+8}, \
  {0x1.a48ce3be80000p+44, 0.0, (-0x1.f4328690d2d50p+7)}, \
  {0x1.0f0cf064dd592p+75, (-0x1.0000000000000p+1), 0.0}, \
  {0x1.20a871cc00200p+60, (-0x1.0000000000000p+0), 0.0}, \
  {0x1.5f93037c00000p+41, 0.0, 0x1.5dbc4f266b3c5p+9}, \
  {0x1.2dbf9ea000000p+37, 0x1.3851eb851eb85p-1, 0x1.784fcc6a9ac05p+13}, \
  {0x1.6b99192fbb3c0p+64, (-0x1.63d70a3d70a3dp+0), 0x1.93845131294f1p+14}, \
  {0x1.001d1bf800000p+46, (-0x1.0a3d70a3d70a4p-2), 0x1.1fd705d6afec6p+6}, \
  {0x1.d970000000000p+14, 0x1.50a3d70a3d70ap+1, 0x1.3072327bb03a1p+11}, \
  {0x1.7d78400000000p+33, 0x1.30a3d70a3d70ap+0, 0x1.2611369490098p+13}, \
  {0x1.39283f4a00000p+41, 0x1.70a3d70a3d70ap-2, 0x1.b3c1120ab0336p+14}, \
  {0x1.5cfa424ea9c92p+76, (-0x1.c000000000000p+0), 0x1.d22edd4d65d8ep+15}, \
  {0x1.0e0198eaee000p+58, (-0x1.4cccccccccccdp-1), 0x1.96e5d98de8289p+15}, \
  {0x1.8efc84ad0c7b0p+65, (-0x1.6666666666666p+0), 0.0}, \
  {0x1.592a7a2071df8p+79, (-0x1.e666666666666p+0), 0x1.8626719ec5abbp+14}
#define CHEM_GEN_NASA {{0x1.d7ff8e3825f4ap+26, 0x1.e80f506d97176p-15, (-0x1.618f1f2124b19p-23), 0x1.a159b3e796e12p-33, (-0x1.58a5073e4b9eap-44), 0x1.dbc2948000000p+26, 0x1.ebf31bfc7e509p-16, (-0x1.db2b52f348540p-25), 0x1.a4ad3a7f28bafp-35, (-0x1.15e9c4e98a5f0p-46), 0x1.ed233bd1877d7p+40},\
   {0x1.a703bf36dacefp+25, 0x1.416ed353acc12p+18, (-0x1.91ad45f2464bap+9), 0x1.a9a81b1e64e16p-1, (-0x1.3eff45c69d9bbp-12), 0x1.aa62d459f3e8ap+26, 0x1.43fea64415103p+18, (-0x1.0deb369d99cf1p+9), 0x1.ad0c943d898adp-2, (-0x1.013b4d2d53f55p-13), (-0x1.1c5226d289a30p+36)},\
   {0x1.57df0702624b6p+23, (-0x1.0a4760fffc8a1p+14), 0x1.142df148e6721p+5, (-0x1.04e222e912be3p-5), 0x1.7064d5077b11cp-17, 0x1.57dbba1b66128p+27, (-0x1.0a44d2be9b351p+17), 0x1.7039b8f006229p+7, (-0x1.04dfa1e972f78p-3), 0x1.26b43cb2fc852p-15, 0x1.19e28b1840f5cp+41},\
   {0x1.b946efc4d2fdfp+22, (-0x1.e6aa8d36d2990p+12), 0x1.99648ecb16b96p+4, (-0x1.9c26a8265042ep-6), 0x1.1acfc9fa7224ep-17, 0x1.b942b38987df5p+27, (-0x1.e6a5e175c5a15p+16), 0x1.10eb15ef57eafp+8, (-0x1.9c22b37b551ccp-3), 0x1.c47b51c30b00dp-15, (-0x1.498ba52fa8e56p+36)},\
   {0x1.be638f3b2cda6p+23, (-0x1.6edbe390f33afp+13), 0x1.69376e7fc9e9ap+4, (-0x1.36de921e0dd57p-6), 0x1.bf89d27355702p-18, 0x1.da7e6bc41fe43p+27, (-0x1.85f4e485c392bp+16), 0x1.fff1fd1306df8p+6, (-0x1.4a7123c5a5705p-4), 0x1.7c92918263fc0p-16, 0x1.17eef572b5062p+38},\
   {0x1.c283f5413bf48p+23, (-0x1.25b50a5c47d8cp+13), 0x1.e17dce03933eep+4, (-0x1.9efa92b9c77c9p-6), 0x1.12695e1c4f3e1p-17, 0x1.fb430727354c2p+27, (-0x1.4ab3c229620eap+16), 0x1.696d238bf995fp+7, (-0x1.d33fbf6ec423bp-4), 0x1.ee5c9ff7dc3cep-16, (-0x1.253957b89215cp+41)},\
   {0x1.fba6572f0804bp+22, (-0x1.75d97aeff7d43p+13), 0x1.aa631fd8dde89p+5, (-0x1.f4f71fad691fap-5), 0x1.88b6573d98807p-16, 0x1.05cf845b8a3e7p+28, (-0x1.819c8661bf38cp+17), 0x1.25338b451e123p+9, (-0x1.025cfd6548c8cp-1), 0x1.440dd8e369053p-13, 0x1.6d41439fa6a7fp+34},\
   {0x1.e8c63adc28e02p+22, (-0x1.4bb7770fc3119p+10), 0x1.4739e99066e29p+5, (-0x1.b0116b1462c59p-5), 0x1.61b13612ab5e8p-16, 0x1.03c620d38a85cp+28, (-0x1.609a0c5c905d5p+14), 0x1.cfc57df369b17p+8, (-0x1.cb4575097b96ap-2), 0x1.2cc4cbc47d3f0p-13, (-0x1.56b30f9872b5cp+40)},\
   {0x1.a06ada57d4d7ap+22, 0x1.053b974b3ad43p+12, (-0x1.786ac086d4cc8p+3), 0x1.12569ebcaabd9p-6, (-0x1.e6f8bd3e66063p-18), 0x1.6c8a22210be0ep+27, 0x1.c96049f42c623p+15, (-0x1.b75d027f34893p+6), 0x1.e05266401eba5p-4, (-0x1.550b13d1e1e8ap-15), (-0x1.3c3691c537d71p+36)}}, \
  {{0x1.d7ff8e6cf0bc7p+26, (-0x1.f32aafd504c46p-10), 0x1.65bd8cc3415b3p-20, (-0x1.ad75cad3044dep-32), 0x1.7226f20725a00p-45, 0x1.dbc294b5367e4p+26, (-0x1.f72524c339726p-11), 0x1.e0c9efcea8c6bp-22, (-0x1.b0e20692518c4p-34), 0x1.2a7b56674e2dap-47, 0x1.ed233bd1877d7p+40},\
   {0x1.6fbb06f3e5b32p+26, (-0x1.fd630b8827036p+10), 0x1.49979c41dcaacp+4, (-0x1.e55c2eb4b1988p-8), 0x1.bb6af52ee8c1dp-21, 0x1.72a95019fb3fap+27, (-0x1.00b92d53b22a4p+11), 0x1.baf5714c0eafbp+3, (-0x1.e93a782375008p-9), 0x1.658fbc3f4a5acp-22, (-0x1.264d47d19950bp+36)},\
   {0x1.f1cc1306e88bfp+22, (-0x1.bec9823789650p+8), 0x1.be74cdd8008b8p-3, (-0x1.b4b6123cca757p-15), 0x1.b6a98c2072389p-28, 0x1.f1c74bec7dcbfp+26, (-0x1.bec538726c729p+11), 0x1.29a05897572fdp+0, (-0x1.b4b1e1396fa60p-13), 0x1.5eeaab74b0bd7p-26, 0x1.1acebcf72db48p+41},\
   {0x1.69fe630cc6790p+22, 0x1.e1b415c971e27p+11, (-0x1.f830494f6138ep+0), 0x1.1d5ca031a53e9p-11, (-0x1.e3b66c62314f8p-25), 0x1.69fae99ebd1aap+27, 0x1.e1af7639f85a8p+15, (-0x1.501cf7007e109p+4), 0x1.1d59e30d0fa49p-8, (-0x1.82f49fe8c734fp-22), (-0x1.5123747d72c09p+36)},\
   {0x1.383eb7ca8f9e3p+23, 0x1.4f24ac9f858fbp+11, 0x1.3ca61bd3dea24p-1, (-0x1.c2d5666ade5a7p-12), 0x1.ed105d8b5cab2p-25, 0x1.4be775538ca1dp+27, 0x1.643e7cb67d8dcp+14, 0x1.c0c7c61421cf8p+1, (-0x1.df37e693eaa6fp-10), 0x1.a349399963805p-23, 0x1.2acb74dfcaccdp+38},\
   {0x1.1e7ac2e3eb2b5p+23, 0x1.39f7f9e39dfb2p+13, (-0x1.83b428cf6d1aap-1), (-0x1.d5a0b6e0c088ap-12), 0x1.4d69be610f4bap-24, 0x1.42906b9f5e9c1p+27, 0x1.618408b867c3ap+16, (-0x1.23068f00b550cp+2), (-0x1.086408eea1af8p-9), 0x1.2c53d604820a8p-22, (-0x1.226c28fd1c9aep+41)},\
   {0x1.cfe50765d5f3fp+22, 0x1.60a2d88e7926dp+12, (-0x1.98a0e352280dap+0), 0x1.2dc519b6f1b6fp-12, (-0x1.d2fde84bdced8p-26), 0x1.de7d4fc00d068p+27, 0x1.6bbb08cadcb91p+16, (-0x1.18fd5d80accffp+4), 0x1.37439ab3dda05p-9, (-0x1.8158e87f20091p-23), 0x1.152bf1da0734dp+33},\
   {0x1.d8328e3a08eebp+22, 0x1.76ee81a4eb6b3p+13, (-0x1.29747758d3647p+2), 0x1.dbb2980f7ec1ap-11, (-0x1.2e431299c67ecp-24), 0x1.f5ed65ced5474p+27, 0x1.8e89a02e0194ap+17, (-0x1.a593c329d7eecp+5), 0x1.f9a5d9eb3b548p-8, (-0x1.0108b9f4bd6f4p-21), (-0x1.59c80eb64f452p+40)},\
   {0x1.5d055c59fd85cp+22, 0x1.14062c7d74511p+12, (-0x1.aff084fd00f68p+0), 0x1.3a3e0c993c2fbp-12, (-0x1.585b9e0d0a636p-26), 0x1.318a1a6ed9168p+27, 0x1.e345fad6614b2p+15, (-0x1.f82bac86184e0p+3), 0x1.1317fa46cc62bp-9, (-0x1.e254ecbc085e2p-24), (-0x1.1dd3b7ba6451fp+36)}}
__constant__ double arr_dev[20][3] = {CHEM_GEN_ARR};
__constant__ double nasa_dev[2][9][11] = {CHEM_GEN_NASA};
#ifdef __CUDA_ARCH__
#define CHEM_GEN_TAB(x) x##_dev
#else
static const double arr_host[20][3] = {CHEM_GEN_ARR};
static const double nasa_host[2][9][11] = {CHEM_GEN_NASA};
#define CHEM_GEN_TAB(x) x##_host
#endif

HD __forceinline__ void tpart(double T, FunT& t) {
  const double Tinv = c_rcp(T);
  const double alogt = c_log(T);
  t.T = T;
  const int hi0 = T > 0x1.f400000000000p+9 ? 1 : 0;
  {   // species 0
    const double* c = CHEM_GEN_TAB(nasa)[hi0][0];
    t.cvk[0] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[0] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 1
    const double* c = CHEM_GEN_TAB(nasa)[hi0][1];
    t.cvk[1] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[1] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 2
    const double* c = CHEM_GEN_TAB(nasa)[hi0][2];
    t.cvk[2] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[2] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 3
    const double* c = CHEM_GEN_TAB(nasa)[hi0][3];
    t.cvk[3] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[3] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 4
    const double* c = CHEM_GEN_TAB(nasa)[hi0][4];
    t.cvk[4] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[4] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 5
    const double* c = CHEM_GEN_TAB(nasa)[hi0][5];
    t.cvk[5] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[5] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 6
    const double* c = CHEM_GEN_TAB(nasa)[hi0][6];
    t.cvk[6] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[6] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 7
    const double* c = CHEM_GEN_TAB(nasa)[hi0][7];
    t.cvk[7] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[7] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
  {   // species 8
    const double* c = CHEM_GEN_TAB(nasa)[hi0][8];
    t.cvk[8] = c[0] + T * (c[1] + T * (c[2] + T * (c[3] + T * c[4])));
    t.u[8] = c[10] + T * (c[5] + T * (c[6] + T * (c[7] + T * (c[8] + T * c[9]))));
  }
#pragma unroll 2
  for (int i = 0; i < 20; ++i) {
    const double* p = CHEM_GEN_TAB(arr)[i];
    t.k[i] = p[0] * fm_exp(p[1] * alogt - p[2] * Tinv);
  }
  t.k[18] = c_div(t.k[18], t.k[3]);
  {
    const double ta = 0x1.0000000000000p-1;
    double fcent = (1.0 - ta) * c_exp(-T * 0x1.93e5939a08ce9p+99) + ta * c_exp(-T * 0x1.4484bfeebc29fp-100);
    const double lnfc = c_log(fmax(fcent, 1.0e-300));
    t.lnfc[0] = lnfc;
    t.trc[0] = kTroeC + 0.67 * lnfc;
    t.trn[0] = kTroeN - 1.27 * lnfc;
  }
  t.k[19] = c_div(t.k[19], t.k[11]);
  {
    const double ta = 0x1.7851eb851eb85p-1;
    double fcent = (1.0 - ta) * c_exp(-T * 0x1.5c9882b931057p-7) + ta * c_exp(-T * 0x1.2a91c92f3c105p-11);
    fcent = fcent + c_exp(-0x1.43e0000000000p+12 * Tinv);
    const double lnfc = c_log(fmax(fcent, 1.0e-300));
    t.lnfc[1] = lnfc;
    t.trc[1] = kTroeC + 0.67 * lnfc;
    t.trn[1] = kTroeN - 1.27 * lnfc;
  }
}

HD __forceinline__ void cpart(const Cell<9>& cell, const double* z, const FunT& t, double* zp) {
  const double* Y = z + 1;
  double cv = 0.0, ctot = 0.0;
  cv = cv + Y[0] * t.cvk[0];
  const double C0 = Y[0] * cell.rw[0];
  ctot = ctot + C0;
  cv = cv + Y[1] * t.cvk[1];
  const double C1 = Y[1] * cell.rw[1];
  ctot = ctot + C1;
  cv = cv + Y[2] * t.cvk[2];
  const double C2 = Y[2] * cell.rw[2];
  ctot = ctot + C2;
  cv = cv + Y[3] * t.cvk[3];
  const double C3 = Y[3] * cell.rw[3];
  ctot = ctot + C3;
  cv = cv + Y[4] * t.cvk[4];
  const double C4 = Y[4] * cell.rw[4];
  ctot = ctot + C4;
  cv = cv + Y[5] * t.cvk[5];
  const double C5 = Y[5] * cell.rw[5];
  ctot = ctot + C5;
  cv = cv + Y[6] * t.cvk[6];
  const double C6 = Y[6] * cell.rw[6];
  ctot = ctot + C6;
  cv = cv + Y[7] * t.cvk[7];
  const double C7 = Y[7] * cell.rw[7];
  ctot = ctot + C7;
  cv = cv + Y[8] * t.cvk[8];
  const double C8 = Y[8] * cell.rw[8];
  ctot = ctot + C8;
  double rop0;
  {   // reaction 0
    double rkft = t.k[0];
    double rkrt = t.k[12];
    double rkf = rkft * C0;
    double rkr = rkrt * C2;
    rkf = rkf * C3;
    rkr = rkr * C4;
    rop0 = rkf - rkr;
  }
  double rop1;
  {   // reaction 1
    double rkft = t.k[1];
    double rkrt = t.k[13];
    double rkf = rkft * C1;
    double rkr = rkrt * C0;
    rkf = rkf * C2;
    rkr = rkr * C4;
    rop1 = rkf - rkr;
  }
  double rop2;
  {   // reaction 2
    double rkft = t.k[2];
    double rkrt = t.k[14];
    double rkf = rkft * C1;
    double rkr = rkrt * C0;
    rkf = rkf * C4;
    rkr = rkr * C5;
    rop2 = rkf - rkr;
  }
  double rop3;
  {   // reaction 3
    double rkft = t.k[3];
    double ctb = ctot;
    ctb = ctb + 0x1.8000000000000p+0 * C1;
    ctb = ctb + 0x1.e000000000000p+3 * C5;
    const double pr = t.k[18] * ctb;
    double pcor = c_div(pr, 1.0 + pr);
    pcor = troe_factor(pr, t.lnfc[0], t.trc[0], t.trn[0]) * pcor;
    rkft = rkft * pcor;
    double rkf = rkft * C0;
    rkf = rkf * C3;
    rop3 = rkf;
  }
  double rop4;
  {   // reaction 4
    double rkft = t.k[4];
    double rkf = rkft * C0;
    rkf = rkf * C6;
    rop4 = rkf;
  }
  double rop5;
  {   // reaction 5
    double rkft = t.k[5];
    double rkrt = t.k[15];
    double rkf = rkft * C0;
    double rkr = rkrt * C1;
    rkf = rkf * C6;
    rkr = rkr * C3;
    rop5 = rkf - rkr;
  }
  double rop6;
  {   // reaction 6
    double rkft = t.k[6];
    double rkf = rkft * C4;
    rkf = rkf * C6;
    rop6 = rkf;
  }
  double rop7;
  {   // reaction 7
    double rkft = t.k[7];
    double rkrt = t.k[16];
    double ctb = ctot;
    ctb = ctb + 0x1.8000000000000p+0 * C1;
    ctb = ctb + 0x1.6000000000000p+3 * C5;
    rkft = rkft * ctb;
    rkrt = rkrt * ctb;
    double rkf = rkft * C0;
    double rkr = rkrt * C5;
    rkf = rkf * C4;
    rop7 = rkf - rkr;
  }
  double rop8;
  {   // reaction 8
    double rkft = t.k[8];
    double rkrt = t.k[17];
    double ctb = ctot;
    ctb = ctb + 0x1.8000000000000p+0 * C1;
    ctb = ctb + 0x1.6000000000000p+3 * C5;
    rkft = rkft * ctb;
    rkrt = rkrt * ctb;
    double rkf = rkft * (C0 * C0);
    double rkr = rkrt * C1;
    rop8 = rkf - rkr;
  }
  double rop9;
  {   // reaction 9
    double rkft = t.k[9];
    double rkf = rkft * (C6 * C6);
    rop9 = rkf;
  }
  double rop10;
  {   // reaction 10
    double rkft = t.k[10];
    double rkf = rkft * C1;
    rkf = rkf * C6;
    rop10 = rkf;
  }
  double rop11;
  {   // reaction 11
    double rkft = t.k[11];
    double ctb = ctot;
    ctb = ctb + 0x1.8000000000000p+0 * C1;
    ctb = ctb + 0x1.4000000000000p+2 * C5;
    const double pr = t.k[19] * ctb;
    double pcor = c_div(pr, 1.0 + pr);
    pcor = troe_factor(pr, t.lnfc[1], t.trc[1], t.trn[1]) * pcor;
    rkft = rkft * pcor;
    double rkf = rkft * C7;
    rop11 = rkf;
  }
  const double wdot0 = - rop0 - rop3 - rop4 - rop5 - rop7 - rop8 * 0x1.0000000000000p+1 + rop1 + rop2 + rop10;
  const double wdot1 = - rop1 - rop2 - rop10 + rop5 + rop8;
  const double wdot2 = - rop1 + rop0;
  const double wdot3 = - rop0 - rop3 + rop6 + rop9 + rop5;
  const double wdot4 = - rop6 - rop2 - rop7 + rop4 * 0x1.0000000000000p+1 + rop11 * 0x1.0000000000000p+1 + rop0 + rop1;
  const double wdot5 = + rop7 + rop2 + rop6;
  const double wdot6 = - rop9 * 0x1.0000000000000p+1 - rop4 - rop5 - rop6 - rop10 + rop3;
  const double wdot7 = - rop11 + rop9 + rop10;
  const double wdot8 = 0.0;
  double sum = 0.0;
  zp[1] = wdot0 * 0x1.020a520000000p+0 * cell.rho_i;
  sum = sum + t.u[0] * wdot0;
  zp[2] = wdot1 * 0x1.020a520000000p+1 * cell.rho_i;
  sum = sum + t.u[1] * wdot1;
  zp[3] = wdot2 * 0x1.fffb160000000p+3 * cell.rho_i;
  sum = sum + t.u[2] * wdot2;
  zp[4] = wdot3 * 0x1.fffb160000000p+4 * cell.rho_i;
  sum = sum + t.u[3] * wdot3;
  zp[5] = wdot4 * 0x1.101e302000000p+4 * cell.rho_i;
  sum = sum + t.u[4] * wdot4;
  zp[6] = wdot5 * 0x1.203ed54000000p+4 * cell.rho_i;
  sum = sum + t.u[5] * wdot5;
  zp[7] = wdot6 * 0x1.080ddd9000000p+5 * cell.rho_i;
  sum = sum + t.u[6] * wdot6;
  zp[8] = wdot7 * 0x1.101e302000000p+5 * cell.rho_i;
  sum = sum + t.u[7] * wdot7;
  zp[9] = 0.0;
  zp[0] = -c_div(sum, cell.rho * cv);
}

// the same from the density alone
HD __forceinline__ void cpart(double rho, const double* z, const FunT& t, double* zp) {
  Cell<9> cell;
  cell_set(rho, cell);
  cpart(cell, z, t, zp);
}

// True when m is the mechanism this file was generated from (every table
// entry the right-hand side reads, bit for bit).
inline bool matches(const izem_mech& m) {
  auto b = [](double x) { unsigned long long u; memcpy(&u, &x, sizeof(u)); return u; };
  if (m.kk != 9 || m.ii != 12 || b(m.ru) != 0x4193d2c630000000ULL) return false;
  if (!(b(m.wt[0]) == 0x3ff020a520000000ULL && b(m.tmid[0]) == 0x408f400000000000ULL && b(m.a[0][0][0]) == 0x4004000000000000ULL && b(m.a[0][0][1]) == 0x3d68d112bff6d580ULL)) return false;
  if (!(b(m.a[0][0][2]) == 0xbce1fa470055807fULL && b(m.a[0][0][3]) == 0x3c4538a620b2373fULL && b(m.a[0][0][4]) == 0xbb91863cffe0b329ULL && b(m.a[0][0][5]) == 0x40d8e06a3bcd35a8ULL)) return false;
  if (!(b(m.a[0][0][6]) == 0xbfdc9673ad546a18ULL && b(m.a[0][1][0]) == 0x40040000015798eeULL && b(m.a[0][1][1]) == 0xbdb961a6ec6a1e45ULL && b(m.a[0][1][2]) == 0x3d1230b4c341c642ULL)) return false;
  if (!(b(m.a[0][1][3]) == 0xbc55d647fbe2e672ULL && b(m.a[0][1][4]) == 0x3b82d244e9510ba2ULL && b(m.a[0][1][5]) == 0x40d8e06a3bcd35a8ULL && b(m.a[0][1][6]) == 0xbfdc9673eed3f77dULL)) return false;
  if (!(b(m.wt[1]) == 0x400020a520000000ULL && b(m.tmid[1]) == 0x408f400000000000ULL && b(m.a[1][0][0]) == 0x4002c130ac9b2911ULL && b(m.a[1][0][1]) == 0x3f8058175d02a941ULL)) return false;
  if (!(b(m.a[1][0][2]) == 0xbef46ca05831775cULL && b(m.a[1][0][3]) == 0x3e55a4c582f87e3dULL && b(m.a[1][0][4]) == 0xbda03862939e564dULL && b(m.a[1][0][5]) == 0xc08caf7b3bfb58d1ULL)) return false;
  if (!(b(m.a[1][0][6]) == 0x3fe5db38496161b4ULL && b(m.a[1][1][0]) == 0x400ab2bf6fecf7e5ULL && b(m.a[1][1][1]) == 0xbf09e6b00cea2ba4ULL && b(m.a[1][1][2]) == 0x3ea0c24d11e93b22ULL)) return false;
  if (!(b(m.a[1][1][3]) == 0xbde8adee4a4b6baeULL && b(m.a[1][1][4]) == 0x3d168bf7de4136dcULL && b(m.a[1][1][5]) == 0xc08db14578e5c4ebULL && b(m.a[1][1][6]) == 0xc009a3e342daf0fdULL)) return false;
  if (!(b(m.wt[2]) == 0x402fffb160000000ULL && b(m.tmid[2]) == 0x408f400000000000ULL && b(m.a[2][0][0]) == 0x4009589c6bdbf12dULL && b(m.a[2][0][1]) == 0xbf6add3ae5787a18ULL)) return false;
  if (!(b(m.a[2][0][2]) == 0x3edbdcef845b6ae0ULL && b(m.a[2][0][3]) == 0xbe3a51e14d5c0503ULL && b(m.a[2][0][4]) == 0x3d82954967e1b470ULL && b(m.a[2][0][5]) == 0x40dc709096bb98c8ULL)) return false;
  if (!(b(m.a[2][0][6]) == 0x40006a5c1702251eULL && b(m.a[2][1][0]) == 0x40048e2c7b5e1a3dULL && b(m.a[2][1][1]) == 0xbf1689a006cdb509ULL && b(m.a[2][1][2]) == 0x3e66855a2fbdda5cULL)) return false;
  if (!(b(m.a[2][1][3]) == 0xbda607823c010ceaULL && b(m.a[2][1][4]) == 0x3cd620b4436bd152ULL && b(m.a[2][1][5]) == 0x40dc88650ff97247ULL && b(m.a[2][1][6]) == 0x40132329ab1f280eULL)) return false;
  if (!(b(m.wt[3]) == 0x403fffb160000000ULL && b(m.tmid[3]) == 0x408f400000000000ULL && b(m.a[3][0][0]) == 0x400e42787ae5fa45ULL && b(m.a[3][0][1]) == 0xbf688c9b66c8c0dfULL)) return false;
  if (!(b(m.a[3][0][2]) == 0x3ee4a6bae1fdae75ULL && b(m.a[3][0][3]) == 0xbe44ca5927ada53cULL && b(m.a[3][0][4]) == 0x3d8c883a18b02bcdULL && b(m.a[3][0][5]) == 0xc0909fc63497b741ULL)) return false;
  if (!(b(m.a[3][0][6]) == 0x400d42eb7e3dc88dULL && b(m.a[3][1][0]) == 0x400a42a332f575b8ULL && b(m.a[3][1][1]) == 0x3f584c851ecf574dULL && b(m.a[3][1][2]) == 0xbea96ee255022a3dULL)) return false;
  if (!(b(m.a[3][1][3]) == 0x3decca1706e20348ULL && b(m.a[3][1][4]) == 0xbd18667712a69c18ULL && b(m.a[3][1][5]) == 0xc09101d4b48d3ae7ULL && b(m.a[3][1][6]) == 0x4015d01bdd004baaULL)) return false;
  if (!(b(m.wt[4]) == 0x403101e302000000ULL && b(m.tmid[4]) == 0x408f400000000000ULL && b(m.a[4][0][0]) == 0x400fefa5c927d1abULL && b(m.a[4][0][1]) == 0xbf63abed86e71c7dULL)) return false;
  if (!(b(m.a[4][0][2]) == 0x3ed35e793e99fbcdULL && b(m.a[4][0][3]) == 0xbe30ab59e9e67441ULL && b(m.a[4][0][4]) == 0x3d77ff6d2c211dd3ULL && b(m.a[4][0][5]) == 0x40ac3e293f290abbULL)) return false;
  if (!(b(m.a[4][0][6]) == 0xbfba9adbdb54f242ULL && b(m.a[4][1][0]) == 0x4008be3be406d029ULL && b(m.a[4][1][1]) == 0x3f41f88fd8e1440eULL && b(m.a[4][1][2]) == 0x3e80faafc0d73234ULL)) return false;
  if (!(b(m.a[4][1][3]) == 0xbdd82ca91827ab6dULL && b(m.a[4][1][4]) == 0x3d0a705cd746f5f8ULL && b(m.a[4][1][5]) == 0x40ae2550624dd2f2ULL && b(m.a[4][1][6]) == 0x4011e82305be85e2ULL)) return false;
  if (!(b(m.wt[5]) == 0x403203ed54000000ULL && b(m.tmid[5]) == 0x408f400000000000ULL && b(m.a[5][0][0]) == 0x4010cb686e536fbfULL && b(m.a[5][0][1]) == 0xbf60aeb63b84c925ULL)) return false;
  if (!(b(m.a[5][0][2]) == 0x3edb593a7c039b70ULL && b(m.a[5][0][3]) == 0xbe37921667072d59ULL && b(m.a[5][0][4]) == 0x3d7f2c47bce627b1ULL && b(m.a[5][0][5]) == 0xc0dd956e8240b780ULL)) return false;
  if (!(b(m.a[5][0][6]) == 0xbfeb2b4597d38a9bULL && b(m.a[5][1][0]) == 0x4008459ddac6e07aULL && b(m.a[5][1][1]) == 0x3f61d553f9364039ULL && b(m.a[5][1][2]) == 0xbe86057d217698d4ULL)) return false;
  if (!(b(m.a[5][1][3]) == 0xbddaacb906a5f7ccULL && b(m.a[5][1][4]) == 0x3d12f01042cd6ffeULL && b(m.a[5][1][5]) == 0xc0dd4d1303afb7e9ULL && b(m.a[5][1][6]) == 0x4013ddf8fb2900aaULL)) return false;
  if (!(b(m.wt[6]) == 0x404080ddd9000000ULL && b(m.tmid[6]) == 0x408f400000000000ULL && b(m.a[6][0][0]) == 0x4011350a899bcaa1ULL && b(m.a[6][0][1]) == 0xbf7373d054674594ULL)) return false;
  if (!(b(m.a[6][0][2]) == 0x3ef62fa28e3a8ea6ULL && b(m.a[6][0][3]) == 0xbe5a110b0905e0fcULL && b(m.a[6][0][4]) == 0x3da46f1288fc5c1cULL && b(m.a[6][0][5]) == 0x40726cedbb59ddc2ULL)) return false;
  if (!(b(m.a[6][0][6]) == 0x400dbbb985c82b7dULL && b(m.a[6][1][0]) == 0x4010119fbbf289f6ULL && b(m.a[6][1][1]) == 0x3f62593e46a1f9dfULL && b(m.a[6][1][2]) == 0xbea5431502070c84ULL)) return false;
  if (!(b(m.a[6][1][3]) == 0x3ddf675fa32f618cULL && b(m.a[6][1][4]) == 0xbd084c80e71ea191ULL && b(m.a[6][1][5]) == 0x405bf6d462c343b7ULL && b(m.a[6][1][6]) == 0x400e47e3a2d22780ULL)) return false;
  if (!(b(m.wt[7]) == 0x404101e302000000ULL && b(m.tmid[7]) == 0x408f400000000000ULL && b(m.a[7][0][0]) == 0x40111abd48f63e0aULL && b(m.a[7][0][1]) == 0xbf41c98643a78c6aULL)) return false;
  if (!(b(m.a[7][0][2]) == 0x3ef18be22e62f026ULL && b(m.a[7][0][3]) == 0xbe572b101d35ae59ULL && b(m.a[7][0][4]) == 0x3da2f72fba30b7c2ULL && b(m.a[7][0][5]) == 0xc0d149a541205bc0ULL)) return false;
  if (!(b(m.a[7][0][6]) == 0x400b7afbe1e3346dULL && b(m.a[7][1][0]) == 0x4010a8f681d1fcb7ULL && b(m.a[7][1][1]) == 0x3f741abe4bc5704bULL && b(m.a[7][1][2]) == 0xbebfe66ae3495cc5ULL)) return false;
  if (!(b(m.a[7][1][3]) == 0x3df981f91177d524ULL && b(m.a[7][1][4]) == 0xbd20353229ef325dULL && b(m.a[7][1][5]) == 0xc0d1717269ad42c4ULL && b(m.a[7][1][6]) == 0x40075449ec074fabULL)) return false;
  if (!(b(m.wt[8]) == 0x403c036e20000000ULL && b(m.tmid[8]) == 0x408f400000000000ULL && b(m.a[8][0][0]) == 0x400a63b0c4588a05ULL && b(m.a[8][0][1]) == 0x3f5712969da04050ULL)) return false;
  if (!(b(m.a[8][0][2]) == 0xbed09f7a2b098bd4ULL && b(m.a[8][0][3]) == 0x3e383ae94da0fe59ULL && b(m.a[8][0][4]) == 0xbd8581526048e0d6ULL && b(m.a[8][0][5]) == 0xc08fe732fec56d5dULL)) return false;
  if (!(b(m.a[8][0][6]) == 0x400f9a5ca29845ddULL && b(m.a[8][1][0]) == 0x400769c23b7952d2ULL && b(m.a[8][1][1]) == 0x3f586106ec5d7fc6ULL && b(m.a[8][1][2]) == 0xbea3132bf1b89c39ULL)) return false;
  if (!(b(m.a[8][1][3]) == 0x3ddbc128a9b8a724ULL && b(m.a[8][1][4]) == 0xbcfe6a15668d1fd9ULL && b(m.a[8][1][5]) == 0xc08cd661b089a027ULL && b(m.a[8][1][6]) == 0x4017ec0f88333fc8ULL)) return false;
  if (!(m.nuk[0][0] == 0 && m.nu[0][0] == -1 && m.nuk[0][1] == 3 && m.nu[0][1] == -1 && m.nuk[0][2] == -1 && m.nu[0][2] == 0 && m.nuk[0][3] == 2 && m.nu[0][3] == 1)) return false;
  if (!(m.nuk[0][4] == 4 && m.nu[0][4] == 1 && m.nuk[0][5] == -1 && m.nu[0][5] == 0 && b(m.par[0][0]) == 0x435f438daa060000ULL && b(m.par[0][1]) == 0xbfe6666666666666ULL)) return false;
  if (!(b(m.par[0][2]) == 0x40c0c6f4493ef159ULL && m.rev[0] == 2 && m.thb[0] == 0 && m.fall[0] == 0 && b(m.lt[0][0]) == 0x0000000000000000ULL && b(m.rlt[0][0]) == 0x0000000000000000ULL && b(m.lt[0][1]) == 0x0000000000000000ULL && b(m.rlt[0][1]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.rpar[0][0]) == 0x42d001d1bf800000ULL && b(m.rpar[0][1]) == 0xbfd0a3d70a3d70a4ULL && b(m.rpar[0][2]) == 0x4051fd705d6afec6ULL && m.nuk[1][0] == 1 && m.nu[1][0] == -1)) return false;
  if (!(m.nuk[1][1] == 2 && m.nu[1][1] == -1 && m.nuk[1][2] == -1 && m.nu[1][2] == 0 && m.nuk[1][3] == 0 && m.nu[1][3] == 1 && m.nuk[1][4] == 4 && m.nu[1][4] == 1)) return false;
  if (!(m.nuk[1][5] == -1 && m.nu[1][5] == 0 && b(m.par[1][0]) == 0x40e8b50000000000ULL && b(m.par[1][1]) == 0x40055c28f5c28f5cULL && b(m.par[1][2]) == 0x40a8bb78dad5b973ULL)) return false;
  if (!(m.rev[1] == 2 && m.thb[1] == 0 && m.fall[1] == 0 && b(m.lt[1][0]) == 0x0000000000000000ULL && b(m.rlt[1][0]) == 0x0000000000000000ULL && b(m.lt[1][1]) == 0x0000000000000000ULL && b(m.rlt[1][1]) == 0x0000000000000000ULL && b(m.rpar[1][0]) == 0x40dd970000000000ULL)) return false;
  if (!(b(m.rpar[1][1]) == 0x40050a3d70a3d70aULL && b(m.rpar[1][2]) == 0x40a3072327bb03a1ULL && m.nuk[2][0] == 1 && m.nu[2][0] == -1 && m.nuk[2][1] == 4 && m.nu[2][1] == -1)) return false;
  if (!(m.nuk[2][2] == -1 && m.nu[2][2] == 0 && m.nuk[2][3] == 0 && m.nu[2][3] == 1 && m.nuk[2][4] == 5 && m.nu[2][4] == 1 && m.nuk[2][5] == -1 && m.nu[2][5] == 0)) return false;
  if (!(b(m.par[2][0]) == 0x41d16f3220000000ULL && b(m.par[2][1]) == 0x3ff4cccccccccccdULL && b(m.par[2][2]) == 0x409c94c533be761cULL && m.rev[2] == 2 && m.thb[2] == 0 && m.fall[2] == 0)) return false;
  if (!(b(m.lt[2][0]) == 0x0000000000000000ULL && b(m.rlt[2][0]) == 0x0000000000000000ULL && b(m.lt[2][1]) == 0x0000000000000000ULL && b(m.rlt[2][1]) == 0x0000000000000000ULL && b(m.rpar[2][0]) == 0x4207d78400000000ULL && b(m.rpar[2][1]) == 0x3ff30a3d70a3d70aULL)) return false;
  if (!(b(m.rpar[2][2]) == 0x40c2611369490098ULL && m.nuk[3][0] == 0 && m.nu[3][0] == -1 && m.nuk[3][1] == 3 && m.nu[3][1] == -1 && m.nuk[3][2] == -1 && m.nu[3][2] == 0)) return false;
  if (!(m.nuk[3][3] == 6 && m.nu[3][3] == 1 && m.nuk[3][4] == -1 && m.nu[3][4] == 0 && m.nuk[3][5] == -1 && m.nu[3][5] == 0 && b(m.par[3][0]) == 0x4290eaa664900000ULL)) return false;
  if (!(b(m.par[3][1]) == 0x3fdc28f5c28f5c29ULL && b(m.par[3][2]) == 0x0000000000000000ULL && m.rev[3] == 0 && m.thb[3] == 1 && m.fall[3] == 3 && b(m.lt[3][0]) == 0x0000000000000000ULL && b(m.rlt[3][0]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.lt[3][1]) == 0x0000000000000000ULL && b(m.rlt[3][1]) == 0x0000000000000000ULL && b(m.eff[3][0]) == 0x3ff0000000000000ULL && b(m.eff[3][1]) == 0x4004000000000000ULL && b(m.eff[3][2]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[3][3]) == 0x3ff0000000000000ULL && b(m.eff[3][4]) == 0x3ff0000000000000ULL && b(m.eff[3][5]) == 0x4030000000000000ULL && b(m.eff[3][6]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[3][7]) == 0x3ff0000000000000ULL && b(m.eff[3][8]) == 0x3ff0000000000000ULL && m.kfal[3] == 0 && b(m.low[3][0]) == 0x4408efc84ad0c7b0ULL)) return false;
  if (!(b(m.low[3][1]) == 0xbff6666666666666ULL && b(m.low[3][2]) == 0x0000000000000000ULL && b(m.troe[3][0]) == 0x3fe0000000000000ULL && b(m.troe[3][1]) == 0x39b4484bfeebc2a0ULL)) return false;
  if (!(b(m.troe[3][2]) == 0x46293e5939a08ceaULL && m.nuk[4][0] == 0 && m.nu[4][0] == -1 && m.nuk[4][1] == 6 && m.nu[4][1] == -1 && m.nuk[4][2] == -1 && m.nu[4][2] == 0)) return false;
  if (!(m.nuk[4][3] == 4 && m.nu[4][3] == 2 && m.nuk[4][4] == -1 && m.nu[4][4] == 0 && m.nuk[4][5] == -1 && m.nu[4][5] == 0 && b(m.par[4][0]) == 0x42d0191a36680000ULL)) return false;
  if (!(b(m.par[4][1]) == 0x0000000000000000ULL && b(m.par[4][2]) == 0x40627e432c1d6dbcULL && m.rev[4] == 0 && m.thb[4] == 0 && m.fall[4] == 0 && b(m.lt[4][0]) == 0x0000000000000000ULL && b(m.rlt[4][0]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.lt[4][1]) == 0x0000000000000000ULL && b(m.rlt[4][1]) == 0x0000000000000000ULL && m.nuk[5][0] == 0 && m.nu[5][0] == -1 && m.nuk[5][1] == 6 && m.nu[5][1] == -1 && m.nuk[5][2] == -1 && m.nu[5][2] == 0)) return false;
  if (!(m.nuk[5][3] == 1 && m.nu[5][3] == 1 && m.nuk[5][4] == 3 && m.nu[5][4] == 1 && m.nuk[5][5] == -1 && m.nu[5][5] == 0 && b(m.par[5][0]) == 0x42ae31fa34e00000ULL)) return false;
  if (!(b(m.par[5][1]) == 0x0000000000000000ULL && b(m.par[5][2]) == 0x4079da4e3b0f0481ULL && m.rev[5] == 2 && m.thb[5] == 0 && m.fall[5] == 0 && b(m.lt[5][0]) == 0x0000000000000000ULL && b(m.rlt[5][0]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.lt[5][1]) == 0x0000000000000000ULL && b(m.rlt[5][1]) == 0x0000000000000000ULL && b(m.rpar[5][0]) == 0x42839283f4a00000ULL && b(m.rpar[5][1]) == 0x3fd70a3d70a3d70aULL && b(m.rpar[5][2]) == 0x40db3c1120ab0336ULL)) return false;
  if (!(m.nuk[6][0] == 4 && m.nu[6][0] == -1 && m.nuk[6][1] == 6 && m.nu[6][1] == -1 && m.nuk[6][2] == -1 && m.nu[6][2] == 0 && m.nuk[6][3] == 3 && m.nu[6][3] == 1)) return false;
  if (!(m.nuk[6][4] == 5 && m.nu[6][4] == 1 && m.nuk[6][5] == -1 && m.nu[6][5] == 0 && b(m.par[6][0]) == 0x42ba48ce3be80000ULL && b(m.par[6][1]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.par[6][2]) == 0xc06f4328690d2d50ULL && m.rev[6] == 0 && m.thb[6] == 0 && m.fall[6] == 0 && b(m.lt[6][0]) == 0x0000000000000000ULL && b(m.rlt[6][0]) == 0x0000000000000000ULL && b(m.lt[6][1]) == 0x0000000000000000ULL && b(m.rlt[6][1]) == 0x0000000000000000ULL)) return false;
  if (!(m.nuk[7][0] == 0 && m.nu[7][0] == -1 && m.nuk[7][1] == 4 && m.nu[7][1] == -1 && m.nuk[7][2] == -1 && m.nu[7][2] == 0 && m.nuk[7][3] == 5 && m.nu[7][3] == 1)) return false;
  if (!(m.nuk[7][4] == -1 && m.nu[7][4] == 0 && m.nuk[7][5] == -1 && m.nu[7][5] == 0 && b(m.par[7][0]) == 0x44a0f0cf064dd592ULL && b(m.par[7][1]) == 0xc000000000000000ULL)) return false;
  if (!(b(m.par[7][2]) == 0x0000000000000000ULL && m.rev[7] == 2 && m.thb[7] == 1 && m.fall[7] == 0 && b(m.lt[7][0]) == 0x0000000000000000ULL && b(m.rlt[7][0]) == 0x0000000000000000ULL && b(m.lt[7][1]) == 0x0000000000000000ULL && b(m.rlt[7][1]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.rpar[7][0]) == 0x44b5cfa424ea9c92ULL && b(m.rpar[7][1]) == 0xbffc000000000000ULL && b(m.rpar[7][2]) == 0x40ed22edd4d65d8eULL && b(m.eff[7][0]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[7][1]) == 0x4004000000000000ULL && b(m.eff[7][2]) == 0x3ff0000000000000ULL && b(m.eff[7][3]) == 0x3ff0000000000000ULL && b(m.eff[7][4]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[7][5]) == 0x4028000000000000ULL && b(m.eff[7][6]) == 0x3ff0000000000000ULL && b(m.eff[7][7]) == 0x3ff0000000000000ULL && b(m.eff[7][8]) == 0x3ff0000000000000ULL)) return false;
  if (!(m.nuk[8][0] == 0 && m.nu[8][0] == -2 && m.nuk[8][1] == -1 && m.nu[8][1] == 0 && m.nuk[8][2] == -1 && m.nu[8][2] == 0 && m.nuk[8][3] == 1 && m.nu[8][3] == 1)) return false;
  if (!(m.nuk[8][4] == -1 && m.nu[8][4] == 0 && m.nuk[8][5] == -1 && m.nu[8][5] == 0 && b(m.par[8][0]) == 0x43b20a871cc00200ULL && b(m.par[8][1]) == 0xbff0000000000000ULL)) return false;
  if (!(b(m.par[8][2]) == 0x0000000000000000ULL && m.rev[8] == 2 && m.thb[8] == 1 && m.fall[8] == 0 && b(m.lt[8][0]) == 0x0000000000000000ULL && b(m.rlt[8][0]) == 0x0000000000000000ULL && b(m.lt[8][1]) == 0x0000000000000000ULL && b(m.rlt[8][1]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.rpar[8][0]) == 0x4390e0198eaee000ULL && b(m.rpar[8][1]) == 0xbfe4cccccccccccdULL && b(m.rpar[8][2]) == 0x40e96e5d98de8289ULL && b(m.eff[8][0]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[8][1]) == 0x4004000000000000ULL && b(m.eff[8][2]) == 0x3ff0000000000000ULL && b(m.eff[8][3]) == 0x3ff0000000000000ULL && b(m.eff[8][4]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[8][5]) == 0x4028000000000000ULL && b(m.eff[8][6]) == 0x3ff0000000000000ULL && b(m.eff[8][7]) == 0x3ff0000000000000ULL && b(m.eff[8][8]) == 0x3ff0000000000000ULL)) return false;
  if (!(m.nuk[9][0] == 6 && m.nu[9][0] == -2 && m.nuk[9][1] == -1 && m.nu[9][1] == 0 && m.nuk[9][2] == -1 && m.nu[9][2] == 0 && m.nuk[9][3] == 3 && m.nu[9][3] == 1)) return false;
  if (!(m.nuk[9][4] == 7 && m.nu[9][4] == 1 && m.nuk[9][5] == -1 && m.nu[9][5] == 0 && b(m.par[9][0]) == 0x4285f93037c00000ULL && b(m.par[9][1]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.par[9][2]) == 0x4085dbc4f266b3c5ULL && m.rev[9] == 0 && m.thb[9] == 0 && m.fall[9] == 0 && b(m.lt[9][0]) == 0x0000000000000000ULL && b(m.rlt[9][0]) == 0x0000000000000000ULL && b(m.lt[9][1]) == 0x0000000000000000ULL && b(m.rlt[9][1]) == 0x0000000000000000ULL)) return false;
  if (!(m.nuk[10][0] == 1 && m.nu[10][0] == -1 && m.nuk[10][1] == 6 && m.nu[10][1] == -1 && m.nuk[10][2] == -1 && m.nu[10][2] == 0 && m.nuk[10][3] == 0 && m.nu[10][3] == 1)) return false;
  if (!(m.nuk[10][4] == 7 && m.nu[10][4] == 1 && m.nuk[10][5] == -1 && m.nu[10][5] == 0 && b(m.par[10][0]) == 0x4242dbf9ea000000ULL && b(m.par[10][1]) == 0x3fe3851eb851eb85ULL)) return false;
  if (!(b(m.par[10][2]) == 0x40c784fcc6a9ac05ULL && m.rev[10] == 0 && m.thb[10] == 0 && m.fall[10] == 0 && b(m.lt[10][0]) == 0x0000000000000000ULL && b(m.rlt[10][0]) == 0x0000000000000000ULL && b(m.lt[10][1]) == 0x0000000000000000ULL && b(m.rlt[10][1]) == 0x0000000000000000ULL)) return false;
  if (!(m.nuk[11][0] == 7 && m.nu[11][0] == -1 && m.nuk[11][1] == -1 && m.nu[11][1] == 0 && m.nuk[11][2] == -1 && m.nu[11][2] == 0 && m.nuk[11][3] == 4 && m.nu[11][3] == 2)) return false;
  if (!(m.nuk[11][4] == -1 && m.nu[11][4] == 0 && m.nuk[11][5] == -1 && m.nu[11][5] == 0 && b(m.par[11][0]) == 0x43f6b99192fbb3c0ULL && b(m.par[11][1]) == 0xbff63d70a3d70a3dULL)) return false;
  if (!(b(m.par[11][2]) == 0x40d93845131294f1ULL && m.rev[11] == 0 && m.thb[11] == 1 && m.fall[11] == 4 && b(m.lt[11][0]) == 0x0000000000000000ULL && b(m.rlt[11][0]) == 0x0000000000000000ULL && b(m.lt[11][1]) == 0x0000000000000000ULL && b(m.rlt[11][1]) == 0x0000000000000000ULL)) return false;
  if (!(b(m.eff[11][0]) == 0x3ff0000000000000ULL && b(m.eff[11][1]) == 0x4004000000000000ULL && b(m.eff[11][2]) == 0x3ff0000000000000ULL && b(m.eff[11][3]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[11][4]) == 0x3ff0000000000000ULL && b(m.eff[11][5]) == 0x4018000000000000ULL && b(m.eff[11][6]) == 0x3ff0000000000000ULL && b(m.eff[11][7]) == 0x3ff0000000000000ULL)) return false;
  if (!(b(m.eff[11][8]) == 0x3ff0000000000000ULL && m.kfal[11] == 0 && b(m.low[11][0]) == 0x44e592a7a2071df8ULL && b(m.low[11][1]) == 0xbffe666666666666ULL)) return false;
  if (!(b(m.low[11][2]) == 0x40d8626719ec5abbULL && b(m.troe[11][0]) == 0x3fe7851eb851eb85ULL && b(m.troe[11][1]) == 0x4057800000000000ULL && b(m.troe[11][2]) == 0x409b700000000000ULL)) return false;
  if (!(b(m.troe[11][3]) == 0x40b43e0000000000ULL)) return false;
  return true;
}

}  // namespace chem_gen
