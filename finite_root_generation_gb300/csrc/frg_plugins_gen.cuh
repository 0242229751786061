// GENERATED by finite_root_generation_gb300/gen/gen_plugins.py from the modules in
// finite_root_generation_gb300/systems -- do not edit.
//
// System plug-ins: the homogenized equations' rows of the homotopy Jacobian (columns
// Z, Z0, then the t column dF/dq . dq/dt) as straight-line code for one thread and as a
// schedule of independent operations for a warp (16 operations a step, one lane per
// real component), and the finite-root-generation start (random unknowns and free
// parameters, then the parameters that make the random point an exact root).
#pragma once

#include "frg_device.cuh"

namespace frg {

// ---- system 1: conic2 (2 unknowns, 12 parameters)
// rows(): 48 complex mul, 32 complex add/sub, 3 real x complex; as a warp's schedule
// 83 operations in 8 steps
static __device__ const uint32_t tape_conic2[128] = {
    0x8010001cu, 0x8000001du, 0x8010041eu, 0x8020081fu, 0x80600820u, 0x80000821u, 0x80c00822u, 0x80101023u, 
    0x80100824u, 0x80102825u, 0x80700826u, 0x80d00827u, 0x80001028u, 0x80001829u, 0x80101c2au, 0x8000282bu, 
    0x81d03c2cu, 0x81c0402du, 0x81d0542eu, 0x81c0582fu, 0x81d00c30u, 0x81e01431u, 0x81d02432u, 0x81e02c33u, 
    0x81e04434u, 0x81e05c35u, 0x81f02036u, 0x81f03837u, 0x82104838u, 0x82106039u, 0x8000803au, 0x8000883bu, 
    0x2d0b01cu, 0x2f0b81du, 0x310c01eu, 0x330c821u, 0x3cu, 0x10043du, 0x20083eu, 0x230803fu, 0x2809840u, 0x2a0a441u, 
    0x2508842u, 0x2b09c43u, 0x44u, 0x44u, 0x44u, 0x44u, 0x3407020u, 0x3507422u, 0x3607828u, 0x3708429u, 0x44u, 
    0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x82404c2au, 0x8000302bu, 
    0x8010342cu, 0x8240642du, 0x80008c2eu, 0x8000942fu, 0x83c00c30u, 0x83d01431u, 0x83e02032u, 0x81f05033u, 
    0x83c0241cu, 0x83d02c1du, 0x83e0381eu, 0x81f06821u, 0x80109834u, 0x80109c35u, 0x3808036u, 0x3908837u, 
    0x3a0a01fu, 0x3b0a423u, 0x2c0ac24u, 0x300fc25u, 0x3110026u, 0x3210427u, 0x1c1083cu, 0x1d10c3du, 0x44u, 0x44u, 
    0x44u, 0x44u, 0x44u, 0x44u, 0x2a0d83eu, 0x2d0dc1cu, 0x2e07c1du, 0x2f08c20u, 0x1e09022u, 0x44u, 0x44u, 0x44u, 
    0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x330f828u, 0x2107029u, 0x340742bu, 0x350802cu, 0x44u, 
    0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u, 0x44u};
static __device__ const uint16_t tape_out_conic2[10] = {
    37, 38, 39, 40, 60, 61, 34, 41, 43, 44};
static __device__ const double tape_const_conic2[1] = {
    0.0};
struct Sys_conic2 {
  static constexpr int ID = 1;
  static constexpr int NV = 2;
  static constexpr int NP = 12;
  static constexpr int NS = 2;
  static constexpr int ROWS_CMUL = 48, ROWS_CADD = 32, ROWS_SMUL = 3;
  static constexpr int TAPE_STEPS = 8, TAPE_REGS = 69, TAPE_CONSTS = 1;
  __device__ static const uint32_t* tape() { return tape_conic2; }
  __device__ static const uint16_t* tape_out() { return tape_out_conic2; }
  __device__ static const double* tape_const() { return tape_const_conic2; }
  template <typename T, int LD>
  __device__ static void rows(const cx<T>* Y, const cx<T>* q, const cx<T>* dq, cx<T>* M, cx<T>* F) {
    const cx<T> u_x = Y[0];
    const cx<T> u_y = Y[1];
    const cx<T> u_Z0 = Y[2];
    const cx<T> p_a1 = q[0];
    const cx<T> dp_a1 = dq[0];
    const cx<T> p_b1 = q[1];
    const cx<T> dp_b1 = dq[1];
    const cx<T> p_c1 = q[2];
    const cx<T> dp_c1 = dq[2];
    const cx<T> p_d1 = q[3];
    const cx<T> dp_d1 = dq[3];
    const cx<T> p_e1 = q[4];
    const cx<T> dp_e1 = dq[4];
    const cx<T> p_f1 = q[5];
    const cx<T> dp_f1 = dq[5];
    const cx<T> p_a2 = q[6];
    const cx<T> dp_a2 = dq[6];
    const cx<T> p_b2 = q[7];
    const cx<T> dp_b2 = dq[7];
    const cx<T> p_c2 = q[8];
    const cx<T> dp_c2 = dq[8];
    const cx<T> p_d2 = q[9];
    const cx<T> dp_d2 = dq[9];
    const cx<T> p_e2 = q[10];
    const cx<T> dp_e2 = dq[10];
    const cx<T> p_f2 = q[11];
    const cx<T> dp_f2 = dq[11];
    const cx<T> r_0 = (u_Z0 * p_d1);
    const cx<T> r_1 = (p_b1 * u_y);
    const cx<T> r_2 = (T(2.0) * (u_x));
    const cx<T> r_3 = (u_Z0 * p_e1);
    const cx<T> r_4 = (T(2.0) * (u_y));
    const cx<T> r_5 = (T(2.0) * (u_Z0));
    const cx<T> r_6 = (u_Z0 * u_x);
    const cx<T> r_7 = (u_Z0 * u_y);
    const cx<T> r_8 = (u_x * u_y);
    const cx<T> r_9 = (u_Z0 * u_Z0);
    const cx<T> r_10 = (u_x * u_x);
    const cx<T> r_11 = (u_y * u_y);
    const cx<T> r_12 = (u_Z0 * p_d2);
    const cx<T> r_13 = (p_b2 * u_y);
    const cx<T> r_14 = (u_Z0 * p_e2);
    M[0 * LD + 0] = (r_0 + r_1 + (p_a1 * r_2));
    M[0 * LD + 1] = (r_3 + (p_b1 * u_x) + (p_c1 * r_4));
    M[0 * LD + 2] = ((p_d1 * u_x) + (p_e1 * u_y) + (p_f1 * r_5));
    M[0 * LD + 3] = ((dp_a1 * r_10) + (dp_b1 * r_8) + (dp_c1 * r_11) + (dp_d1 * r_6) + (dp_e1 * r_7) + (dp_f1 * r_9));
    M[1 * LD + 0] = (r_12 + r_13 + (p_a2 * r_2));
    M[1 * LD + 1] = (r_14 + (p_b2 * u_x) + (p_c2 * r_4));
    M[1 * LD + 2] = ((p_d2 * u_x) + (p_e2 * u_y) + (p_f2 * r_5));
    M[1 * LD + 3] = ((dp_a2 * r_10) + (dp_b2 * r_8) + (dp_c2 * r_11) + (dp_d2 * r_6) + (dp_e2 * r_7) + (dp_f2 * r_9));
    if (F) {
      F[0] = ((p_a1 * r_10) + (p_c1 * r_11) + (p_f1 * r_9) + (r_0 * u_x) + (r_1 * u_x) + (r_3 * u_y));
      F[1] = ((p_a2 * r_10) + (p_c2 * r_11) + (p_f2 * r_9) + (r_12 * u_x) + (r_13 * u_x) + (r_14 * u_y));
    }
  }
  __device__ static void start(Rng& rng, int dist, double range, cd* z, cd* q) {
    typedef double T;
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[0] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[1] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[0] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[1] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[2] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[3] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[4] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[6] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[7] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[8] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[9] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[10] = cd(re, im); }
    const cx<T> u_x = z[0];
    const cx<T> u_y = z[1];
    const cx<T> p_a1 = q[0];
    const cx<T> p_b1 = q[1];
    const cx<T> p_c1 = q[2];
    const cx<T> p_d1 = q[3];
    const cx<T> p_e1 = q[4];
    const cx<T> p_a2 = q[6];
    const cx<T> p_b2 = q[7];
    const cx<T> p_c2 = q[8];
    const cx<T> p_d2 = q[9];
    const cx<T> p_e2 = q[10];
    const cx<T> s_0 = (u_x * u_y);
    const cx<T> s_1 = (u_x * u_x);
    const cx<T> s_2 = (u_y * u_y);
    cx<T> A[4], b[2], s[2];
    A[0] = cx<T>(T(1.0));
    A[1] = cx<T>(T(0));
    A[2] = cx<T>(T(0));
    A[3] = cx<T>(T(1.0));
    b[0] = ((-(p_a1 * s_1)) - (p_b1 * s_0) - (p_c1 * s_2) - (p_d1 * u_x) - (p_e1 * u_y));
    b[1] = ((-(p_a2 * s_1)) - (p_b2 * s_0) - (p_c2 * s_2) - (p_d2 * u_x) - (p_e2 * u_y));
    small_solve<2>(A, b, s);
    q[5] = s[0];
    q[11] = s[1];
  }
  __device__ static void canonical(const cd* root, const cd*, cd* out) {
    for (int i = 0; i < NV; ++i) out[i] = root[i];
  }
};

// ---- system 2: burmester5 (5 unknowns, 20 parameters)
// rows(): 158 complex mul, 101 complex add/sub, 5 real x complex; as a warp's schedule
// 259 operations in 19 steps
static __device__ const uint32_t tape_burmester5[304] = {
    0x8030542fu, 0x80204030u, 0x80c01431u, 0x80204432u, 0x80305c33u, 0x80204834u, 0x80306035u, 0x80204c36u, 
    0x80306437u, 0x80205038u, 0x80601439u, 0x8030583au, 0x8080143bu, 0x8090143cu, 0x80a0143du, 0x8010003eu, 
    0x8050103fu, 0x80b01440u, 0x80701441u, 0x80d01442u, 0x80e01443u, 0x80f01444u, 0x8300bc45u, 0x8320c446u, 
    0x8340cc47u, 0x8360d448u, 0x8380dc49u, 0x8390bc4au, 0x83a0c84bu, 0x83b0cc4cu, 0x83c0d44du, 0x83d0dc4eu, 
    0x43f0f84fu, 0x42f00450u, 0x43100451u, 0x43300452u, 0x43500453u, 0x43700454u, 0x43000055u, 0x410c856u, 
    0x3b0d057u, 0x3c0d858u, 0x3d0e059u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x4513c3eu, 0x4613c3fu, 0x4713c5au, 
    0x4813c5bu, 0x4913c5cu, 0x4401405du, 0x43a1445eu, 0x4421485fu, 0x44314c60u, 0x44415061u, 0x43915462u, 
    0x40015863u, 0x40015c64u, 0x40016065u, 0x40016466u, 0x89u, 0x83010045u, 0x83a10446u, 0x83410847u, 0x83610c48u, 
    0x83811049u, 0x80b0004fu, 0x80b04050u, 0x81a01451u, 0x81f01452u, 0x80c00053u, 0x80c04454u, 0x81b01455u, 
    0x82001456u, 0x80d00057u, 0x80d04858u, 0x81c01459u, 0x82101467u, 0x80e00068u, 0x80e04c69u, 0x81d0146au, 
    0x8220146bu, 0x80f0006cu, 0x80f0506du, 0x81e0146eu, 0x8230146fu, 0x82f00070u, 0x83100071u, 0x83300072u, 
    0x83500073u, 0x83700074u, 0x80600475u, 0x80605476u, 0x4a0f82fu, 0x4b0fc31u, 0x4c16833u, 0x4d16c35u, 0x4e17037u, 
    0x4f01077u, 0x5301078u, 0x5701079u, 0x680107au, 0x6c0107bu, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 
    0x85d0903eu, 0x8070043fu, 0x8070584au, 0x85e0944bu, 0x8080044cu, 0x80805c4du, 0x85f0984eu, 0x8090044fu, 
    0x80906053u, 0x86009c57u, 0x80a0045au, 0x80a0645bu, 0x8610a05cu, 0x84000068u, 0x83a0006cu, 0x8420007cu, 
    0x450bc3au, 0x460c440u, 0x470cc42u, 0x480d47du, 0x490dc7eu, 0x751dc7fu, 0x3f1e080u, 0x4c1e481u, 0x4f1e882u, 
    0x5a1ec83u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x8430002fu, 0x84400031u, 0x80501433u, 0x80214035u, 
    0x85d14437u, 0x8621483fu, 0x8620a445u, 0x80215046u, 0x85e15447u, 0x86315848u, 0x8630a849u, 0x8021604cu, 
    0x85f1644fu, 0x86419c5au, 0x8640ac75u, 0x8021a477u, 0x8601a878u, 0x8651ac79u, 0x8650b07au, 0x8021b47bu, 
    0x8611b843u, 0x8661bc44u, 0x8660b450u, 0x83000451u, 0x80b01852u, 0x83200454u, 0x80c01c55u, 0x83400456u, 
    0x80d02058u, 0x83600459u, 0x80e02467u, 0x83800469u, 0x4700e830u, 0x47110032u, 0x47210834u, 0x4731f436u, 
    0x4741f838u, 0x4351fc6au, 0x3f0dc6bu, 0x4462006du, 0x44811c6eu, 0x44c2046fu, 0x45a13c84u, 0x47720885u, 
    0x4791e086u, 0x47b20c87u, 0x44410c88u, 0x89u, 0x80f02835u, 0x8031d837u, 0x80b0e43au, 0x8020f83fu, 0x80312840u, 
    0x80c10442u, 0x80212c43u, 0x80313444u, 0x80d0ec46u, 0x80213847u, 0x80314c48u, 0x80e0f04cu, 0x80215c4fu, 
    0x80316c5au, 0x80f0f470u, 0x80217071u, 0x4680c072u, 0x46c0c873u, 0x47c0d074u, 0x42f0d877u, 0x4310e078u, 
    0x4371a879u, 0x3a0e87bu, 0x3f1ac7du, 0x4401b47eu, 0x421087fu, 0x431b880u, 0x4441bc81u, 0x4611882u, 0x4721083u, 
    0x4482143eu, 0x4c1304au, 0x8390044bu, 0x8410044du, 0x83b0044eu, 0x83c00453u, 0x83d00457u, 0x8031145bu, 
    0x8031245cu, 0x8031d476u, 0x8031e82fu, 0x80314030u, 0x83314831u, 0x83315432u, 0x83316034u, 0x83319c36u, 
    0x8330d437u, 0x85d04038u, 0x4511c83au, 0x4541cc3fu, 0x4561d040u, 0x4591dc42u, 0x4691e043u, 0x4f21844u, 
    0x45a21c46u, 0x701c047u, 0x7122048u, 0x47b1e44cu, 0x5b1f468u, 0x47f1f86au, 0x45c2006bu, 0x4822046cu, 
    0x47620c6du, 0x44a0f86eu, 0x8620546fu, 0x85e0447cu, 0x86305884u, 0x85f04885u, 0x86405c33u, 0x86004c35u, 
    0x86506039u, 0x8610503bu, 0x8660643cu, 0x80000089u, 0x80000089u, 0x80000089u, 0x80000089u, 0x80000089u, 
    0x80000089u, 0x80000089u, 0x44b0e83du, 0x44d0fc41u, 0x44e10045u, 0x45310849u, 0x45710c50u, 0x42f11052u, 
    0x44711855u, 0x43012058u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x310f467u, 0x3210475u, 
    0x341147au, 0x361243eu, 0x371404au, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u, 0x89u};
static __device__ const uint16_t tape_out_burmester5[40] = {
    93, 98, 1080, 1135, 1029, 1100, 1128, 94, 1123, 1148, 132, 1029, 1130, 1131, 95, 1124, 1157, 51, 1029, 1132, 
    1133, 96, 1125, 1077, 57, 1029, 1134, 1106, 97, 1126, 1083, 60, 1029, 1109, 1112, 103, 117, 122, 62, 74};
static __device__ const double tape_const_burmester5[1] = {
    0.0};
struct Sys_burmester5 {
  static constexpr int ID = 2;
  static constexpr int NV = 5;
  static constexpr int NP = 20;
  static constexpr int NS = 5;
  static constexpr int ROWS_CMUL = 158, ROWS_CADD = 101, ROWS_SMUL = 5;
  static constexpr int TAPE_STEPS = 19, TAPE_REGS = 138, TAPE_CONSTS = 1;
  __device__ static const uint32_t* tape() { return tape_burmester5; }
  __device__ static const uint16_t* tape_out() { return tape_out_burmester5; }
  __device__ static const double* tape_const() { return tape_const_burmester5; }
  template <typename T, int LD>
  __device__ static void rows(const cx<T>* Y, const cx<T>* q, const cx<T>* dq, cx<T>* M, cx<T>* F) {
    const cx<T> u_G = Y[0];
    const cx<T> u_Gc = Y[1];
    const cx<T> u_z = Y[2];
    const cx<T> u_zc = Y[3];
    const cx<T> u_R = Y[4];
    const cx<T> u_Z0 = Y[5];
    const cx<T> p_d0 = q[0];
    const cx<T> dp_d0 = dq[0];
    const cx<T> p_d1 = q[1];
    const cx<T> dp_d1 = dq[1];
    const cx<T> p_d2 = q[2];
    const cx<T> dp_d2 = dq[2];
    const cx<T> p_d3 = q[3];
    const cx<T> dp_d3 = dq[3];
    const cx<T> p_d4 = q[4];
    const cx<T> dp_d4 = dq[4];
    const cx<T> p_dc0 = q[5];
    const cx<T> dp_dc0 = dq[5];
    const cx<T> p_dc1 = q[6];
    const cx<T> dp_dc1 = dq[6];
    const cx<T> p_dc2 = q[7];
    const cx<T> dp_dc2 = dq[7];
    const cx<T> p_dc3 = q[8];
    const cx<T> dp_dc3 = dq[8];
    const cx<T> p_dc4 = q[9];
    const cx<T> dp_dc4 = dq[9];
    const cx<T> p_T0 = q[10];
    const cx<T> dp_T0 = dq[10];
    const cx<T> p_T1 = q[11];
    const cx<T> dp_T1 = dq[11];
    const cx<T> p_T2 = q[12];
    const cx<T> dp_T2 = dq[12];
    const cx<T> p_T3 = q[13];
    const cx<T> dp_T3 = dq[13];
    const cx<T> p_T4 = q[14];
    const cx<T> dp_T4 = dq[14];
    const cx<T> p_Tc0 = q[15];
    const cx<T> dp_Tc0 = dq[15];
    const cx<T> p_Tc1 = q[16];
    const cx<T> dp_Tc1 = dq[16];
    const cx<T> p_Tc2 = q[17];
    const cx<T> dp_Tc2 = dq[17];
    const cx<T> p_Tc3 = q[18];
    const cx<T> dp_Tc3 = dq[18];
    const cx<T> p_Tc4 = q[19];
    const cx<T> dp_Tc4 = dq[19];
    const cx<T> r_0 = (-(u_Gc));
    const cx<T> r_1 = (p_Tc0 * u_zc);
    const cx<T> r_2 = (u_Z0 * p_dc0);
    const cx<T> r_3 = (r_0 + r_1 + r_2);
    const cx<T> r_4 = (-(u_G));
    const cx<T> r_5 = (p_T0 * u_z);
    const cx<T> r_6 = (u_Z0 * p_d0);
    const cx<T> r_7 = (r_4 + r_5 + r_6);
    const cx<T> r_8 = (-(u_Z0));
    const cx<T> r_9 = (p_Tc1 * u_zc);
    const cx<T> r_10 = (u_Z0 * p_dc1);
    const cx<T> r_11 = (r_0 + r_10 + r_9);
    const cx<T> r_12 = (p_T1 * u_z);
    const cx<T> r_13 = (u_Z0 * p_d1);
    const cx<T> r_14 = (r_12 + r_13 + r_4);
    const cx<T> r_15 = (p_Tc2 * u_zc);
    const cx<T> r_16 = (u_Z0 * p_dc2);
    const cx<T> r_17 = (r_0 + r_15 + r_16);
    const cx<T> r_18 = (p_T2 * u_z);
    const cx<T> r_19 = (u_Z0 * p_d2);
    const cx<T> r_20 = (r_18 + r_19 + r_4);
    const cx<T> r_21 = (p_Tc3 * u_zc);
    const cx<T> r_22 = (u_Z0 * p_dc3);
    const cx<T> r_23 = (r_0 + r_21 + r_22);
    const cx<T> r_24 = (p_T3 * u_z);
    const cx<T> r_25 = (u_Z0 * p_d3);
    const cx<T> r_26 = (r_24 + r_25 + r_4);
    const cx<T> r_27 = (p_Tc4 * u_zc);
    const cx<T> r_28 = (u_Z0 * p_dc4);
    const cx<T> r_29 = (r_0 + r_27 + r_28);
    const cx<T> r_30 = (p_T4 * u_z);
    const cx<T> r_31 = (u_Z0 * p_d4);
    const cx<T> r_32 = (r_30 + r_31 + r_4);
    const cx<T> r_33 = (u_Z0 * u_Z0);
    const cx<T> r_34 = ((u_G * u_Gc) - (u_R * u_Z0));
    M[0 * LD + 0] = (-(r_3));
    M[0 * LD + 1] = (-(r_7));
    M[0 * LD + 2] = (p_T0 * r_3);
    M[0 * LD + 3] = (p_Tc0 * r_7);
    M[0 * LD + 4] = r_8;
    M[0 * LD + 5] = ((-u_R) - (u_G * p_dc0) - (u_Gc * p_d0) + (p_T0 * p_dc0 * u_z) + (p_Tc0 * p_d0 * u_zc) + (T(2.0) * ((u_Z0 * p_d0 * p_dc0))));
    M[0 * LD + 6] = ((u_Z0 * dp_d0 * r_3) + (u_Z0 * dp_dc0 * r_7) + (dp_T0 * r_3 * u_z) + (dp_Tc0 * r_7 * u_zc));
    M[1 * LD + 0] = (-(r_11));
    M[1 * LD + 1] = (-(r_14));
    M[1 * LD + 2] = (p_T1 * r_11);
    M[1 * LD + 3] = (p_Tc1 * r_14);
    M[1 * LD + 4] = r_8;
    M[1 * LD + 5] = ((-u_R) - (u_G * p_dc1) - (u_Gc * p_d1) + (p_T1 * p_dc1 * u_z) + (p_Tc1 * p_d1 * u_zc) + (T(2.0) * ((u_Z0 * p_d1 * p_dc1))));
    M[1 * LD + 6] = ((u_Z0 * dp_d1 * r_11) + (u_Z0 * dp_dc1 * r_14) + (dp_T1 * r_11 * u_z) + (dp_Tc1 * r_14 * u_zc));
    M[2 * LD + 0] = (-(r_17));
    M[2 * LD + 1] = (-(r_20));
    M[2 * LD + 2] = (p_T2 * r_17);
    M[2 * LD + 3] = (p_Tc2 * r_20);
    M[2 * LD + 4] = r_8;
    M[2 * LD + 5] = ((-u_R) - (u_G * p_dc2) - (u_Gc * p_d2) + (p_T2 * p_dc2 * u_z) + (p_Tc2 * p_d2 * u_zc) + (T(2.0) * ((u_Z0 * p_d2 * p_dc2))));
    M[2 * LD + 6] = ((u_Z0 * dp_d2 * r_17) + (u_Z0 * dp_dc2 * r_20) + (dp_T2 * r_17 * u_z) + (dp_Tc2 * r_20 * u_zc));
    M[3 * LD + 0] = (-(r_23));
    M[3 * LD + 1] = (-(r_26));
    M[3 * LD + 2] = (p_T3 * r_23);
    M[3 * LD + 3] = (p_Tc3 * r_26);
    M[3 * LD + 4] = r_8;
    M[3 * LD + 5] = ((-u_R) - (u_G * p_dc3) - (u_Gc * p_d3) + (p_T3 * p_dc3 * u_z) + (p_Tc3 * p_d3 * u_zc) + (T(2.0) * ((u_Z0 * p_d3 * p_dc3))));
    M[3 * LD + 6] = ((u_Z0 * dp_d3 * r_23) + (u_Z0 * dp_dc3 * r_26) + (dp_T3 * r_23 * u_z) + (dp_Tc3 * r_26 * u_zc));
    M[4 * LD + 0] = (-(r_29));
    M[4 * LD + 1] = (-(r_32));
    M[4 * LD + 2] = (p_T4 * r_29);
    M[4 * LD + 3] = (p_Tc4 * r_32);
    M[4 * LD + 4] = r_8;
    M[4 * LD + 5] = ((-u_R) - (u_G * p_dc4) - (u_Gc * p_d4) + (p_T4 * p_dc4 * u_z) + (p_Tc4 * p_d4 * u_zc) + (T(2.0) * ((u_Z0 * p_d4 * p_dc4))));
    M[4 * LD + 6] = ((u_Z0 * dp_d4 * r_29) + (u_Z0 * dp_dc4 * r_32) + (dp_T4 * r_29 * u_z) + (dp_Tc4 * r_32 * u_zc));
    if (F) {
      F[0] = (r_34 + (r_1 * r_5) + (r_1 * r_6) + (r_2 * r_5) - (u_G * r_1) - (u_G * r_2) - (u_Gc * r_5) - (u_Gc * r_6) + (p_d0 * p_dc0 * r_33));
      F[1] = (r_34 + (r_10 * r_12) + (r_12 * r_9) + (r_13 * r_9) - (u_G * r_10) - (u_G * r_9) - (u_Gc * r_12) - (u_Gc * r_13) + (p_d1 * p_dc1 * r_33));
      F[2] = (r_34 + (r_15 * r_18) + (r_15 * r_19) + (r_16 * r_18) - (u_G * r_15) - (u_G * r_16) - (u_Gc * r_18) - (u_Gc * r_19) + (p_d2 * p_dc2 * r_33));
      F[3] = (r_34 + (r_21 * r_24) + (r_21 * r_25) + (r_22 * r_24) - (u_G * r_21) - (u_G * r_22) - (u_Gc * r_24) - (u_Gc * r_25) + (p_d3 * p_dc3 * r_33));
      F[4] = (r_34 + (r_27 * r_30) + (r_27 * r_31) + (r_28 * r_30) - (u_G * r_27) - (u_G * r_28) - (u_Gc * r_30) - (u_Gc * r_31) + (p_d4 * p_dc4 * r_33));
    }
  }
  __device__ static void start(Rng& rng, int dist, double range, cd* z, cd* q) {
    typedef double T;
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[0] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[1] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[2] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[3] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); z[4] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[5] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[6] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[7] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[8] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[9] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[10] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[11] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[12] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[13] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[14] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[15] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[16] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[17] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[18] = cd(re, im); }
    { const double re = start_value(rng, dist, range); const double im = start_value(rng, dist, range); q[19] = cd(re, im); }
    const cx<T> u_G = z[0];
    const cx<T> u_Gc = z[1];
    const cx<T> u_z = z[2];
    const cx<T> u_zc = z[3];
    const cx<T> u_R = z[4];
    const cx<T> p_dc0 = q[5];
    const cx<T> p_dc1 = q[6];
    const cx<T> p_dc2 = q[7];
    const cx<T> p_dc3 = q[8];
    const cx<T> p_dc4 = q[9];
    const cx<T> p_T0 = q[10];
    const cx<T> p_T1 = q[11];
    const cx<T> p_T2 = q[12];
    const cx<T> p_T3 = q[13];
    const cx<T> p_T4 = q[14];
    const cx<T> p_Tc0 = q[15];
    const cx<T> p_Tc1 = q[16];
    const cx<T> p_Tc2 = q[17];
    const cx<T> p_Tc3 = q[18];
    const cx<T> p_Tc4 = q[19];
    const cx<T> s_0 = (-(u_Gc));
    const cx<T> s_1 = (p_Tc0 * u_zc);
    const cx<T> s_2 = (p_Tc1 * u_zc);
    const cx<T> s_3 = (p_Tc2 * u_zc);
    const cx<T> s_4 = (p_Tc3 * u_zc);
    const cx<T> s_5 = (p_Tc4 * u_zc);
    const cx<T> s_6 = (u_R - (u_G * u_Gc));
    cx<T> A[25], b[5], s[5];
    A[0] = (p_dc0 + s_0 + s_1);
    A[1] = cx<T>(T(0));
    A[2] = cx<T>(T(0));
    A[3] = cx<T>(T(0));
    A[4] = cx<T>(T(0));
    A[5] = cx<T>(T(0));
    A[6] = (p_dc1 + s_0 + s_2);
    A[7] = cx<T>(T(0));
    A[8] = cx<T>(T(0));
    A[9] = cx<T>(T(0));
    A[10] = cx<T>(T(0));
    A[11] = cx<T>(T(0));
    A[12] = (p_dc2 + s_0 + s_3);
    A[13] = cx<T>(T(0));
    A[14] = cx<T>(T(0));
    A[15] = cx<T>(T(0));
    A[16] = cx<T>(T(0));
    A[17] = cx<T>(T(0));
    A[18] = (p_dc3 + s_0 + s_4);
    A[19] = cx<T>(T(0));
    A[20] = cx<T>(T(0));
    A[21] = cx<T>(T(0));
    A[22] = cx<T>(T(0));
    A[23] = cx<T>(T(0));
    A[24] = (p_dc4 + s_0 + s_5);
    b[0] = (s_6 + (u_G * p_dc0) + (u_G * s_1) + (u_Gc * p_T0 * u_z) - (p_T0 * p_dc0 * u_z) - (p_T0 * p_Tc0 * u_z * u_zc));
    b[1] = (s_6 + (u_G * p_dc1) + (u_G * s_2) + (u_Gc * p_T1 * u_z) - (p_T1 * p_dc1 * u_z) - (p_T1 * p_Tc1 * u_z * u_zc));
    b[2] = (s_6 + (u_G * p_dc2) + (u_G * s_3) + (u_Gc * p_T2 * u_z) - (p_T2 * p_dc2 * u_z) - (p_T2 * p_Tc2 * u_z * u_zc));
    b[3] = (s_6 + (u_G * p_dc3) + (u_G * s_4) + (u_Gc * p_T3 * u_z) - (p_T3 * p_dc3 * u_z) - (p_T3 * p_Tc3 * u_z * u_zc));
    b[4] = (s_6 + (u_G * p_dc4) + (u_G * s_5) + (u_Gc * p_T4 * u_z) - (p_T4 * p_dc4 * u_z) - (p_T4 * p_Tc4 * u_z * u_zc));
    small_solve<5>(A, b, s);
    q[0] = s[0];
    q[1] = s[1];
    q[2] = s[2];
    q[3] = s[3];
    q[4] = s[4];
  }
  __device__ static void canonical(const cd* root, const cd*, cd* out) {
    for (int i = 0; i < NV; ++i) out[i] = root[i];
  }
};

}  // namespace frg

// X(id, name, struct) for every plug-in
#define FRG_PLUGIN_LIST(X) \
  X(1, "conic2", frg::Sys_conic2) \
  X(2, "burmester5", frg::Sys_burmester5) \

#define FRG_NUM_PLUGINS 2
