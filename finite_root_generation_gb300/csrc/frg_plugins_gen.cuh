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
    0x80100024u, 0x80000026u, 0x80100427u, 0x80200825u, 0x8060081cu, 0x80000822u, 0x80c00828u, 0x8010101du, 
    0x80100823u, 0x80102829u, 0x8070081fu, 0x80d0082au, 0x8000102eu, 0x80001832u, 0x80101c33u, 0x80002845u, 
    0x82603c37u, 0x82404038u, 0x8260544eu, 0x8240584fu, 0x82600c59u, 0x8270145au, 0x82602464u, 0x82702c65u, 
    0x8270443au, 0x82705c51u, 0x8250205cu, 0x82503867u, 0x8220483cu, 0x82206053u, 0x8000705eu, 0x8000a069u, 
    0x380dc39u, 0x4f13850u, 0x5a1645bu, 0x6519066u, 0x1eu, 0x100420u, 0x200821u, 0x1d0702bu, 0x2e07c2fu, 0x330c834u, 
    0x290a042u, 0x450a846u, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x3a0e43bu, 0x5114052u, 0x5c16c5du, 0x6719868u, 0x6fu, 
    0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x82304c3eu, 0x80003049u, 
    0x8010344au, 0x82306455u, 0x80007460u, 0x8000a46bu, 0x81e00c2cu, 0x82001430u, 0x82102035u, 0x82505040u, 
    0x81e02443u, 0x82002c47u, 0x8210384cu, 0x82506857u, 0x80107c62u, 0x8010a86du, 0x3c0ec3du, 0x5314854u, 
    0x5e1745fu, 0x691a06au, 0x4a1244bu, 0x2c0ac2du, 0x300bc31u, 0x350d036u, 0x4310844u, 0x4711848u, 0x6fu, 0x6fu, 
    0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x3e0f43fu, 0x5515056u, 0x6017c61u, 0x6b1a86cu, 0x4c12c4du, 0x6fu, 0x6fu, 0x6fu, 
    0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x400fc41u, 0x5715858u, 0x6218463u, 0x6d1b06eu, 0x6fu, 
    0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu, 0x6fu};
static __device__ const uint16_t tape_out_conic2[10] = {
    45, 49, 54, 65, 68, 72, 77, 88, 99, 110};
static __device__ const double tape_const_conic2[1] = {
    0.0};
struct Sys_conic2 {
  static constexpr int ID = 1;
  static constexpr int NV = 2;
  static constexpr int NP = 12;
  static constexpr int NS = 2;
  static constexpr int ROWS_CMUL = 48, ROWS_CADD = 32, ROWS_SMUL = 3;
  static constexpr int TAPE_STEPS = 8, TAPE_REGS = 112, TAPE_CONSTS = 1;
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
    0x8030542fu, 0x80204033u, 0x80c01438u, 0x8020443bu, 0x80305c3fu, 0x80204843u, 0x80306047u, 0x80204c4bu, 
    0x8030644fu, 0x80205053u, 0x80601434u, 0x80305837u, 0x80801444u, 0x8090144cu, 0x80a01454u, 0x80100058u, 
    0x80501059u, 0x80b01430u, 0x8070143cu, 0x80d01440u, 0x80e01448u, 0x80f01450u, 0x8330bcddu, 0x83b0e0eeu, 
    0x8430fcffu, 0x84b11d10u, 0x85313d21u, 0x8340bcdfu, 0x8370ecf0u, 0x8440fd01u, 0x84c11d12u, 0x85413d23u, 
    0x4591605au, 0x42f00431u, 0x43800439u, 0x43f00441u, 0x44700449u, 0x44f00451u, 0x43300035u, 0x3c0ec3du, 
    0x4410c45u, 0x4c12c4du, 0x5414c55u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0xdd168deu, 0xee168efu, 0xff16900u, 
    0x11016911u, 0x12116922u, 0x4300c432u, 0x4370e43au, 0x44010442u, 0x4481244au, 0x45014452u, 0x4340d436u, 
    0x4000f43eu, 0x40011446u, 0x4001344eu, 0x40015456u, 0x132u, 0x8330c0e1u, 0x8370f0f2u, 0x84310103u, 0x84b12114u, 
    0x85314125u, 0x80b0005du, 0x80b04061u, 0x81a0146au, 0x81f0146cu, 0x80c00077u, 0x80c0447bu, 0x81b01484u, 
    0x82001486u, 0x80d00091u, 0x80d04895u, 0x81c0149eu, 0x821014a0u, 0x80e000abu, 0x80e04cafu, 0x81d014b8u, 
    0x822014bau, 0x80f000c5u, 0x80f050c9u, 0x81e014d2u, 0x823014d4u, 0x82f000e3u, 0x838000f4u, 0x83f00105u, 
    0x84700116u, 0x84f00127u, 0x8060045fu, 0x80605464u, 0xdf378e0u, 0xf03bcf1u, 0x10140102u, 0x11244513u, 
    0x12348924u, 0x5d0105eu, 0x7701078u, 0x9101092u, 0xab010acu, 0xc5010c6u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 
    0x132u, 0x8320906fu, 0x80700479u, 0x8070587eu, 0x83a09489u, 0x80800493u, 0x80805c98u, 0x842098a3u, 0x809004adu, 
    0x809060b2u, 0x84a09cbdu, 0x80a004c7u, 0x80a064ccu, 0x8520a0d7u, 0x830000e5u, 0x837000f6u, 0x84000107u, 
    0xe1380e2u, 0xf23c4f3u, 0x10340904u, 0x11444d15u, 0x12549126u, 0x5f17860u, 0x791e07au, 0x9324894u, 0xad2b0aeu, 
    0xc7318c8u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x84800118u, 0x85000129u, 0x80501457u, 0x80218462u, 
    0x8321a86bu, 0x8361b06du, 0x8360a472u, 0x8021ec7cu, 0x83a21085u, 0x83e21887u, 0x83e0a88cu, 0x80225496u, 
    0x8422789fu, 0x846280a1u, 0x8460aca6u, 0x8022bcb0u, 0x84a2e0b9u, 0x84e2e8bbu, 0x84e0b0c0u, 0x802324cau, 
    0x852348d3u, 0x856350d5u, 0x8560b4dau, 0x833004e7u, 0x80b018ebu, 0x83b004f8u, 0x80c01cfcu, 0x84300509u, 
    0x80d0210du, 0x84b0051au, 0x80e0251eu, 0x8530052bu, 0x4e3388e4u, 0x4f43ccf5u, 0x50541106u, 0x51645517u, 
    0x52749928u, 0x46218063u, 0x6d1ac6eu, 0x47c1e87du, 0x48721488u, 0x49625097u, 0x4a127ca2u, 0x4b02b8b1u, 
    0x4bb2e4bcu, 0x4ca320cbu, 0x4d534cd6u, 0x132u, 0x80f0292fu, 0x80319065u, 0x80b0d067u, 0x8021bc70u, 0x8031f87fu, 
    0x80c0f081u, 0x8022248au, 0x80326099u, 0x80d1109bu, 0x80228ca4u, 0x8032c8b3u, 0x80e130b5u, 0x8022f4beu, 
    0x803330cdu, 0x80f150cfu, 0x80235cd8u, 0x4e5390e6u, 0x4f63d4f7u, 0x50741908u, 0x51845d19u, 0x5294a12au, 
    0x46518c66u, 0x6719c68u, 0x701b871u, 0x47f1f480u, 0x8120482u, 0x8a2208bu, 0x49925c9au, 0x9b26c9cu, 0xa4288a5u, 
    0x4b32c4b4u, 0xb52d4b6u, 0x834004e9u, 0x83c004fau, 0x8440050bu, 0x84c0051cu, 0x8540052du, 0x8031c873u, 
    0x8032308du, 0x803298a7u, 0x803300c1u, 0x803368dbu, 0x8573acecu, 0x8573f0fdu, 0x8574350eu, 0x8574791fu, 
    0x8574bd30u, 0x8320405bu, 0x4e7398e8u, 0x4f83dcf9u, 0x5094210au, 0x51a4651bu, 0x52b4a92cu, 0xbe2f0bfu, 
    0x4cd32cceu, 0xcf33cd0u, 0xd8358d9u, 0x46819869u, 0x731c474u, 0x48220083u, 0x48d22c8eu, 0x49c2689du, 
    0x4a7294a8u, 0x4b62d0b7u, 0x8360545cu, 0x83a04475u, 0x83e05876u, 0x8420488fu, 0x84605c90u, 0x84a04ca9u, 
    0x84e060aau, 0x852050c3u, 0x856064c4u, 0x80000132u, 0x80000132u, 0x80000132u, 0x80000132u, 0x80000132u, 
    0x80000132u, 0x80000132u, 0x4e93a0eau, 0x4fa3e4fbu, 0x50b4290cu, 0x51c46d1du, 0x52d4b12eu, 0x4c12fcc2u, 
    0x4d0338d1u, 0x4db364dcu, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0xec3a8edu, 
    0xfd3ecfeu, 0x10e4310fu, 0x11f47520u, 0x1304b931u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 0x132u, 
    0x132u, 0x132u, 0x132u, 0x132u};
static __device__ const uint16_t tape_out_burmester5[40] = {
    50, 54, 1115, 1116, 1029, 1129, 1140, 58, 1086, 1141, 118, 1029, 1155, 1166, 66, 1094, 1167, 144, 1029, 1181, 
    1192, 74, 1102, 1193, 170, 1029, 1207, 1218, 82, 1110, 1219, 196, 1029, 1233, 1244, 237, 254, 271, 288, 305};
static __device__ const double tape_const_burmester5[1] = {
    0.0};
struct Sys_burmester5 {
  static constexpr int ID = 2;
  static constexpr int NV = 5;
  static constexpr int NP = 20;
  static constexpr int NS = 5;
  static constexpr int ROWS_CMUL = 158, ROWS_CADD = 101, ROWS_SMUL = 5;
  static constexpr int TAPE_STEPS = 19, TAPE_REGS = 307, TAPE_CONSTS = 1;
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
