// GENERATED by finite_root_generation_gb300/gen/gen_system.py -- do not edit.
//
// One j-group of the Stephenson II loop-closure system (reference FSYS,
// htpykinematics.cu:36-122): the three equations (rows j-1, j+6, j+13), their
// nonzero partial derivatives over Z (JVAR's sparsity, htpykinematics.cu:129-1129)
// and the t-derivative dF/dq . dq/dt (JH's last column, htpysupport.cu:113-121).
// Straight-line cost per group: 352 complex mul, 239 complex add/sub,
// 5 real-scalar x complex.
// The three equations alone: 62 complex mul, 57 complex add/sub, 0 real x complex.
#pragma once

#define FRG_GEN_CMUL 352
#define FRG_GEN_CADD 239
#define FRG_GEN_SMUL 5

// Output slots: fI, dI[8] over {A,C,H,Ac,Cc,Hc,U_j,Z0}, tI;
//               fII, dII[6] over {B,F,Bc,Fc,U_j,Z0}, tII;
//               fIII, dIII[16] over {A..H,Ac..Hc,U_j,Z0}, tIII.
template <typename T>
struct FrgGroupOut {
  cx<T> fI, dI[8], tI;
  cx<T> fII, dII[6], tII;
  cx<T> fIII, dIII[16], tIII;
};

// Column in Z of each derivative slot (U_j's column is 13 + j, marked -1).
#define FRG_COLS_I {0, 2, 6, 7, 9, 13, -1, 21}
#define FRG_COLS_II {1, 4, 8, 11, -1, 21}
#define FRG_COLS_III {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, -1, 21}

template <typename T>
__device__ __forceinline__ void frg_group_eval(
    const cx<T> A, const cx<T> B, const cx<T> C, const cx<T> D, const cx<T> F, const cx<T> G,
    const cx<T> H, const cx<T> Ac, const cx<T> Bc, const cx<T> Cc, const cx<T> Dc, const cx<T> Fc,
    const cx<T> Gc, const cx<T> Hc, const cx<T> z,
    const cx<T> e1, const cx<T> e2, const cx<T> ec1, const cx<T> ec2,
    const cx<T> z2, const cx<T> z3,
    const cx<T> P0, const cx<T> Pc0, const cx<T> dP0, const cx<T> dPc0,
    const cx<T> U, const cx<T> iU, const cx<T> Pj, const cx<T> Pcj, const cx<T> Qj, const cx<T> Qcj,
    const cx<T> dPj, const cx<T> dPcj, const cx<T> dQj, const cx<T> dQcj,
    FrgGroupOut<T>& o) {
  const cx<T> x0 = P0*Pc0 + Pcj*Pj;
  const cx<T> x1 = x0*z3;
  const cx<T> x2 = Pc0*z;
  const cx<T> x3 = (-(x2));
  const cx<T> x4 = Cc + x3;
  const cx<T> x5 = x4*z;
  const cx<T> x6 = P0*z;
  const cx<T> x7 = (-(x6));
  const cx<T> x8 = C + x7;
  const cx<T> x9 = Hc*z;
  const cx<T> x10 = (-(Ac));
  const cx<T> x11 = Pcj*z;
  const cx<T> x12 = x10 + x11;
  const cx<T> x13 = Cc + x12;
  const cx<T> x14 = x13*z;
  const cx<T> x15 = (-(A));
  const cx<T> x16 = Pj*z;
  const cx<T> x17 = x15 + x16;
  const cx<T> x18 = C + x17;
  const cx<T> x19 = Ac*z;
  const cx<T> x20 = Ac - Cc;
  const cx<T> x21 = Qcj*x20;
  const cx<T> x22 = (-(x16));
  const cx<T> x23 = A + x22;
  const cx<T> x24 = x23*z;
  const cx<T> x25 = A - C;
  const cx<T> x26 = Qj*x25;
  const cx<T> x27 = (-(x11));
  const cx<T> x28 = Ac + x27;
  const cx<T> x29 = x28*z;
  const cx<T> x30 = (-x12) - x21;
  const cx<T> x31 = H + x7;
  const cx<T> x32 = U*x31;
  const cx<T> x33 = (-x17) - x26;
  const cx<T> x34 = Hc + x3;
  const cx<T> x35 = iU*x34;
  const cx<T> x36 = x35*z2;
  const cx<T> x37 = Qj*x29;
  const cx<T> x38 = (-cx<T>(T(1.0))) + Qj;
  const cx<T> x39 = x28 - Qcj*x20;
  const cx<T> x40 = U*x39;
  const cx<T> x41 = A*z;
  const cx<T> x42 = Qcj*x24;
  const cx<T> x43 = (-cx<T>(T(1.0))) + Qcj;
  const cx<T> x44 = (-(Qj*x25));
  const cx<T> x45 = x23 + x44;
  const cx<T> x46 = iU*x45;
  const cx<T> x47 = x46*z2;
  const cx<T> x48 = z2*(iU*iU);
  const cx<T> x49 = (T(3.0)*(x0*z2));
  const cx<T> x50 = Pj*z2;
  const cx<T> x51 = iU*z2;
  const cx<T> x52 = Pc0*z3;
  const cx<T> x53 = P0*z3;
  const cx<T> x54 = Pj*z3;
  const cx<T> x55 = Pcj*z3;
  const cx<T> x56 = Bc + x3;
  const cx<T> x57 = x56*z;
  const cx<T> x58 = B + x7;
  const cx<T> x59 = Fc*z;
  const cx<T> x60 = B*Pcj + Bc*Pj;
  const cx<T> x61 = Bc + x27;
  const cx<T> x62 = F + x7;
  const cx<T> x63 = B + x22;
  const cx<T> x64 = Fc + x3;
  const cx<T> x65 = x51*x64;
  const cx<T> x66 = U*x61;
  const cx<T> x67 = U*x62;
  const cx<T> x68 = x51*x63;
  const cx<T> x69 = iU*z3;
  const cx<T> x70 = (-(G));
  const cx<T> x71 = D + x70;
  const cx<T> x72 = (-(Gc));
  const cx<T> x73 = Dc + x72;
  const cx<T> x74 = x73*z;
  const cx<T> x75 = B - D;
  const cx<T> x76 = e1*x75;
  const cx<T> x77 = C + x70;
  const cx<T> x78 = e2*x77;
  const cx<T> x79 = x62*x76 - x31*x78;
  const cx<T> x80 = Bc - Dc;
  const cx<T> x81 = ec1*x80;
  const cx<T> x82 = Cc + x72;
  const cx<T> x83 = ec2*x82;
  const cx<T> x84 = x64*x81 - x34*x83;
  const cx<T> x85 = x79*x84;
  const cx<T> x86 = ec2*x39;
  const cx<T> x87 = Bc + x10 + x21 + x61*x81 - x82*x86;
  const cx<T> x88 = U*x79;
  const cx<T> x89 = e2*x45;
  const cx<T> x90 = B + x15 + x26 + x63*x76 - x77*x89;
  const cx<T> x91 = x51*x84;
  const cx<T> x92 = x87*z;
  const cx<T> x93 = x91 - x92;
  const cx<T> x94 = x84*z;
  const cx<T> x95 = e1*x63;
  const cx<T> x96 = cx<T>(T(1.0)) + x76 + x95;
  const cx<T> x97 = (-(x84));
  const cx<T> x98 = x97*z;
  const cx<T> x99 = x62*x98;
  const cx<T> x100 = (-(x87));
  const cx<T> x101 = x100*x67;
  const cx<T> x102 = x100*z;
  const cx<T> x103 = x101 - x99 + x68*x97 - x102*x63;
  const cx<T> x104 = x32*x87;
  const cx<T> x105 = Qj + x89 + Qj*x78;
  const cx<T> x106 = x51*x97;
  const cx<T> x107 = U*x100;
  const cx<T> x108 = x100*x32;
  const cx<T> x109 = x90*z;
  const cx<T> x110 = x88 - x109;
  const cx<T> x111 = (-(e2*x77));
  const cx<T> x112 = (-x111*x31) - x62*x76;
  const cx<T> x113 = (-(x80));
  const cx<T> x114 = (-(x113*x61));
  const cx<T> x115 = (-(x64*x80));
  const cx<T> x116 = (-(e1*x75));
  const cx<T> x117 = A + x44 - B + x116*x63 - x111*x45;
  const cx<T> x118 = U*x112*x114 + x112*x115*z - x114*x117*z - x115*x117*x51;
  const cx<T> x119 = ec1*x61;
  const cx<T> x120 = cx<T>(T(1.0)) + x119 + x81;
  const cx<T> x121 = (-(x79));
  const cx<T> x122 = U*x121;
  const cx<T> x123 = (-(x90));
  const cx<T> x124 = x121*z;
  const cx<T> x125 = ec1*x123*x65 - ec1*x124*x64;
  const cx<T> x126 = Qcj + x86 + Qcj*x83;
  const cx<T> x127 = x36*x90;
  const cx<T> x128 = x71*z;
  const cx<T> x129 = x123*z;
  const cx<T> x130 = x121*x40;
  const cx<T> x131 = x123*x36;
  const cx<T> x132 = x76 - x78;
  const cx<T> x133 = x81 - x83;
  const cx<T> x134 = (-(x133));
  const cx<T> x135 = (-(x132));
  const cx<T> x136 = U*x87;
  const cx<T> x137 = x51*x90;
  o.fI = (-x1) + A*x14 + x18*x19 + x21*x24 + x26*x29 + x30*x32 + x33*x36 - H*x5 - x8*x9;
  o.dI[0] = x14 + x37 - x19 + x21*z - x36*x38;
  o.dI[1] = x19 - x37 - x9 + Qj*x36;
  o.dI[2] = x40 - x5;
  o.dI[3] = x42 - x41 + x18*z + x26*z - x32*x43;
  o.dI[4] = x41 - x42 + Qcj*x32 - H*z;
  o.dI[5] = x47 - x8*z;
  o.dI[6] = x31*x39 - x34*x45*x48;
  o.dI[7] = (-x49) + A*x11 + A*x13 + Ac*x16 + Ac*x18 + H*x2 + Hc*x6 + x21*x23 + x26*x28 - H*x4 - Hc*x8 - Pcj*x32 - x11*x26 - x16*x21 - x35*x50 - P0*U*x30 - Pc0*x33*x51 + (T(2.0)*(x33*x35*z));
  o.tI = (-dP0*(x52 + x40*z - Hc*z2)) - dPc0*(x53 + x46*z3 - H*z2) - dPcj*(x54 + x26*z2 + x32*z - A*z2) - dPj*(x55 + x21*z2 + x35*z3 - Ac*z2) - dQcj*x20*(x32 - x24) - dQj*x25*(x36 - x29);
  o.fII = (-x1) + x60*z2 - F*x57 - x58*x59 + U*x61*x62 + iU*x63*x64*z2;
  o.dII[0] = x65 - x59 + Pcj*z2;
  o.dII[1] = x66 - x57;
  o.dII[2] = x50 + x67 - F*z;
  o.dII[3] = x68 - x58*z;
  o.dII[4] = x61*x62 - x48*x63*x64;
  o.dII[5] = (-x49) - F*x56 - Fc*x58 - P0*x66 - Pc0*x68 - Pcj*x67 + (T(2.0)*(x60*z)) + F*Pc0*z + Fc*P0*z - iU*x50*x64 + (T(2.0)*(iU*x63*x64*z));
  o.tII = (-dP0*(x52 + x66*z - Fc*z2)) - dPc0*(x53 + x63*x69 - F*z2) - dPcj*(x54 + x67*z - B*z2) - dPj*(x55 + x64*x69 - Bc*z2);
  o.fIII = x71*x74 + x87*x88 + x90*x91 - x85*z - x90*x92;
  o.dIII[0] = x93*(x38 + x38*x78);
  o.dIII[1] = (-x92*x96) - e1*x62*x94 - x103*x75*(e1*e1) + U*e1*x62*x87 + iU*x84*x96*z2;
  o.dIII[2] = x105*x92 - e2*x104 - x105*x91 + e2*x31*x94 + x77*(e2*e2)*((-x104) - x33*x91 + x31*x84*z + x33*x87*z);
  o.dIII[3] = x74 + e1*x101 + x106*x95 - e1*x99 - x102*x95;
  o.dIII[4] = x76*(x98 - x107 + e1*x103);
  o.dIII[5] = (-x74) - e2*x108 - x106*x89 + e2*x100*x45*z + e2*x31*x97*z;
  o.dIII[6] = x78*(x107 - x98 - e2*(x108 + x47*x97 - x102*x45 - x31*x98));
  o.dIII[7] = x110*(x43 + x43*x83);
  o.dIII[8] = (-x125) - x118*(ec1*ec1) - x120*x122 + x120*x123*z;
  o.dIII[9] = x109*x126 - ec2*x127 - x126*x88 + x82*(ec2*ec2)*((-x127) - x30*x88 + x30*x90*z + x34*x79*z) + ec2*x34*x79*z;
  o.dIII[10] = x125 + x128 - x119*x129 + ec1*x121*x66;
  o.dIII[11] = ec1*(ec1*x118 + x124*x80 - x123*x51*x80);
  o.dIII[12] = (-x128) - ec2*x130 - ec2*x131 + ec2*x121*x34*z + ec2*x123*x39*z;
  o.dIII[13] = x83*((-x124) - ec2*(x130 + x131 - x124*x34 - x129*x39) + iU*x123*z2);
  o.dIII[14] = x100*x121 - x123*x48*x97;
  o.dIII[15] = (-x85) + x71*x73 - x87*x90 - P0*x132*x136 - Pc0*x133*x137 - x11*x134*x90 - x135*x16*x87 + P0*x132*x84*z + Pc0*x133*x79*z + Pcj*U*x134*x79 + (T(2.0)*(iU*x84*x90*z)) + Pj*iU*x135*x84*z2;
  o.tIII = dQcj*x110*(x20 + x20*x83) + dQj*x93*(x25 + x25*x78) + dP0*x132*z*((-x136) + x84*z) + dPc0*x133*z*((-x137) + x79*z) - dPcj*z*(x122 - x129)*(ec1*x113 + ec2*x82) - dPj*z*(x106 - x102)*(x116 - x111);
}

// What one path's step needs besides its point: computed by the path's own warp, read by
// the slices below. Side 0 holds a quantity's plain form, side 1 its conjugate partner.
//   sa: pz, fp, hp, bd, ebd, cg, ecg, v, ac   (the same for every group)
//   sb: pjz, ap, bp, qa, aq, eaq, w   (per group j)
//   pz   = P0*z
//   fp   = F - pz0
//   hp   = H - pz0
//   bd   = B - D
//   ebd  = e1*bd0
//   cg   = C - G
//   ecg  = e2*cg0
//   v    = fp0*ebd0 - hp0*ecg0
//   ac   = A - C
//   pjz  = Pj*z
//   ap   = A - pjz0
//   bp   = B - pjz0
//   qa   = Qj*ac0
//   aq   = ap0 - qa0
//   eaq  = e2*aq0
//   w    = B - A + qa0 + bp0*ebd0 - cg0*eaq0; for the residual alone B + qa0 - A + bp0*ebd0 - ecg0*aq0
#define FRG_IN_PZ 0
#define FRG_IN_FP 1
#define FRG_IN_HP 2
#define FRG_IN_BD 3
#define FRG_IN_EBD 4
#define FRG_IN_CG 5
#define FRG_IN_ECG 6
#define FRG_IN_V 7
#define FRG_IN_AC 8
#define FRG_IN_PJZ 0
#define FRG_IN_AP 1
#define FRG_IN_BP 2
#define FRG_IN_QA 3
#define FRG_IN_AQ 4
#define FRG_IN_EAQ 5
#define FRG_IN_W 6
template <typename T>
struct FrgEvalIn {
  cx<T> z2, z3, e[4], q[32], iU[8];  // e: e1, e2, ec1, ec2; q(t); 1 / U_j at [j - 1]
  cx<T> sa[2][9], sb[2][7][8];
};

// One quarter of group j's evaluation (frg_group_eval's operations in its order): rows of
// the group into M[(row * 18 + column) * 8 + g], columns 0..13 links, 14 Z0, 15 t, 16 U_j, 17 F.
// CX: cx<T>, or a type with its operators whose values several lanes share.
template <int SLICE, typename CX, typename T>
__device__ __forceinline__ void frg_eval_slice(const cx<T>* Y, const FrgEvalIn<T>& in, const cx<T>* dq, int j,
                                               int g, cx<T>* M) {
  if constexpr (SLICE == 0) {
    const CX C(Y[2]);
    const CX D(Y[3]);
    const CX Dc(Y[10]);
    const CX G(Y[5]);
    const CX Gc(Y[12]);
    const CX P0(in.q[0]);
    const CX Pc0(in.q[8]);
    const CX Pcj(in.q[8 + j]);
    const CX Pj(in.q[j]);
    const CX Qj(in.q[15 + j]);
    const CX U(Y[13 + j]);
    const CX e1(in.e[0]);
    const CX e2(in.e[1]);
    const CX iU(in.iU[j - 1]);
    const CX x11(in.sb[1][FRG_IN_PJZ][j - 1]);
    const CX x16(in.sb[0][FRG_IN_PJZ][j - 1]);
    const CX x31(in.sa[0][FRG_IN_HP]);
    const CX x33(in.sb[0][FRG_IN_AQ][j - 1]);
    const CX x45(in.sb[0][FRG_IN_AQ][j - 1]);
    const CX x6(in.sa[0][FRG_IN_PZ]);
    const CX x62(in.sa[0][FRG_IN_FP]);
    const CX x63(in.sb[0][FRG_IN_BP][j - 1]);
    const CX x75(in.sa[0][FRG_IN_BD]);
    const CX x76(in.sa[0][FRG_IN_EBD]);
    const CX x77(in.sa[0][FRG_IN_CG]);
    const CX x78(in.sa[0][FRG_IN_ECG]);
    const CX x79(in.sa[0][FRG_IN_V]);
    const CX x81(in.sa[1][FRG_IN_EBD]);
    const CX x83(in.sa[1][FRG_IN_ECG]);
    const CX x84(in.sa[1][FRG_IN_V]);
    const CX x87(in.sb[1][FRG_IN_W][j - 1]);
    const CX x89(in.sb[0][FRG_IN_EAQ][j - 1]);
    const CX x90(in.sb[0][FRG_IN_W][j - 1]);
    const CX z(Y[21]);
    const CX z2(in.z2);
    const CX x7 = (-(x6));
    const CX x8 = C + x7;
    const CX x32 = U*x31;
    const CX x46 = iU*x45;
    const CX x47 = x46*z2;
    const CX x51 = iU*z2;
    const CX x67 = U*x62;
    const CX x68 = x51*x63;
    const CX x70 = (-(G));
    const CX x71 = D + x70;
    const CX x72 = (-(Gc));
    const CX x73 = Dc + x72;
    const CX x74 = x73*z;
    const CX x85 = x79*x84;
    const CX x91 = x51*x84;
    const CX x92 = x87*z;
    const CX x94 = x84*z;
    const CX x95 = e1*x63;
    const CX x96 = CX(T(1.0)) + x76 + x95;
    const CX x97 = (-(x84));
    const CX x98 = x97*z;
    const CX x99 = x62*x98;
    const CX x100 = (-(x87));
    const CX x101 = x100*x67;
    const CX x102 = x100*z;
    const CX x103 = x101 - x99 + x68*x97 - x102*x63;
    const CX x104 = x32*x87;
    const CX x105 = Qj + x89 + Qj*x78;
    const CX x106 = x51*x97;
    const CX x107 = U*x100;
    const CX x108 = x100*x32;
    const CX x132 = x76 - x78;
    const CX x133 = x81 - x83;
    const CX x134 = (-(x133));
    const CX x135 = (-(x132));
    const CX x136 = U*x87;
    const CX x137 = x51*x90;
    cx_put(M + 104 + g, x47 - x8*z);
    cx_put(M + 296 + g, (-x92*x96) - e1*x62*x94 - x103*x75*(e1*e1) + U*e1*x62*x87 + iU*x84*x96*z2);
    cx_put(M + 304 + g, x105*x92 - e2*x104 - x105*x91 + e2*x31*x94 + x77*(e2*e2)*((-x104) - x33*x91 + x31*x84*z + x33*x87*z));
    cx_put(M + 312 + g, x74 + e1*x101 + x106*x95 - e1*x99 - x102*x95);
    cx_put(M + 320 + g, x76*(x98 - x107 + e1*x103));
    cx_put(M + 328 + g, (-x74) - e2*x108 - x106*x89 + e2*x100*x45*z + e2*x31*x97*z);
    cx_put(M + 336 + g, x78*(x107 - x98 - e2*(x108 + x47*x97 - x102*x45 - x31*x98)));
    cx_put(M + 400 + g, (-x85) + x71*x73 - x87*x90 - P0*x132*x136 - Pc0*x133*x137 - x11*x134*x90 - x135*x16*x87 + P0*x132*x84*z + Pc0*x133*x79*z + Pcj*U*x134*x79 + (T(2.0)*(iU*x84*x90*z)) + Pj*iU*x135*x84*z2);
  }
  if constexpr (SLICE == 1) {
    const CX A(Y[0]);
    const CX Ac(Y[7]);
    const CX B(Y[1]);
    const CX Bc(Y[8]);
    const CX C(Y[2]);
    const CX Cc(Y[9]);
    const CX F(Y[4]);
    const CX Fc(Y[11]);
    const CX H(Y[6]);
    const CX Hc(Y[13]);
    const CX P0(in.q[0]);
    const CX Pc0(in.q[8]);
    const CX Pcj(in.q[8 + j]);
    const CX Pj(in.q[j]);
    const CX Qj(in.q[15 + j]);
    const CX U(Y[13 + j]);
    const CX dP0(dq[0]);
    const CX dPc0(dq[8]);
    const CX dPcj(dq[8 + j]);
    const CX dPj(dq[j]);
    const CX dQcj(dq[22 + j]);
    const CX dQj(dq[15 + j]);
    const CX iU(in.iU[j - 1]);
    const CX x11(in.sb[1][FRG_IN_PJZ][j - 1]);
    const CX x16(in.sb[0][FRG_IN_PJZ][j - 1]);
    const CX x2(in.sa[1][FRG_IN_PZ]);
    const CX x20(in.sa[1][FRG_IN_AC]);
    const CX x21(in.sb[1][FRG_IN_QA][j - 1]);
    const CX x23(in.sb[0][FRG_IN_AP][j - 1]);
    const CX x25(in.sa[0][FRG_IN_AC]);
    const CX x26(in.sb[0][FRG_IN_QA][j - 1]);
    const CX x28(in.sb[1][FRG_IN_AP][j - 1]);
    const CX x30(in.sb[1][FRG_IN_AQ][j - 1]);
    const CX x31(in.sa[0][FRG_IN_HP]);
    const CX x33(in.sb[0][FRG_IN_AQ][j - 1]);
    const CX x34(in.sa[1][FRG_IN_HP]);
    const CX x39(in.sb[1][FRG_IN_AQ][j - 1]);
    const CX x45(in.sb[0][FRG_IN_AQ][j - 1]);
    const CX x6(in.sa[0][FRG_IN_PZ]);
    const CX x61(in.sb[1][FRG_IN_BP][j - 1]);
    const CX x62(in.sa[0][FRG_IN_FP]);
    const CX x63(in.sb[0][FRG_IN_BP][j - 1]);
    const CX x64(in.sa[1][FRG_IN_FP]);
    const CX x79(in.sa[0][FRG_IN_V]);
    const CX x84(in.sa[1][FRG_IN_V]);
    const CX x87(in.sb[1][FRG_IN_W][j - 1]);
    const CX x90(in.sb[0][FRG_IN_W][j - 1]);
    const CX z(Y[21]);
    const CX z2(in.z2);
    const CX z3(in.z3);
    const CX x0 = P0*Pc0 + Pcj*Pj;
    const CX x1 = x0*z3;
    const CX x3 = (-(x2));
    const CX x4 = Cc + x3;
    const CX x5 = x4*z;
    const CX x7 = (-(x6));
    const CX x8 = C + x7;
    const CX x9 = Hc*z;
    const CX x10 = (-(Ac));
    const CX x12 = x10 + x11;
    const CX x13 = Cc + x12;
    const CX x14 = x13*z;
    const CX x15 = (-(A));
    const CX x17 = x15 + x16;
    const CX x18 = C + x17;
    const CX x19 = Ac*z;
    const CX x24 = x23*z;
    const CX x29 = x28*z;
    const CX x32 = U*x31;
    const CX x35 = iU*x34;
    const CX x36 = x35*z2;
    const CX x37 = Qj*x29;
    const CX x38 = (-CX(T(1.0))) + Qj;
    const CX x40 = U*x39;
    const CX x46 = iU*x45;
    const CX x48 = z2*(iU*iU);
    const CX x51 = iU*z2;
    const CX x52 = Pc0*z3;
    const CX x53 = P0*z3;
    const CX x54 = Pj*z3;
    const CX x55 = Pcj*z3;
    const CX x56 = Bc + x3;
    const CX x57 = x56*z;
    const CX x58 = B + x7;
    const CX x59 = Fc*z;
    const CX x60 = B*Pcj + Bc*Pj;
    const CX x65 = x51*x64;
    const CX x66 = U*x61;
    const CX x67 = U*x62;
    const CX x69 = iU*z3;
    const CX x97 = (-(x84));
    const CX x100 = (-(x87));
    const CX x121 = (-(x79));
    const CX x123 = (-(x90));
    cx_put(M + 136 + g, (-x1) + A*x14 + x18*x19 + x21*x24 + x26*x29 + x30*x32 + x33*x36 - H*x5 - x8*x9);
    cx_put(M + 0 + g, x14 + x37 - x19 + x21*z - x36*x38);
    cx_put(M + 16 + g, x19 - x37 - x9 + Qj*x36);
    cx_put(M + 48 + g, x40 - x5);
    cx_put(M + 128 + g, x31*x39 - x34*x45*x48);
    cx_put(M + 120 + g, (-dP0*(x52 + x40*z - Hc*z2)) - dPc0*(x53 + x46*z3 - H*z2) - dPcj*(x54 + x26*z2 + x32*z - A*z2) - dPj*(x55 + x21*z2 + x35*z3 - Ac*z2) - dQcj*x20*(x32 - x24) - dQj*x25*(x36 - x29));
    cx_put(M + 280 + g, (-x1) + x60*z2 - F*x57 - x58*x59 + U*x61*x62 + iU*x63*x64*z2);
    cx_put(M + 152 + g, x65 - x59 + Pcj*z2);
    cx_put(M + 176 + g, x66 - x57);
    cx_put(M + 272 + g, x61*x62 - x48*x63*x64);
    cx_put(M + 264 + g, (-dP0*(x52 + x66*z - Fc*z2)) - dPc0*(x53 + x63*x69 - F*z2) - dPcj*(x54 + x67*z - B*z2) - dPj*(x55 + x64*x69 - Bc*z2));
    cx_put(M + 416 + g, x100*x121 - x123*x48*x97);
  }
  if constexpr (SLICE == 2) {
    const CX A(Y[0]);
    const CX B(Y[1]);
    const CX D(Y[3]);
    const CX Dc(Y[10]);
    const CX G(Y[5]);
    const CX Gc(Y[12]);
    const CX Qcj(in.q[22 + j]);
    const CX Qj(in.q[15 + j]);
    const CX U(Y[13 + j]);
    const CX dP0(dq[0]);
    const CX dPc0(dq[8]);
    const CX dPcj(dq[8 + j]);
    const CX dPj(dq[j]);
    const CX dQcj(dq[22 + j]);
    const CX dQj(dq[15 + j]);
    const CX e1(in.e[0]);
    const CX e2(in.e[1]);
    const CX ec1(in.e[2]);
    const CX ec2(in.e[3]);
    const CX iU(in.iU[j - 1]);
    const CX x20(in.sa[1][FRG_IN_AC]);
    const CX x25(in.sa[0][FRG_IN_AC]);
    const CX x30(in.sb[1][FRG_IN_AQ][j - 1]);
    const CX x31(in.sa[0][FRG_IN_HP]);
    const CX x34(in.sa[1][FRG_IN_HP]);
    const CX x45(in.sb[0][FRG_IN_AQ][j - 1]);
    const CX x61(in.sb[1][FRG_IN_BP][j - 1]);
    const CX x62(in.sa[0][FRG_IN_FP]);
    const CX x63(in.sb[0][FRG_IN_BP][j - 1]);
    const CX x64(in.sa[1][FRG_IN_FP]);
    const CX x75(in.sa[0][FRG_IN_BD]);
    const CX x76(in.sa[0][FRG_IN_EBD]);
    const CX x77(in.sa[0][FRG_IN_CG]);
    const CX x78(in.sa[0][FRG_IN_ECG]);
    const CX x79(in.sa[0][FRG_IN_V]);
    const CX x80(in.sa[1][FRG_IN_BD]);
    const CX x81(in.sa[1][FRG_IN_EBD]);
    const CX x82(in.sa[1][FRG_IN_CG]);
    const CX x83(in.sa[1][FRG_IN_ECG]);
    const CX x84(in.sa[1][FRG_IN_V]);
    const CX x86(in.sb[1][FRG_IN_EAQ][j - 1]);
    const CX x87(in.sb[1][FRG_IN_W][j - 1]);
    const CX x90(in.sb[0][FRG_IN_W][j - 1]);
    const CX z(Y[21]);
    const CX z2(in.z2);
    const CX x35 = iU*x34;
    const CX x36 = x35*z2;
    const CX x38 = (-CX(T(1.0))) + Qj;
    const CX x43 = (-CX(T(1.0))) + Qcj;
    const CX x44 = (-(Qj*x25));
    const CX x51 = iU*z2;
    const CX x65 = x51*x64;
    const CX x70 = (-(G));
    const CX x71 = D + x70;
    const CX x72 = (-(Gc));
    const CX x73 = Dc + x72;
    const CX x74 = x73*z;
    const CX x85 = x79*x84;
    const CX x88 = U*x79;
    const CX x91 = x51*x84;
    const CX x92 = x87*z;
    const CX x93 = x91 - x92;
    const CX x97 = (-(x84));
    const CX x100 = (-(x87));
    const CX x102 = x100*z;
    const CX x106 = x51*x97;
    const CX x109 = x90*z;
    const CX x110 = x88 - x109;
    const CX x111 = (-(e2*x77));
    const CX x112 = (-x111*x31) - x62*x76;
    const CX x113 = (-(x80));
    const CX x114 = (-(x113*x61));
    const CX x115 = (-(x64*x80));
    const CX x116 = (-(e1*x75));
    const CX x117 = A + x44 - B + x116*x63 - x111*x45;
    const CX x118 = U*x112*x114 + x112*x115*z - x114*x117*z - x115*x117*x51;
    const CX x119 = ec1*x61;
    const CX x120 = CX(T(1.0)) + x119 + x81;
    const CX x121 = (-(x79));
    const CX x122 = U*x121;
    const CX x123 = (-(x90));
    const CX x124 = x121*z;
    const CX x125 = ec1*x123*x65 - ec1*x124*x64;
    const CX x126 = Qcj + x86 + Qcj*x83;
    const CX x127 = x36*x90;
    const CX x129 = x123*z;
    const CX x132 = x76 - x78;
    const CX x133 = x81 - x83;
    const CX x136 = U*x87;
    const CX x137 = x51*x90;
    cx_put(M + 424 + g, x71*x74 + x87*x88 + x90*x91 - x85*z - x90*x92);
    cx_put(M + 288 + g, x93*(x38 + x38*x78));
    cx_put(M + 344 + g, x110*(x43 + x43*x83));
    cx_put(M + 352 + g, (-x125) - x118*(ec1*ec1) - x120*x122 + x120*x123*z);
    cx_put(M + 360 + g, x109*x126 - ec2*x127 - x126*x88 + x82*(ec2*ec2)*((-x127) - x30*x88 + x30*x90*z + x34*x79*z) + ec2*x34*x79*z);
    cx_put(M + 376 + g, ec1*(ec1*x118 + x124*x80 - x123*x51*x80));
    cx_put(M + 408 + g, dQcj*x110*(x20 + x20*x83) + dQj*x93*(x25 + x25*x78) + dP0*x132*z*((-x136) + x84*z) + dPc0*x133*z*((-x137) + x79*z) - dPcj*z*(x122 - x129)*(ec1*x113 + ec2*x82) - dPj*z*(x106 - x102)*(x116 - x111));
  }
  if constexpr (SLICE == 3) {
    const CX A(Y[0]);
    const CX Ac(Y[7]);
    const CX B(Y[1]);
    const CX Bc(Y[8]);
    const CX C(Y[2]);
    const CX Cc(Y[9]);
    const CX D(Y[3]);
    const CX F(Y[4]);
    const CX Fc(Y[11]);
    const CX G(Y[5]);
    const CX H(Y[6]);
    const CX Hc(Y[13]);
    const CX P0(in.q[0]);
    const CX Pc0(in.q[8]);
    const CX Pcj(in.q[8 + j]);
    const CX Pj(in.q[j]);
    const CX Qcj(in.q[22 + j]);
    const CX U(Y[13 + j]);
    const CX ec1(in.e[2]);
    const CX ec2(in.e[3]);
    const CX iU(in.iU[j - 1]);
    const CX x11(in.sb[1][FRG_IN_PJZ][j - 1]);
    const CX x16(in.sb[0][FRG_IN_PJZ][j - 1]);
    const CX x2(in.sa[1][FRG_IN_PZ]);
    const CX x21(in.sb[1][FRG_IN_QA][j - 1]);
    const CX x23(in.sb[0][FRG_IN_AP][j - 1]);
    const CX x26(in.sb[0][FRG_IN_QA][j - 1]);
    const CX x28(in.sb[1][FRG_IN_AP][j - 1]);
    const CX x30(in.sb[1][FRG_IN_AQ][j - 1]);
    const CX x31(in.sa[0][FRG_IN_HP]);
    const CX x33(in.sb[0][FRG_IN_AQ][j - 1]);
    const CX x34(in.sa[1][FRG_IN_HP]);
    const CX x39(in.sb[1][FRG_IN_AQ][j - 1]);
    const CX x6(in.sa[0][FRG_IN_PZ]);
    const CX x61(in.sb[1][FRG_IN_BP][j - 1]);
    const CX x62(in.sa[0][FRG_IN_FP]);
    const CX x63(in.sb[0][FRG_IN_BP][j - 1]);
    const CX x64(in.sa[1][FRG_IN_FP]);
    const CX x79(in.sa[0][FRG_IN_V]);
    const CX x83(in.sa[1][FRG_IN_ECG]);
    const CX x90(in.sb[0][FRG_IN_W][j - 1]);
    const CX z(Y[21]);
    const CX z2(in.z2);
    const CX x0 = P0*Pc0 + Pcj*Pj;
    const CX x3 = (-(x2));
    const CX x4 = Cc + x3;
    const CX x7 = (-(x6));
    const CX x8 = C + x7;
    const CX x10 = (-(Ac));
    const CX x12 = x10 + x11;
    const CX x13 = Cc + x12;
    const CX x15 = (-(A));
    const CX x17 = x15 + x16;
    const CX x18 = C + x17;
    const CX x24 = x23*z;
    const CX x32 = U*x31;
    const CX x35 = iU*x34;
    const CX x36 = x35*z2;
    const CX x40 = U*x39;
    const CX x41 = A*z;
    const CX x42 = Qcj*x24;
    const CX x43 = (-CX(T(1.0))) + Qcj;
    const auto x49 = (T(3.0)*(x0*z2));
    const CX x50 = Pj*z2;
    const CX x51 = iU*z2;
    const CX x56 = Bc + x3;
    const CX x58 = B + x7;
    const CX x60 = B*Pcj + Bc*Pj;
    const CX x65 = x51*x64;
    const CX x66 = U*x61;
    const CX x67 = U*x62;
    const CX x68 = x51*x63;
    const CX x70 = (-(G));
    const CX x71 = D + x70;
    const CX x119 = ec1*x61;
    const CX x121 = (-(x79));
    const CX x123 = (-(x90));
    const CX x124 = x121*z;
    const CX x125 = ec1*x123*x65 - ec1*x124*x64;
    const CX x128 = x71*z;
    const CX x129 = x123*z;
    const CX x130 = x121*x40;
    const CX x131 = x123*x36;
    cx_put(M + 56 + g, x42 - x41 + x18*z + x26*z - x32*x43);
    cx_put(M + 72 + g, x41 - x42 + Qcj*x32 - H*z);
    cx_put(M + 112 + g, (-x49) + A*x11 + A*x13 + Ac*x16 + Ac*x18 + H*x2 + Hc*x6 + x21*x23 + x26*x28 - H*x4 - Hc*x8 - Pcj*x32 - x11*x26 - x16*x21 - x35*x50 - P0*U*x30 - Pc0*x33*x51 + (T(2.0)*(x33*x35*z)));
    cx_put(M + 208 + g, x50 + x67 - F*z);
    cx_put(M + 232 + g, x68 - x58*z);
    cx_put(M + 256 + g, (-x49) - F*x56 - Fc*x58 - P0*x66 - Pc0*x68 - Pcj*x67 + (T(2.0)*(x60*z)) + F*Pc0*z + Fc*P0*z - iU*x50*x64 + (T(2.0)*(iU*x63*x64*z)));
    cx_put(M + 368 + g, x125 + x128 - x119*x129 + ec1*x121*x66);
    cx_put(M + 384 + g, (-x128) - ec2*x130 - ec2*x131 + ec2*x121*x34*z + ec2*x123*x39*z);
    cx_put(M + 392 + g, x83*((-x124) - ec2*(x130 + x131 - x124*x34 - x129*x39) + iU*x123*z2));
  }
}

// The three equations at a point alone (their own common subexpressions) as schedules for a
// part's four warps, residual_part in frg_team.cuh executes them. Warp k: steps START[k] ..
// START[k + 1] of 16 words OP(result, a, b, b subtracted, product), values by
// number in Y (the point), IN (FrgEvalIn) and T (temporaries; the last takes idle lanes' results), two steps
// of padding at the end; then OUT(value, equation, group, negated), 7 per warp.
#define FRG_RESIDUAL_TEMPS 208
#define FRG_RESIDUAL_START {0, 17, 34, 51, 64}
#define FRG_RESIDUAL_CODE(OP, Y, IN, T) \
    OP(T(0), IN(18), Y(21), 0, 1), OP(T(1), IN(17), Y(21), 0, 1), OP(T(2), IN(16), Y(21), 0, 1), \
    OP(T(3), IN(15), Y(21), 0, 1), OP(T(4), Y(21), Y(21), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(5), Y(7), T(0), 1, 0), OP(T(6), Y(7), T(1), 1, 0), \
    OP(T(7), Y(7), T(2), 1, 0), OP(T(8), Y(7), T(3), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(2), T(4), Y(21), 0, 1), \
    OP(T(3), IN(10), Y(21), 0, 1), OP(T(9), IN(18), IN(10), 0, 1), OP(T(10), IN(9), Y(21), 0, 1), \
    OP(T(11), IN(17), IN(9), 0, 1), OP(T(12), IN(8), Y(21), 0, 1), OP(T(13), IN(16), IN(8), 0, 1), \
    OP(T(14), IN(14), Y(21), 0, 1), OP(T(15), IN(6), Y(21), 0, 1), OP(T(16), Y(7), Y(21), 0, 1), \
    OP(T(17), IN(7), Y(21), 0, 1), OP(T(18), Y(0), Y(21), 0, 1), OP(T(19), IN(15), IN(7), 0, 1), \
    OP(T(20), IN(6), IN(14), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(21), Y(9), T(5), 1, 0), OP(T(22), Y(9), T(6), 1, 0), OP(T(23), Y(9), T(7), 1, 0), \
    OP(T(24), Y(9), T(8), 1, 0), OP(T(25), Y(0), T(3), 1, 0), OP(T(26), T(20), T(9), 0, 0), \
    OP(T(27), Y(0), T(10), 1, 0), OP(T(28), T(20), T(11), 0, 0), OP(T(29), Y(0), T(12), 1, 0), \
    OP(T(30), T(20), T(13), 0, 0), OP(T(31), Y(6), T(15), 1, 0), OP(T(32), Y(0), T(17), 1, 0), \
    OP(T(33), T(20), T(19), 0, 0), OP(T(34), Y(7), Y(9), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(9), T(18), T(21), 0, 1), OP(T(11), T(18), T(22), 0, 1), \
    OP(T(12), T(18), T(23), 0, 1), OP(T(13), T(18), T(24), 0, 1), OP(T(17), T(2), T(26), 0, 1), \
    OP(T(19), T(2), T(28), 0, 1), OP(T(20), T(2), T(30), 0, 1), OP(T(35), T(2), T(33), 0, 1), \
    OP(T(36), Y(17), T(31), 0, 1), OP(T(37), Y(16), T(31), 0, 1), OP(T(38), Y(15), T(31), 0, 1), \
    OP(T(39), Y(14), T(31), 0, 1), OP(T(40), IN(32), T(34), 0, 1), OP(T(41), IN(31), T(34), 0, 1), \
    OP(T(42), IN(30), T(34), 0, 1), OP(T(43), IN(29), T(34), 0, 1), OP(T(2), T(17), T(9), 1, 0), \
    OP(T(18), T(19), T(11), 1, 0), OP(T(21), T(20), T(12), 1, 0), OP(T(22), T(35), T(13), 1, 0), \
    OP(T(23), T(40), T(5), 1, 0), OP(T(24), Y(2), T(25), 1, 0), OP(T(26), T(41), T(6), 1, 0), \
    OP(T(28), Y(2), T(27), 1, 0), OP(T(30), T(42), T(7), 1, 0), OP(T(31), Y(2), T(29), 1, 0), \
    OP(T(33), T(43), T(8), 1, 0), OP(T(34), Y(2), T(32), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(9), T(36), T(23), 0, 1), OP(T(11), T(37), T(26), 0, 1), OP(T(12), T(38), T(30), 0, 1), \
    OP(T(13), T(39), T(33), 0, 1), OP(T(20), T(16), T(24), 0, 1), OP(T(35), T(16), T(28), 0, 1), \
    OP(T(44), T(16), T(31), 0, 1), OP(T(45), T(16), T(34), 0, 1), OP(T(46), T(25), T(40), 0, 1), \
    OP(T(47), T(27), T(41), 0, 1), OP(T(48), T(29), T(42), 0, 1), OP(T(49), T(32), T(43), 0, 1), \
    OP(T(50), Y(8), IN(10), 0, 1), OP(T(51), Y(1), IN(18), 0, 1), OP(T(52), Y(8), IN(9), 0, 1), \
    OP(T(53), Y(1), IN(17), 0, 1), OP(T(16), T(2), T(20), 1, 0), OP(T(23), T(18), T(35), 1, 0), \
    OP(T(24), T(21), T(44), 1, 0), OP(T(26), T(22), T(45), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(28), T(16), T(9), 0, 0), \
    OP(T(30), T(23), T(11), 0, 0), OP(T(31), T(24), T(12), 0, 0), OP(T(33), T(26), T(13), 0, 0), \
    OP(T(34), Y(1), T(3), 1, 0), OP(T(36), T(51), T(50), 0, 0), OP(T(37), Y(1), T(10), 1, 0), \
    OP(T(38), T(53), T(52), 0, 0), OP(T(39), Y(2), T(15), 1, 0), OP(T(40), Y(9), T(14), 1, 0), \
    OP(T(41), Y(13), T(14), 1, 0), OP(T(42), Y(0), Y(2), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(43), T(46), Y(21), 0, 1), OP(T(2), T(47), Y(21), 0, 1), OP(T(18), T(48), Y(21), 0, 1), \
    OP(T(20), T(49), Y(21), 0, 1), OP(T(21), IN(41), T(34), 0, 1), OP(T(22), T(4), T(36), 0, 1), \
    OP(T(35), IN(40), T(37), 0, 1), OP(T(44), T(4), T(38), 0, 1), OP(T(45), IN(41), T(4), 0, 1), \
    OP(T(3), IN(40), T(4), 0, 1), OP(T(9), IN(39), T(4), 0, 1), OP(T(10), IN(38), T(4), 0, 1), \
    OP(T(11), IN(25), T(42), 0, 1), OP(T(12), IN(24), T(42), 0, 1), OP(T(13), IN(23), T(42), 0, 1), \
    OP(T(16), IN(22), T(42), 0, 1), OP(T(23), T(28), T(43), 1, 0), OP(T(24), T(30), T(2), 1, 0), \
    OP(T(26), T(31), T(18), 1, 0), OP(T(50), T(33), T(20), 1, 0), OP(T(51), T(17), T(22), 1, 0), \
    OP(T(52), T(19), T(44), 1, 0), OP(T(53), T(11), T(25), 1, 0), OP(T(34), T(12), T(27), 1, 0), \
    OP(T(36), T(13), T(29), 1, 0), OP(T(37), T(16), T(32), 1, 0), OP(T(38), Y(8), T(0), 1, 0), \
    OP(T(42), Y(11), T(14), 1, 0), OP(T(46), Y(1), T(15), 1, 0), OP(T(47), Y(8), T(14), 1, 0), \
    OP(T(48), Y(4), T(15), 1, 0), OP(T(49), Y(8), T(1), 1, 0), OP(T(0), T(21), T(42), 0, 1), \
    OP(T(1), T(35), T(42), 0, 1), OP(T(2), T(41), T(45), 0, 1), OP(T(14), T(41), T(3), 0, 1), \
    OP(T(15), T(41), T(9), 0, 1), OP(T(17), T(41), T(10), 0, 1), OP(T(18), Y(17), T(38), 0, 1), \
    OP(T(19), Y(16), T(49), 0, 1), OP(T(20), T(5), T(11), 0, 1), OP(T(22), T(6), T(12), 0, 1), \
    OP(T(25), T(7), T(13), 0, 1), OP(T(27), T(8), T(16), 0, 1), OP(T(28), Y(11), Y(21), 0, 1), \
    OP(T(29), Y(4), Y(21), 0, 1), OP(T(30), Y(13), Y(21), 0, 1), OP(T(31), Y(6), Y(21), 0, 1), \
    OP(T(32), T(0), T(4), 0, 1), OP(T(33), T(1), T(4), 0, 1), OP(T(43), T(2), T(53), 0, 1), \
    OP(T(44), T(14), T(34), 0, 1), OP(T(3), T(15), T(36), 0, 1), OP(T(5), T(17), T(37), 0, 1), \
    OP(T(6), T(18), T(48), 0, 1), OP(T(7), T(19), T(48), 0, 1), OP(T(8), T(20), Y(21), 0, 1), \
    OP(T(9), T(22), Y(21), 0, 1), OP(T(10), T(25), Y(21), 0, 1), OP(T(11), T(27), Y(21), 0, 1), \
    OP(T(12), T(28), T(46), 0, 1), OP(T(13), T(29), T(47), 0, 1), OP(T(16), T(30), T(39), 0, 1), \
    OP(T(21), T(31), T(40), 0, 1), OP(T(35), T(23), T(8), 1, 0), OP(T(38), T(24), T(9), 1, 0), \
    OP(T(41), T(26), T(10), 1, 0), OP(T(42), T(50), T(11), 1, 0), OP(T(45), T(51), T(6), 1, 0), \
    OP(T(49), T(52), T(7), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(0), T(35), T(43), 0, 0), \
    OP(T(1), T(38), T(44), 0, 0), OP(T(2), T(41), T(3), 0, 0), OP(T(4), T(42), T(5), 0, 0), \
    OP(T(14), T(45), T(13), 0, 0), OP(T(15), T(49), T(13), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(17), T(0), T(21), 0, 0), OP(T(18), T(1), T(21), 0, 0), OP(T(19), T(2), T(21), 0, 0), \
    OP(T(20), T(4), T(21), 0, 0), OP(T(22), T(14), T(12), 0, 0), OP(T(25), T(15), T(12), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(27), T(17), T(16), 0, 0), OP(T(28), T(18), T(16), 0, 0), \
    OP(T(29), T(19), T(16), 0, 0), OP(T(30), T(20), T(16), 0, 0), OP(T(31), T(22), T(32), 1, 0), \
    OP(T(34), T(25), T(33), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(54), IN(13), Y(21), 0, 1), \
    OP(T(55), IN(21), Y(21), 0, 1), OP(T(56), IN(12), Y(21), 0, 1), OP(T(57), IN(20), Y(21), 0, 1), \
    OP(T(58), IN(11), Y(21), 0, 1), OP(T(59), IN(19), Y(21), 0, 1), OP(T(60), Y(21), Y(21), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(61), Y(0), T(54), 1, 0), OP(T(62), Y(7), T(55), 1, 0), OP(T(63), Y(0), T(56), 1, 0), \
    OP(T(64), Y(7), T(57), 1, 0), OP(T(65), Y(0), T(58), 1, 0), OP(T(66), Y(7), T(59), 1, 0), \
    OP(T(67), Y(0), Y(2), 1, 0), OP(T(68), Y(7), Y(9), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(54), T(60), Y(21), 0, 1), OP(T(55), IN(34), T(68), 0, 1), \
    OP(T(69), IN(26), T(67), 0, 1), OP(T(70), IN(33), T(68), 0, 1), OP(T(71), IN(21), IN(13), 0, 1), \
    OP(T(72), IN(20), IN(12), 0, 1), OP(T(73), IN(6), Y(21), 0, 1), OP(T(74), Y(7), Y(21), 0, 1), \
    OP(T(75), Y(0), Y(21), 0, 1), OP(T(76), IN(19), IN(11), 0, 1), OP(T(77), IN(6), IN(14), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(78), Y(2), T(61), 1, 0), \
    OP(T(79), Y(9), T(62), 1, 0), OP(T(80), Y(2), T(63), 1, 0), OP(T(81), Y(9), T(64), 1, 0), \
    OP(T(82), Y(2), T(65), 1, 0), OP(T(83), Y(9), T(66), 1, 0), OP(T(84), T(77), T(71), 0, 0), \
    OP(T(85), T(77), T(72), 0, 0), OP(T(86), Y(6), T(73), 1, 0), OP(T(87), T(77), T(76), 0, 0), \
    OP(T(88), Y(8), Y(10), 1, 0), OP(T(89), Y(1), Y(3), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(71), T(74), T(78), 0, 1), OP(T(72), T(75), T(79), 0, 1), OP(T(76), T(74), T(80), 0, 1), \
    OP(T(77), T(75), T(81), 0, 1), OP(T(90), T(74), T(82), 0, 1), OP(T(91), T(75), T(83), 0, 1), \
    OP(T(92), T(54), T(84), 0, 1), OP(T(93), T(54), T(85), 0, 1), OP(T(94), T(54), T(87), 0, 1), \
    OP(T(95), Y(20), T(86), 0, 1), OP(T(96), Y(19), T(86), 0, 1), OP(T(97), Y(18), T(86), 0, 1), \
    OP(T(98), IN(4), T(88), 0, 1), OP(T(99), IN(2), T(89), 0, 1), OP(T(100), IN(35), T(68), 0, 1), \
    OP(T(101), IN(27), T(67), 0, 1), OP(T(54), T(92), T(72), 1, 0), OP(T(68), T(93), T(77), 1, 0), \
    OP(T(74), T(94), T(91), 1, 0), OP(T(75), Y(1), T(101), 0, 0), OP(T(78), Y(8), T(55), 0, 0), \
    OP(T(79), Y(1), T(69), 0, 0), OP(T(80), Y(8), T(70), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(81), T(54), T(71), 1, 0), \
    OP(T(82), T(68), T(76), 1, 0), OP(T(83), T(74), T(90), 1, 0), OP(T(84), T(75), Y(0), 1, 0), \
    OP(T(85), T(78), Y(7), 1, 0), OP(T(87), T(79), Y(0), 1, 0), OP(T(88), T(80), Y(7), 1, 0), \
    OP(T(89), T(100), T(62), 1, 0), OP(T(72), T(55), T(64), 1, 0), OP(T(77), T(70), T(66), 1, 0), \
    OP(T(91), Y(1), T(56), 1, 0), OP(T(92), Y(8), T(57), 1, 0), OP(T(93), Y(1), T(58), 1, 0), \
    OP(T(94), Y(8), T(59), 1, 0), OP(T(102), Y(9), Y(12), 1, 0), OP(T(103), Y(2), Y(5), 1, 0), \
    OP(T(54), T(95), T(89), 0, 1), OP(T(56), T(96), T(72), 0, 1), OP(T(57), T(97), T(77), 0, 1), \
    OP(T(58), T(91), T(99), 0, 1), OP(T(59), T(92), T(98), 0, 1), OP(T(68), T(93), T(99), 0, 1), \
    OP(T(71), T(94), T(98), 0, 1), OP(T(74), T(61), T(100), 0, 1), OP(T(75), T(63), T(55), 0, 1), \
    OP(T(76), T(65), T(70), 0, 1), OP(T(78), IN(5), T(102), 0, 1), OP(T(79), IN(3), T(103), 0, 1), \
    OP(T(80), IN(14), Y(21), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(90), T(81), T(54), 0, 0), OP(T(72), T(82), T(56), 0, 0), \
    OP(T(77), T(83), T(57), 0, 0), OP(T(89), T(84), T(58), 0, 0), OP(T(91), T(85), T(59), 0, 0), \
    OP(T(92), T(87), T(68), 0, 0), OP(T(93), T(88), T(71), 0, 0), OP(T(94), T(63), T(101), 1, 0), \
    OP(T(95), T(64), T(55), 1, 0), OP(T(96), T(65), T(69), 1, 0), OP(T(97), T(66), T(70), 1, 0), \
    OP(T(100), Y(11), T(80), 1, 0), OP(T(102), Y(4), T(73), 1, 0), OP(T(103), Y(13), T(80), 1, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(54), T(74), Y(21), 0, 1), \
    OP(T(55), T(75), Y(21), 0, 1), OP(T(56), T(76), Y(21), 0, 1), OP(T(57), T(79), T(94), 0, 1), \
    OP(T(58), T(78), T(95), 0, 1), OP(T(59), T(79), T(96), 0, 1), OP(T(68), T(78), T(97), 0, 1), \
    OP(T(70), T(103), T(78), 0, 1), OP(T(71), T(100), T(98), 0, 1), OP(T(81), T(86), T(79), 0, 1), \
    OP(T(82), T(102), T(99), 0, 1), OP(T(83), IN(44), T(60), 0, 1), OP(T(84), IN(43), T(60), 0, 1), \
    OP(T(85), IN(42), T(60), 0, 1), OP(T(87), IN(28), T(67), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(88), T(90), T(54), 1, 0), OP(T(60), T(72), T(55), 1, 0), OP(T(67), T(77), T(56), 1, 0), \
    OP(T(74), T(89), T(57), 1, 0), OP(T(75), T(91), T(58), 1, 0), OP(T(76), T(92), T(59), 1, 0), \
    OP(T(78), T(93), T(68), 1, 0), OP(T(79), T(71), T(70), 1, 0), OP(T(86), T(82), T(81), 1, 0), \
    OP(T(94), T(87), T(61), 1, 0), OP(T(95), T(101), T(63), 1, 0), OP(T(96), T(69), T(65), 1, 0), \
    OP(T(97), Y(2), T(73), 1, 0), OP(T(98), Y(9), T(80), 1, 0), OP(T(99), Y(10), Y(12), 1, 0), \
    OP(T(100), Y(3), Y(5), 1, 0), OP(T(102), T(75), T(74), 0, 1), OP(T(54), T(78), T(76), 0, 1), \
    OP(T(55), T(84), T(79), 0, 1), OP(T(56), Y(19), T(86), 0, 1), OP(T(57), T(86), T(79), 0, 1), \
    OP(T(58), T(85), T(79), 0, 1), OP(T(59), Y(18), T(86), 0, 1), OP(T(61), T(103), T(83), 0, 1), \
    OP(T(63), T(103), T(84), 0, 1), OP(T(65), T(103), T(85), 0, 1), OP(T(68), T(62), T(87), 0, 1), \
    OP(T(70), T(64), T(101), 0, 1), OP(T(71), T(66), T(69), 0, 1), OP(T(72), Y(21), T(100), 0, 1), \
    OP(T(73), Y(13), Y(21), 0, 1), OP(T(77), Y(6), Y(21), 0, 1), OP(T(80), T(102), Y(21), 0, 1), \
    OP(T(81), T(54), Y(21), 0, 1), OP(T(82), T(55), T(74), 0, 1), OP(T(89), T(56), T(75), 0, 1), \
    OP(T(90), T(57), Y(21), 0, 1), OP(T(91), T(58), T(76), 0, 1), OP(T(92), T(59), T(78), 0, 1), \
    OP(T(93), T(61), T(94), 0, 1), OP(T(62), T(63), T(95), 0, 1), OP(T(64), T(65), T(96), 0, 1), \
    OP(T(66), T(68), Y(21), 0, 1), OP(T(69), T(70), Y(21), 0, 1), OP(T(79), T(71), Y(21), 0, 1), \
    OP(T(83), T(72), T(99), 0, 1), OP(T(84), T(73), T(97), 0, 1), OP(T(85), T(77), T(98), 0, 1), \
    OP(T(86), T(88), T(66), 1, 0), OP(T(87), T(60), T(69), 1, 0), OP(T(100), T(67), T(79), 1, 0), \
    OP(T(101), T(89), T(82), 0, 0), OP(T(103), T(92), T(91), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(54), T(86), T(93), 0, 0), OP(T(55), T(87), T(62), 0, 0), \
    OP(T(56), T(100), T(64), 0, 0), OP(T(57), T(101), T(83), 0, 0), OP(T(58), T(103), T(83), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(59), T(54), T(85), 0, 0), \
    OP(T(61), T(55), T(85), 0, 0), OP(T(63), T(56), T(85), 0, 0), OP(T(65), T(57), T(90), 1, 0), \
    OP(T(68), T(58), T(90), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(70), T(59), T(84), 0, 0), OP(T(71), T(61), T(84), 0, 0), OP(T(72), T(63), T(84), 0, 0), \
    OP(T(73), T(65), T(80), 1, 0), OP(T(74), T(68), T(81), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(104), Y(0), Y(2), 1, 0), OP(T(105), Y(9), Y(12), 1, 0), \
    OP(T(106), Y(8), Y(10), 1, 0), OP(T(107), Y(7), Y(9), 1, 0), OP(T(108), Y(2), Y(5), 1, 0), \
    OP(T(109), Y(1), Y(3), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(110), IN(9), Y(21), 0, 1), \
    OP(T(111), IN(17), Y(21), 0, 1), OP(T(112), IN(8), Y(21), 0, 1), OP(T(113), IN(16), Y(21), 0, 1), \
    OP(T(114), IN(7), Y(21), 0, 1), OP(T(115), IN(14), Y(21), 0, 1), OP(T(116), Y(21), Y(21), 0, 1), \
    OP(T(117), IN(15), Y(21), 0, 1), OP(T(118), IN(6), Y(21), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(119), Y(0), T(110), 1, 0), OP(T(120), Y(1), T(110), 1, 0), OP(T(121), Y(7), T(111), 1, 0), \
    OP(T(122), Y(8), T(111), 1, 0), OP(T(123), Y(0), T(112), 1, 0), OP(T(124), Y(1), T(112), 1, 0), \
    OP(T(125), Y(7), T(113), 1, 0), OP(T(126), Y(8), T(113), 1, 0), OP(T(127), Y(0), T(114), 1, 0), \
    OP(T(128), Y(1), T(114), 1, 0), OP(T(129), Y(13), T(115), 1, 0), OP(T(130), Y(11), T(115), 1, 0), \
    OP(T(131), Y(7), T(117), 1, 0), OP(T(132), Y(8), T(117), 1, 0), OP(T(133), Y(6), T(118), 1, 0), \
    OP(T(134), Y(4), T(118), 1, 0), OP(T(110), IN(28), T(104), 0, 1), OP(T(111), IN(35), T(107), 0, 1), \
    OP(T(112), IN(25), T(104), 0, 1), OP(T(113), IN(32), T(107), 0, 1), OP(T(114), IN(24), T(104), 0, 1), \
    OP(T(115), IN(31), T(107), 0, 1), OP(T(117), IN(23), T(104), 0, 1), OP(T(118), IN(30), T(107), 0, 1), \
    OP(T(135), IN(22), T(104), 0, 1), OP(T(136), IN(4), T(106), 0, 1), OP(T(137), IN(29), T(107), 0, 1), \
    OP(T(138), IN(2), T(109), 0, 1), OP(T(139), IN(13), Y(21), 0, 1), OP(T(140), IN(21), Y(21), 0, 1), \
    OP(T(141), IN(10), Y(21), 0, 1), OP(T(142), IN(18), Y(21), 0, 1), OP(T(104), Y(1), T(110), 0, 0), \
    OP(T(106), Y(8), T(111), 0, 0), OP(T(107), Y(1), T(112), 0, 0), OP(T(109), Y(8), T(113), 0, 0), \
    OP(T(143), Y(1), T(114), 0, 0), OP(T(144), Y(8), T(115), 0, 0), OP(T(145), Y(1), T(117), 0, 0), \
    OP(T(146), Y(8), T(118), 0, 0), OP(T(147), Y(1), T(135), 0, 0), OP(T(148), Y(8), T(137), 0, 0), \
    OP(T(149), Y(7), T(140), 1, 0), OP(T(150), Y(8), T(140), 1, 0), OP(T(151), Y(0), T(141), 1, 0), \
    OP(T(152), Y(1), T(141), 1, 0), OP(T(153), Y(7), T(142), 1, 0), OP(T(154), Y(8), T(142), 1, 0), \
    OP(T(140), T(104), Y(0), 1, 0), OP(T(141), T(106), Y(7), 1, 0), OP(T(142), T(107), Y(0), 1, 0), \
    OP(T(155), T(109), Y(7), 1, 0), OP(T(156), T(143), Y(0), 1, 0), OP(T(157), T(144), Y(7), 1, 0), \
    OP(T(158), T(145), Y(0), 1, 0), OP(T(159), T(146), Y(7), 1, 0), OP(T(160), T(147), Y(0), 1, 0), \
    OP(T(161), T(148), Y(7), 1, 0), OP(T(162), T(123), T(117), 1, 0), OP(T(163), T(125), T(118), 1, 0), \
    OP(T(164), T(127), T(135), 1, 0), OP(T(165), T(131), T(137), 1, 0), OP(T(166), Y(0), T(139), 1, 0), \
    OP(T(167), Y(1), T(139), 1, 0), OP(T(104), T(167), T(138), 0, 1), OP(T(106), T(150), T(136), 0, 1), \
    OP(T(107), T(152), T(138), 0, 1), OP(T(109), T(154), T(136), 0, 1), OP(T(117), T(120), T(138), 0, 1), \
    OP(T(118), T(122), T(136), 0, 1), OP(T(123), T(124), T(138), 0, 1), OP(T(125), T(126), T(136), 0, 1), \
    OP(T(127), T(128), T(138), 0, 1), OP(T(131), T(132), T(136), 0, 1), OP(T(135), IN(40), T(116), 0, 1), \
    OP(T(137), IN(39), T(116), 0, 1), OP(T(139), IN(38), T(116), 0, 1), OP(T(143), IN(5), T(105), 0, 1), \
    OP(T(144), IN(3), T(108), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(145), T(140), T(104), 0, 0), \
    OP(T(146), T(141), T(106), 0, 0), OP(T(147), T(142), T(107), 0, 0), OP(T(148), T(155), T(109), 0, 0), \
    OP(T(105), T(156), T(117), 0, 0), OP(T(108), T(157), T(118), 0, 0), OP(T(120), T(158), T(123), 0, 0), \
    OP(T(122), T(159), T(125), 0, 0), OP(T(124), T(160), T(127), 0, 0), OP(T(126), T(161), T(131), 0, 0), \
    OP(T(128), T(166), T(110), 1, 0), OP(T(132), T(149), T(111), 1, 0), OP(T(150), T(151), T(112), 1, 0), \
    OP(T(152), T(153), T(113), 1, 0), OP(T(154), T(119), T(114), 1, 0), OP(T(167), T(121), T(115), 1, 0), \
    OP(T(104), T(144), T(128), 0, 1), OP(T(106), T(143), T(132), 0, 1), OP(T(107), T(144), T(150), 0, 1), \
    OP(T(109), T(143), T(152), 0, 1), OP(T(110), T(144), T(154), 0, 1), OP(T(111), T(143), T(167), 0, 1), \
    OP(T(112), T(144), T(162), 0, 1), OP(T(113), T(143), T(163), 0, 1), OP(T(114), T(144), T(164), 0, 1), \
    OP(T(115), T(143), T(165), 0, 1), OP(T(117), T(129), T(143), 0, 1), OP(T(118), T(130), T(136), 0, 1), \
    OP(T(119), T(133), T(144), 0, 1), OP(T(121), T(134), T(138), 0, 1), OP(T(123), IN(44), T(116), 0, 1), \
    OP(T(125), IN(41), T(116), 0, 1), OP(T(127), T(145), T(104), 1, 0), OP(T(131), T(146), T(106), 1, 0), \
    OP(T(140), T(147), T(107), 1, 0), OP(T(141), T(148), T(109), 1, 0), OP(T(142), T(105), T(110), 1, 0), \
    OP(T(149), T(108), T(111), 1, 0), OP(T(151), T(120), T(112), 1, 0), OP(T(153), T(122), T(113), 1, 0), \
    OP(T(155), T(124), T(114), 1, 0), OP(T(156), T(126), T(115), 1, 0), OP(T(157), T(118), T(117), 1, 0), \
    OP(T(158), T(121), T(119), 1, 0), OP(T(159), Y(3), Y(5), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(160), T(123), T(157), 0, 1), \
    OP(T(161), Y(20), T(158), 0, 1), OP(T(166), T(125), T(157), 0, 1), OP(T(116), Y(17), T(158), 0, 1), \
    OP(T(128), T(135), T(157), 0, 1), OP(T(129), Y(16), T(158), 0, 1), OP(T(130), T(137), T(157), 0, 1), \
    OP(T(132), Y(15), T(158), 0, 1), OP(T(133), T(139), T(157), 0, 1), OP(T(134), Y(14), T(158), 0, 1), \
    OP(T(136), Y(21), T(159), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(138), T(131), T(127), 0, 1), OP(T(143), T(160), T(127), 0, 1), OP(T(144), T(161), T(131), 0, 1), \
    OP(T(150), T(141), T(140), 0, 1), OP(T(152), T(166), T(140), 0, 1), OP(T(154), T(116), T(141), 0, 1), \
    OP(T(162), T(149), T(142), 0, 1), OP(T(163), T(128), T(142), 0, 1), OP(T(164), T(129), T(149), 0, 1), \
    OP(T(165), T(153), T(151), 0, 1), OP(T(167), T(130), T(151), 0, 1), OP(T(104), T(132), T(153), 0, 1), \
    OP(T(105), T(156), T(155), 0, 1), OP(T(106), T(133), T(155), 0, 1), OP(T(107), T(134), T(156), 0, 1), \
    OP(T(108), T(158), T(157), 0, 1), OP(T(109), T(144), T(143), 0, 0), OP(T(110), T(154), T(152), 0, 0), \
    OP(T(111), T(164), T(163), 0, 0), OP(T(112), T(104), T(167), 0, 0), OP(T(113), T(107), T(106), 0, 0), \
    OP(T(114), Y(10), Y(12), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(115), T(138), Y(21), 0, 1), \
    OP(T(117), T(150), Y(21), 0, 1), OP(T(118), T(162), Y(21), 0, 1), OP(T(119), T(165), Y(21), 0, 1), \
    OP(T(120), T(105), Y(21), 0, 1), OP(T(121), T(108), Y(21), 0, 1), OP(T(122), T(136), T(114), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(124), T(109), T(122), 0, 0), OP(T(126), T(110), T(122), 0, 0), OP(T(145), T(111), T(122), 0, 0), \
    OP(T(146), T(112), T(122), 0, 0), OP(T(147), T(113), T(122), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(148), T(124), T(121), 1, 0), OP(T(123), T(126), T(121), 1, 0), \
    OP(T(125), T(145), T(121), 1, 0), OP(T(135), T(146), T(121), 1, 0), OP(T(137), T(147), T(121), 1, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(139), T(148), T(115), 1, 0), \
    OP(T(159), T(123), T(117), 1, 0), OP(T(116), T(125), T(118), 1, 0), OP(T(127), T(135), T(119), 1, 0), \
    OP(T(128), T(137), T(120), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(168), IN(6), IN(14), 0, 1), OP(T(169), Y(21), Y(21), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(170), Y(8), IN(13), 0, 1), OP(T(171), Y(1), IN(21), 0, 1), \
    OP(T(172), IN(21), IN(13), 0, 1), OP(T(173), Y(8), IN(12), 0, 1), OP(T(174), Y(1), IN(20), 0, 1), \
    OP(T(175), IN(20), IN(12), 0, 1), OP(T(176), Y(8), IN(11), 0, 1), OP(T(177), Y(1), IN(19), 0, 1), \
    OP(T(178), IN(19), IN(11), 0, 1), OP(T(179), Y(8), IN(8), 0, 1), OP(T(180), Y(1), IN(16), 0, 1), \
    OP(T(181), IN(16), IN(8), 0, 1), OP(T(182), IN(15), Y(21), 0, 1), OP(T(183), Y(8), IN(7), 0, 1), \
    OP(T(184), Y(1), IN(15), 0, 1), OP(T(185), IN(15), IN(7), 0, 1), OP(T(186), T(171), T(170), 0, 0), \
    OP(T(187), T(168), T(172), 0, 0), OP(T(188), T(174), T(173), 0, 0), OP(T(189), T(168), T(175), 0, 0), \
    OP(T(190), T(177), T(176), 0, 0), OP(T(191), T(168), T(178), 0, 0), OP(T(192), T(180), T(179), 0, 0), \
    OP(T(193), T(168), T(181), 0, 0), OP(T(194), Y(8), T(182), 1, 0), OP(T(195), T(184), T(183), 0, 0), \
    OP(T(196), T(168), T(185), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(168), T(169), Y(21), 0, 1), OP(T(170), IN(8), Y(21), 0, 1), OP(T(171), IN(16), Y(21), 0, 1), \
    OP(T(172), IN(7), Y(21), 0, 1), OP(T(173), IN(14), Y(21), 0, 1), OP(T(174), IN(6), Y(21), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(175), T(168), T(187), 0, 1), OP(T(176), T(168), T(189), 0, 1), \
    OP(T(177), T(168), T(191), 0, 1), OP(T(178), T(168), T(193), 0, 1), OP(T(179), T(168), T(196), 0, 1), \
    OP(T(180), T(169), T(186), 0, 1), OP(T(181), T(169), T(188), 0, 1), OP(T(182), T(169), T(190), 0, 1), \
    OP(T(183), T(169), T(192), 0, 1), OP(T(184), T(169), T(195), 0, 1), OP(T(185), IN(13), Y(21), 0, 1), \
    OP(T(197), IN(21), Y(21), 0, 1), OP(T(198), IN(12), Y(21), 0, 1), OP(T(199), IN(20), Y(21), 0, 1), \
    OP(T(200), IN(11), Y(21), 0, 1), OP(T(201), IN(19), Y(21), 0, 1), OP(T(168), T(175), T(180), 1, 0), \
    OP(T(186), T(176), T(181), 1, 0), OP(T(187), T(177), T(182), 1, 0), OP(T(188), T(178), T(183), 1, 0), \
    OP(T(189), T(179), T(184), 1, 0), OP(T(190), Y(1), T(185), 1, 0), OP(T(191), Y(8), T(197), 1, 0), \
    OP(T(192), Y(1), T(198), 1, 0), OP(T(193), Y(8), T(199), 1, 0), OP(T(195), Y(1), T(200), 1, 0), \
    OP(T(196), Y(8), T(201), 1, 0), OP(T(202), Y(1), T(170), 1, 0), OP(T(203), Y(8), T(171), 1, 0), \
    OP(T(204), Y(11), T(173), 1, 0), OP(T(205), Y(1), T(172), 1, 0), OP(T(206), Y(4), T(174), 1, 0), \
    OP(T(170), IN(44), T(190), 0, 1), OP(T(171), Y(20), T(191), 0, 1), OP(T(172), IN(43), T(192), 0, 1), \
    OP(T(175), Y(19), T(193), 0, 1), OP(T(176), IN(42), T(195), 0, 1), OP(T(177), Y(18), T(196), 0, 1), \
    OP(T(178), IN(39), T(202), 0, 1), OP(T(179), Y(15), T(203), 0, 1), OP(T(180), IN(38), T(205), 0, 1), \
    OP(T(181), Y(14), T(194), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(182), T(170), T(204), 0, 1), OP(T(183), T(171), T(206), 0, 1), \
    OP(T(184), T(172), T(204), 0, 1), OP(T(185), T(175), T(206), 0, 1), OP(T(197), T(176), T(204), 0, 1), \
    OP(T(198), T(177), T(206), 0, 1), OP(T(199), T(178), T(204), 0, 1), OP(T(200), T(179), T(206), 0, 1), \
    OP(T(201), T(180), T(204), 0, 1), OP(T(190), T(181), T(206), 0, 1), OP(T(191), Y(11), Y(21), 0, 1), \
    OP(T(192), Y(4), Y(21), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(193), T(168), T(183), 1, 0), \
    OP(T(194), T(186), T(185), 1, 0), OP(T(195), T(187), T(198), 1, 0), OP(T(196), T(188), T(200), 1, 0), \
    OP(T(202), T(189), T(190), 1, 0), OP(T(203), Y(1), T(174), 1, 0), OP(T(205), Y(8), T(173), 1, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(170), T(182), T(169), 0, 1), OP(T(171), T(184), T(169), 0, 1), OP(T(172), T(197), T(169), 0, 1), \
    OP(T(175), T(199), T(169), 0, 1), OP(T(176), T(201), T(169), 0, 1), OP(T(177), T(191), T(203), 0, 1), \
    OP(T(178), T(192), T(205), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), OP(T(207), Y(0), Y(0), 0, 1), \
    OP(T(207), Y(0), Y(0), 0, 1), OP(T(179), T(193), T(178), 0, 0), OP(T(180), T(194), T(178), 0, 0), \
    OP(T(181), T(195), T(178), 0, 0), OP(T(204), T(196), T(178), 0, 0), OP(T(206), T(202), T(178), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(168), T(179), T(177), 0, 0), \
    OP(T(173), T(180), T(177), 0, 0), OP(T(174), T(181), T(177), 0, 0), OP(T(183), T(204), T(177), 0, 0), \
    OP(T(185), T(206), T(177), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(186), T(168), T(170), 1, 0), OP(T(187), T(173), T(171), 1, 0), OP(T(188), T(174), T(172), 1, 0), \
    OP(T(189), T(183), T(175), 1, 0), OP(T(190), T(185), T(176), 1, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), OP(T(207), Y(0), Y(0), 0, 0), \
    OP(T(207), Y(0), Y(0), 0, 0), 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, \
    0, 0, 0, 0, 0, 0
#define FRG_RESIDUAL_OUTS(OUT, T) \
    OUT(T(30), 0, 0, 1), OUT(T(29), 0, 1, 1), OUT(T(28), 0, 2, 1), OUT(T(27), 0, 3, 1), OUT(T(34), 1, 2, 1), \
    OUT(T(31), 1, 3, 1), 0xffff, OUT(T(72), 0, 4, 1), OUT(T(71), 0, 5, 1), OUT(T(70), 0, 6, 1), \
    OUT(T(74), 2, 4, 0), OUT(T(73), 2, 5, 0), 0xffff, 0xffff, OUT(T(128), 2, 0, 0), OUT(T(127), 2, 1, 0), \
    OUT(T(116), 2, 2, 0), OUT(T(159), 2, 3, 0), OUT(T(139), 2, 6, 0), 0xffff, 0xffff, OUT(T(190), 1, 0, 1), \
    OUT(T(189), 1, 1, 1), OUT(T(188), 1, 4, 1), OUT(T(187), 1, 5, 1), OUT(T(186), 1, 6, 1), 0xffff, 0xffff
