// GENERATED by csrc/gen/gen_fsc.py -- do not edit.
//
// Free-surface correction of a triangle side: strain (e[slip][component], tensor
// components 11, 22, 33, 12, 13, 23) and displacement (d[3 component + slip]) in the
// side's coordinates as linear combinations of the accumulators of FscAcc / FscDispAcc
// (end B minus end A), without the factor 1 / (4 pi (1 - nu)).
#pragma once

namespace cad {

template <typename T>
struct FscRows {
    T e[104];
};

CAD_HD void fsc_rows_setup(double s, double c, double nu, FscRows<double>& k)
{
    const double is = 1.0 / s, is2 = is * is;
    k.e[0] = 0.5*c*(2*nu - 1)*(-c*c)*is;
    k.e[1] = -c*(-c*c);
    k.e[2] = 0.5*(2*nu - 1)*(5*nu*(s*s) - 4*nu - 4*(s*s) + 4)*is2;
    k.e[3] = c*(2*nu - 1)*(-c*c)*(-2*nu + (s*s) + 2)*is2;
    k.e[4] = 0.25*(2*nu - 1)*(4*(s*s) - 3);
    k.e[5] = -0.25*(-8*nu*(s*s) + 6*nu + 5*(s*s*s*s) - 2*(s*s) - 3);
    k.e[6] = -0.5*c*(-c*c)*(-2*nu + 2*(s*s) + 1)*is;
    k.e[7] = 0.25*c*s*(3*(s*s) - 7);
    k.e[8] = 0.25*(s*s)*(3*(s*s) - 2);
    k.e[9] = 0.5*c*(2*nu - 1)*is;
    k.e[10] = -c;
    k.e[11] = -0.5*(2*nu - 1)*(nu*(s*s) - 4*nu - 4*(s*s) + 4)*is2;
    k.e[12] = -c*(2*nu - 1)*(2*nu + (s*s) - 2)*is2;
    k.e[13] = 0.75*(2*nu - 1);
    k.e[14] = 0.75*(2*nu + (s*s) - 1);
    k.e[15] = 0.75*c*s;
    k.e[16] = 0.75*(s*s);
    k.e[17] = 0.5*c*s*(2*nu - 1);
    k.e[18] = c*(s*s);
    k.e[19] = 2*nu*(2*nu - 1);
    k.e[20] = c*(-2*nu + (s*s))*(2*nu - 1);
    k.e[21] = (s*s)*(2*nu - 1);
    k.e[22] = 0.25*(s*s)*(-8*nu + 5*(s*s) - 5);
    k.e[23] = 0.5*c*s*(-2*nu + 2*(s*s) - 1);
    k.e[24] = -0.25*c*s*(3*(s*s) - 4);
    k.e[25] = -0.25*(s*s)*(3*(s*s) + 1);
    k.e[26] = -0.5*(2*nu - 1)*(-c*c)*is;
    k.e[27] = (-c*c);
    k.e[28] = 0.5*c*(2*nu - 1)*(2*nu + (s*s) - 2)*is;
    k.e[29] = -0.5*(2*nu - 1)*(3*nu*(s*s) - 4*nu - 4*(s*s) + 4)*is2;
    k.e[30] = 2*(nu - 1)*(2*nu - 1)*(-c*c)*is2;
    k.e[31] = -0.25*(2*nu - 1)*(2*(s*s) - 3);
    k.e[32] = 0.25*(-4*nu*(s*s) + 6*nu + (s*s*s*s) + 2*(s*s) - 3);
    k.e[33] = -0.25*c*s*(-4*nu + (s*s) + 1);
    k.e[34] = 0.5*(-c*c)*(-2*nu + (s*s) + 1)*is;
    k.e[35] = -0.5*c*s*(-c*c);
    k.e[36] = -0.25*(s*s)*(2*(s*s) - 3);
    k.e[37] = -0.25*c*s*((s*s) + 3);
    k.e[38] = -s*(-c*c);
    k.e[39] = 0.25*c*s*(-8*nu + 5*(s*s) - 1);
    k.e[40] = -(-nu + (s*s))*(-c*c);
    k.e[41] = 0.25*(s*s)*(3*(s*s) - 7);
    k.e[42] = -0.25*c*s*(3*(s*s) + 1);
    k.e[43] = -c*s;
    k.e[44] = -0.25*(s*s)*(-4*nu + (s*s) - 1);
    k.e[45] = -0.5*c*(-2*nu + (s*s));
    k.e[46] = -0.5*(s*s)*(-c*c);
    k.e[47] = 0.25*c*s*(2*(s*s) - 1);
    k.e[48] = -0.25*(s*s)*((s*s) + 3);
    k.e[49] = -0.5*c*(2*nu - 1)*(4*nu*(s*s) - 2*nu - (s*s) + 2)*is;
    k.e[50] = -0.5*(2*nu - 1)*(7*nu*(s*s) - 4*nu - 4*(s*s) + 4)*is2;
    k.e[51] = -2*(2*nu - 1)*(-c*c)*(nu*(s*s) - nu + 1)*is2;
    k.e[52] = 0.25*(4*nu*(s*s*s*s) - 16*nu*(s*s) + 6*nu + (s*s*s*s) + 2*(s*s) - 3);
    k.e[53] = -0.25*c*s*(4*nu*(s*s) + (s*s) + 1);
    k.e[54] = 0.5*(-c*c)*(2*nu*(s*s) - 2*nu + (s*s) + 1)*is;
    k.e[55] = -0.5*(2*nu - 1)*is;
    k.e[56] = -c*(nu - 1)*(2*nu - 1)*is;
    k.e[57] = 0.25*(4*nu*(s*s) - 6*nu - 3*(s*s) + 3);
    k.e[58] = -0.25*c*s*(4*nu - 3);
    k.e[59] = -0.5*c*s;
    k.e[60] = -0.5*(s*s);
    k.e[61] = -0.25*c*s;
    k.e[62] = -0.5*s*(2*nu - 1);
    k.e[63] = -(s*s);
    k.e[64] = -0.5*c*s*(2*nu - 1)*(4*nu - 1);
    k.e[65] = -2*nu*(2*nu - 1)*(-c*c);
    k.e[66] = -0.5*(s*s)*(2*nu - 1);
    k.e[67] = -0.25*(s*s)*(4*nu*(s*s) - 12*nu + (s*s) - 1);
    k.e[68] = 0.25*c*s*(4*nu*(s*s) + 4*nu + (s*s) - 2);
    k.e[69] = -0.5*s*(2*nu + 1)*(-c*c);
    k.e[70] = 0.5*c*(s*s*s);
    k.e[71] = 0.25*(s*s)*(2*(s*s) - 1);
    k.e[72] = 0.25*c*s*((s*s) + 4);
    k.e[73] = c*(2*nu - 1)*(2*nu*(s*s) - 2*nu - (s*s) + 2)*is2;
    k.e[74] = -0.25*(8*nu*(s*s) - 6*nu - 3*(s*s) + 3);
    k.e[75] = -0.5*c*(2*nu*(s*s) - 2*nu + 1)*is;
    k.e[76] = -0.25*c*s*(4*nu*(s*s) - 12*nu + (s*s) + 1);
    k.e[77] = -0.25*(s*s)*(4*nu*(s*s) + (s*s) - 1);
    k.e[78] = -0.5*c*(2*nu*(s*s) - 2*nu + (s*s));
    k.e[79] = -s;
    k.e[80] = 0.25*c*s*(8*nu - 3);
    k.e[81] = -nu*(-c*c);
    k.e[82] = -0.5*(2*nu - 1)*(-c*c);
    k.e[83] = -s*(2*nu - 1)*(-c*c);
    k.e[84] = c*s*(2*nu - 1);
    k.e[85] = -1.25*c*s*(-c*c);
    k.e[86] = 0.5*(-c*c)*(2*(s*s) - 1);
    k.e[87] = -0.5*(2*nu - 1);
    k.e[88] = s*(2*nu - 1);
    k.e[89] = -0.5;
    k.e[90] = -(s*s*s);
    k.e[91] = -s*(2*nu - 1)*((s*s) - 2);
    k.e[92] = 0.25*c*s*(5*(s*s) - 8);
    k.e[93] = -0.5*(s*s)*(2*(s*s) - 3);
    k.e[94] = 0.25*(s*s)*(3*(s*s) - 4);
    k.e[95] = -0.25*c*s*(3*(s*s) + 4);
    k.e[96] = -0.5*c*(2*nu - 1);
    k.e[97] = 0.25*c*s*(-c*c);
    k.e[98] = 0.25*(s*s)*((s*s) - 3);
    k.e[99] = 0.5*c*(-c*c);
    k.e[100] = -0.25*(s*s)*(5*(s*s) - 9);
    k.e[101] = -c*s*(-c*c);
    k.e[102] = -0.25*c*s*(s - 2)*(s + 2);
    k.e[103] = 0.5*s*((s*s) - 2);
}

template <typename T>
struct FscDispRows {
    T d[34];
};

CAD_HD void fsc_rows_setup(double s, double c, double nu, FscDispRows<double>& k)
{
    const double is = 1.0 / s, is2 = is * is;
    k.d[0] = 2*(nu - 1)*(2*nu - 1)*(-c*c)*is2;
    k.d[1] = (2*nu - 1)*(-c*c)*is;
    k.d[2] = -0.5*(-c*c);
    k.d[3] = -(-c*c)*(-2*nu + (s*s) + 1)*is;
    k.d[4] = c*s;
    k.d[5] = -(2*nu - 1)*(3*nu*(s*s) - 2*nu - 2*(s*s) + 2)*is2;
    k.d[6] = c*(2*nu - 1)*(2*nu*(s*s) - 2*nu - (s*s) + 2)*is2;
    k.d[7] = c*(2*nu - 1)*is;
    k.d[8] = -0.5*c;
    k.d[9] = -c*(2*nu*(s*s) - 2*nu + 1)*is;
    k.d[10] = -0.5*(2*nu - 1);
    k.d[11] = 0.5*(4*nu*(s*s) - 2*nu - (s*s) + 1);
    k.d[12] = -0.5*c*s;
    k.d[13] = -0.5*(s*s);
    k.d[14] = c*(2*nu - 1);
    k.d[15] = -c*(-c*c);
    k.d[16] = -(s*s);
    k.d[17] = -(2*nu - 1)*(nu*(s*s) - 2*nu - 2*(s*s) + 2)*is2;
    k.d[18] = -c*(2*nu - 1)*(2*nu + (s*s) - 2)*is2;
    k.d[19] = -0.5*(2*nu + (s*s) - 1);
    k.d[20] = (2*nu - 1)*is;
    k.d[21] = -0.5;
    k.d[22] = s*(2*nu - 1);
    k.d[23] = 1 - 2*nu;
    k.d[24] = 0.5*s;
    k.d[25] = 2*c*(nu - 1)*(2*nu - 1)*is;
    k.d[26] = 2*c*(nu - 1);
    k.d[27] = c*(-2*nu + (s*s));
    k.d[28] = -2*(nu - 1)*(2*nu - 1)*(-c*c)*is;
    k.d[29] = -2*(nu - 1);
    k.d[30] = -2*nu*(-c*c);
    k.d[31] = -0.5*c*s*(4*nu - 1);
    k.d[32] = -2*s*(nu - 1);
    k.d[33] = -s*((s*s) - 2);
}

template <typename R>
CAD_HD void fsc_rows(const FscRows<R>& k, const FscAcc<R>& a, R z, R e[3][6])
{
    e[0][0] = a.Mi + k.e[0] * a.Oi + k.e[1] * a.Ni + k.e[2] * a.h1i + k.e[3] * a.g1i + k.e[4] * a.At2 + z * (k.e[5] * a.t2 + k.e[6] * a.w2i + k.e[7] * a.s12 + k.e[8] * a.s2q);
    e[0][1] = -a.Mi + k.e[9] * a.Oi + k.e[10] * a.Ni + k.e[11] * a.h1i + k.e[12] * a.g1i + k.e[13] * a.At2 + z * (k.e[14] * a.t2 + k.e[9] * a.w2i + k.e[15] * a.s12 + k.e[16] * a.s2q);
    e[0][2] = k.e[17] * a.Oi + k.e[18] * a.Ni + k.e[19] * a.h1i + k.e[20] * a.g1i + k.e[21] * a.At2 + z * (k.e[22] * a.t2 + k.e[23] * a.w2i + k.e[24] * a.s12 + k.e[25] * a.s2q);
    e[0][3] = -a.Mr + k.e[26] * a.Or + k.e[27] * a.Nr + k.e[28] * a.h0 + k.e[29] * a.h1r + k.e[30] * a.g1r + k.e[31] * a.At1 + k.e[17] * a.Atq + z * (k.e[32] * a.t1 + k.e[33] * a.tq + k.e[34] * a.w2r + k.e[35] * a.s11 + k.e[36] * a.s1q + k.e[37] * a.s22);
    e[0][4] = a.Yi + k.e[38] * a.Ni + z * (k.e[39] * a.t2 + k.e[40] * a.w2i + k.e[41] * a.s12 + k.e[42] * a.s2q);
    e[0][5] = -a.Yr + k.e[43] * a.Nr + z * (k.e[33] * a.t1 + k.e[44] * a.tq + k.e[45] * a.w2r + k.e[46] * a.s11 + k.e[47] * a.s1q + k.e[48] * a.s22);
    e[1][0] = -a.Mr + k.e[26] * a.Or + k.e[27] * a.Nr + k.e[49] * a.h0 + k.e[50] * a.h1r + k.e[51] * a.g1r + k.e[31] * a.At1 + k.e[17] * a.Atq + z * (k.e[52] * a.t1 + k.e[53] * a.tq + k.e[54] * a.w2r + k.e[35] * a.s11 + k.e[36] * a.s1q + k.e[37] * a.s22);
    e[1][1] = a.Mr + k.e[55] * a.Or + a.Nr + k.e[56] * a.h0 - k.e[29] * a.h1r - k.e[30] * a.g1r - k.e[13] * a.At1 + z * (k.e[57] * a.t1 + k.e[58] * a.tq - k.e[26] * a.w2r + k.e[59] * a.s11 + k.e[60] * a.s1q + k.e[61] * a.s22);
    e[1][2] = k.e[62] * a.Or + k.e[63] * a.Nr + k.e[64] * a.h0 - k.e[19] * a.h1r + k.e[65] * a.g1r + k.e[66] * a.At1 + k.e[17] * a.Atq + z * (k.e[67] * a.t1 + k.e[68] * a.tq + k.e[69] * a.w2r + k.e[70] * a.s11 + k.e[71] * a.s1q + k.e[72] * a.s22);
    e[1][3] = -a.Mi + k.e[9] * a.Oi + k.e[10] * a.Ni - k.e[2] * a.h1i + k.e[73] * a.g1i + k.e[13] * a.At2 + z * (k.e[74] * a.t2 + k.e[75] * a.w2i + k.e[15] * a.s12 + k.e[16] * a.s2q);
    e[1][4] = -a.Yr + k.e[43] * a.Nr + z * (k.e[76] * a.t1 + k.e[77] * a.tq + k.e[78] * a.w2r + k.e[46] * a.s11 + k.e[47] * a.s1q + k.e[48] * a.s22);
    e[1][5] = -a.Yi + k.e[79] * a.Ni + z * (k.e[80] * a.t2 + k.e[81] * a.w2i + k.e[16] * a.s12 - k.e[15] * a.s2q);
    e[2][0] = a.Si + k.e[82] * a.Oi - k.e[38] * a.Ni + k.e[83] * a.g1i + k.e[84] * a.At2 + z * (k.e[85] * a.t2 + k.e[86] * a.w2i - k.e[41] * a.s12 - k.e[42] * a.s2q);
    e[2][1] = -a.Si + k.e[87] * a.Oi - k.e[79] * a.Ni + k.e[88] * a.g1i + z * (k.e[15] * a.t2 + k.e[89] * a.w2i - k.e[16] * a.s12 + k.e[15] * a.s2q);
    e[2][2] = k.e[66] * a.Oi + k.e[90] * a.Ni + k.e[91] * a.g1i + k.e[84] * a.At2 + z * (k.e[92] * a.t2 + k.e[93] * a.w2i + k.e[94] * a.s12 + k.e[95] * a.s2q);
    e[2][3] = -a.Sr + k.e[96] * a.Or - k.e[43] * a.Nr + k.e[66] * a.h0 - k.e[17] * a.At1 + k.e[66] * a.Atq + z * (k.e[97] * a.t1 + k.e[98] * a.tq + k.e[99] * a.w2r - k.e[46] * a.s11 - k.e[47] * a.s1q - k.e[48] * a.s22);
    e[2][4] = -k.e[18] * a.Ni + z * (k.e[100] * a.t2 + k.e[101] * a.w2i - k.e[24] * a.s12 - k.e[25] * a.s2q);
    e[2][5] = -k.e[63] * a.Nr + z * (k.e[98] * a.t1 + k.e[102] * a.tq + k.e[103] * a.w2r - k.e[70] * a.s11 - k.e[71] * a.s1q - k.e[72] * a.s22);
}

template <typename R>
CAD_HD void fsc_disp_rows(const FscDispRows<R>& k, const FscDispAcc<R>& a, R d[9])
{
    d[0] = k.d[0] * a.F + a.Bi + k.d[1] * a.O1i + k.d[2] * a.O2i + k.d[3] * a.zg1i + k.d[4] * a.azt2;
    d[1] = k.d[5] * a.phi + k.d[6] * a.chi - a.Br + k.d[7] * a.O1r + k.d[8] * a.O2r + k.d[9] * a.zg1r + k.d[10] * a.ah0 + k.d[11] * a.zh0 + k.d[12] * a.azt1 + k.d[13] * a.aztq;
    d[2] = a.B3i + k.d[14] * a.O1i + k.d[12] * a.O2i + k.d[15] * a.zg1i + k.d[16] * a.azt2;
    d[3] = k.d[17] * a.phi + k.d[18] * a.chi - a.Br + k.d[7] * a.O1r + k.d[8] * a.O2r + k.d[7] * a.zg1r + k.d[10] * a.ah0 + k.d[19] * a.zh0 + k.d[12] * a.azt1 + k.d[13] * a.aztq;
    d[4] = -k.d[0] * a.F - a.Bi + k.d[20] * a.O1i + k.d[21] * a.O2i - k.d[1] * a.zg1i;
    d[5] = k.d[22] * a.chi - a.B3r + k.d[23] * a.O1r + k.d[24] * a.O2r - a.zg1r + k.d[12] * a.zh0 - k.d[13] * a.azt1 + k.d[12] * a.aztq;
    d[6] = k.d[25] * a.F + a.B4i + k.d[26] * a.O1i - k.d[12] * a.O2i + k.d[27] * a.zg1i - k.d[16] * a.azt2;
    d[7] = -k.d[25] * a.phi + k.d[28] * a.chi - a.B4r + k.d[29] * a.O1r - k.d[24] * a.O2r + k.d[30] * a.zg1r + k.d[31] * a.zh0 + k.d[13] * a.azt1 - k.d[12] * a.aztq;
    d[8] = k.d[29] * a.F + k.d[32] * a.O1i + k.d[13] * a.O2i + k.d[33] * a.zg1i + k.d[4] * a.azt2;
}

}  // namespace cad
