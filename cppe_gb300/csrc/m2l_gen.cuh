// Generated by gen_m2l.py -- do not edit.
#pragma once

// M2L between reduced coefficients, source order 1, expansion order 5: 35 multipole, 25 local, 46 tensor entries, 265 terms
template <typename T>
__device__ __forceinline__ void m2l_m1_p5(T x, T y, T z, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  { const T mk = Mb[0];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D31, mk, acc[0]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D32, mk, acc[0]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D33, mk, acc[0]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D34, mk, acc[0]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D35, mk, acc[0]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D37, mk, acc[0]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D38, mk, acc[0]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D40, mk, acc[0]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D41, mk, acc[0]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D43, mk, acc[0]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D44, mk, acc[0]);
  }
}
template <typename T>
__device__ __forceinline__ void dtensor_m1_p5(T x, T y, T z, T* __restrict__ Dout) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  Dout[0] = D0;
  Dout[1] = D1;
  Dout[2] = D2;
  Dout[3] = D3;
  Dout[4] = D4;
  Dout[5] = D5;
  Dout[6] = D6;
  Dout[7] = D7;
  Dout[8] = D8;
  Dout[9] = D9;
  Dout[10] = D10;
  Dout[11] = D11;
  Dout[12] = D12;
  Dout[13] = D13;
  Dout[14] = D14;
  Dout[15] = D15;
  Dout[16] = D16;
  Dout[17] = D17;
  Dout[18] = D18;
  Dout[19] = D19;
  Dout[20] = D20;
  Dout[21] = D21;
  Dout[22] = D22;
  Dout[23] = D23;
  Dout[24] = D24;
  Dout[25] = D25;
  Dout[26] = D26;
  Dout[27] = D27;
  Dout[28] = D28;
  Dout[29] = D29;
  Dout[30] = D30;
  Dout[31] = D31;
  Dout[32] = D32;
  Dout[33] = D33;
  Dout[34] = D34;
  Dout[35] = D35;
  Dout[36] = D36;
  Dout[37] = D37;
  Dout[38] = D38;
  Dout[39] = D39;
  Dout[40] = D40;
  Dout[41] = D41;
  Dout[42] = D42;
  Dout[43] = D43;
  Dout[44] = D44;
  Dout[45] = D45;
}
template <typename T>
__device__ __forceinline__ void m2l_m1_p5_pre(const T* __restrict__ Dt, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T D0 = Dt[0];
  const T D1 = Dt[1];
  const T D2 = Dt[2];
  const T D3 = Dt[3];
  const T D4 = Dt[4];
  const T D5 = Dt[5];
  const T D6 = Dt[6];
  const T D7 = Dt[7];
  const T D8 = Dt[8];
  const T D9 = Dt[9];
  const T D10 = Dt[10];
  const T D11 = Dt[11];
  const T D12 = Dt[12];
  const T D13 = Dt[13];
  const T D14 = Dt[14];
  const T D15 = Dt[15];
  const T D16 = Dt[16];
  const T D17 = Dt[17];
  const T D18 = Dt[18];
  const T D19 = Dt[19];
  const T D20 = Dt[20];
  const T D21 = Dt[21];
  const T D22 = Dt[22];
  const T D23 = Dt[23];
  const T D24 = Dt[24];
  const T D25 = Dt[25];
  const T D26 = Dt[26];
  const T D27 = Dt[27];
  const T D28 = Dt[28];
  const T D29 = Dt[29];
  const T D30 = Dt[30];
  const T D31 = Dt[31];
  const T D32 = Dt[32];
  const T D33 = Dt[33];
  const T D34 = Dt[34];
  const T D35 = Dt[35];
  const T D36 = Dt[36];
  const T D37 = Dt[37];
  const T D38 = Dt[38];
  const T D39 = Dt[39];
  const T D40 = Dt[40];
  const T D41 = Dt[41];
  const T D42 = Dt[42];
  const T D43 = Dt[43];
  const T D44 = Dt[44];
  const T D45 = Dt[45];
  { const T mk = Mb[0];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D31, mk, acc[0]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D32, mk, acc[0]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D33, mk, acc[0]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D34, mk, acc[0]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D35, mk, acc[0]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D37, mk, acc[0]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D38, mk, acc[0]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D40, mk, acc[0]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D41, mk, acc[0]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D43, mk, acc[0]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D44, mk, acc[0]);
  }
}
static __constant__ unsigned char m2l_w_m1_p5[265] = {
  1, 4, 5, 6, 10, 11, 12, 13, 14, 19, 20, 21, 22, 23, 25, 26, 31, 32, 33, 34, 35, 37, 38, 40, 41, 2, 5, 7, 8, 11, 13, 14, 16, 17, 20, 22, 23, 25, 26, 28, 29, 32, 34, 35, 37, 38, 40, 41, 43, 44, 3, 6, 8, 9, 12, 14, 15, 17, 18, 21, 23, 24, 26, 27, 29, 30, 33, 35, 36, 38, 39, 41, 42, 44, 45, 4, 10, 11, 12, 19, 20, 21, 22, 23, 31, 32, 33, 34, 35, 37, 38, 5, 11, 13, 14, 20, 22, 23, 25, 26, 32, 34, 35, 37, 38, 40, 41, 6, 12, 14, 15, 21, 23, 24, 26, 27, 33, 35, 36, 38, 39, 41, 42, 7, 13, 16, 17, 22, 25, 26, 28, 29, 34, 37, 38, 40, 41, 43, 44, 8, 14, 17, 18, 23, 26, 27, 29, 30, 35, 38, 39, 41, 42, 44, 45, 10, 19, 20, 21, 31, 32, 33, 34, 35, 11, 20, 22, 23, 32, 34, 35, 37, 38, 12, 21, 23, 24, 33, 35, 36, 38, 39, 13, 22, 25, 26, 34, 37, 38, 40, 41, 14, 23, 26, 27, 35, 38, 39, 41, 42, 16, 25, 28, 29, 37, 40, 41, 43, 44, 17, 26, 29, 30, 38, 41, 42, 44, 45, 19, 31, 32, 33, 20, 32, 34, 35, 21, 33, 35, 36, 22, 34, 37, 38, 23, 35, 38, 39, 25, 37, 40, 41, 26, 38, 41, 42, 28, 40, 43, 44, 29, 41, 44, 45, 31, 32, 33, 34, 35, 37, 38, 40, 41, 43, 44};
static __device__ const signed char m2l_fold_m1_p5[35][4][2] = {
  {{0, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {8, -1}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {8, -1}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{9, 1}, {14, -1}, {0, 0}, {0, 0}},
  {{10, 1}, {17, -1}, {0, 0}, {0, 0}},
  {{11, 1}, {18, -1}, {0, 0}, {0, 0}},
  {{12, 1}, {14, -1}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{15, 1}, {17, -1}, {0, 0}, {0, 0}},
  {{16, 1}, {18, -1}, {0, 0}, {0, 0}},
  {{19, 1}, {24, -1}, {33, 1}, {0, 0}},
  {{20, 1}, {27, -1}, {0, 0}, {0, 0}},
  {{21, 1}, {28, -1}, {0, 0}, {0, 0}},
  {{22, 1}, {24, -1}, {31, -1}, {33, 2}},
  {{23, 1}, {32, -1}, {0, 0}, {0, 0}},
  {{25, 1}, {27, -1}, {0, 0}, {0, 0}},
  {{26, 1}, {28, -1}, {0, 0}, {0, 0}},
  {{29, 1}, {31, -1}, {33, 1}, {0, 0}},
  {{30, 1}, {32, -1}, {0, 0}, {0, 0}},
  {{34, 1}, {39, -1}, {48, 1}, {0, 0}},
  {{35, 1}, {42, -1}, {53, 1}, {0, 0}},
  {{36, 1}, {43, -1}, {54, 1}, {0, 0}},
  {{37, 1}, {39, -1}, {46, -1}, {48, 2}},
  {{38, 1}, {47, -1}, {0, 0}, {0, 0}},
  {{40, 1}, {42, -1}, {51, -1}, {53, 2}},
  {{41, 1}, {43, -1}, {52, -1}, {54, 2}},
  {{44, 1}, {46, -1}, {48, 1}, {0, 0}},
  {{45, 1}, {47, -1}, {0, 0}, {0, 0}},
  {{49, 1}, {51, -1}, {53, 1}, {0, 0}},
  {{50, 1}, {52, -1}, {54, 1}, {0, 0}},
};
static __device__ const signed char m2l_unfold_m1_p5[35][3][2] = {
  {{0, 1}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}},
  {{7, -1}, {4, -1}, {0, 0}},
  {{9, 1}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}},
  {{11, 1}, {0, 0}, {0, 0}},
  {{12, 1}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}},
  {{12, -1}, {9, -1}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}},
  {{15, 1}, {0, 0}, {0, 0}},
  {{14, -1}, {10, -1}, {0, 0}},
  {{15, -1}, {11, -1}, {0, 0}},
  {{16, 1}, {0, 0}, {0, 0}},
  {{17, 1}, {0, 0}, {0, 0}},
  {{18, 1}, {0, 0}, {0, 0}},
  {{19, 1}, {0, 0}, {0, 0}},
  {{20, 1}, {0, 0}, {0, 0}},
  {{19, -1}, {16, -1}, {0, 0}},
  {{21, 1}, {0, 0}, {0, 0}},
  {{22, 1}, {0, 0}, {0, 0}},
  {{21, -1}, {17, -1}, {0, 0}},
  {{22, -1}, {18, -1}, {0, 0}},
  {{23, 1}, {0, 0}, {0, 0}},
  {{24, 1}, {0, 0}, {0, 0}},
  {{23, -1}, {19, -1}, {0, 0}},
  {{24, -1}, {20, -1}, {0, 0}},
  {{23, 1}, {19, 2}, {16, 1}},
};

// M2L between reduced coefficients, source order 1, expansion order 6: 48 multipole, 36 local, 64 tensor entries, 483 terms
template <typename T>
__device__ __forceinline__ void m2l_m1_p6(T x, T y, T z, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  const T w6_6 = crat<T>(-150, 6) * ir2;
  const T x6_1 = crat<T>(-11, 6) * xr;
  const T x6_6 = T(6) * x6_1;
  const T D46 = fma(x6_6, D31, w6_6 * D19);
  const T w6_5 = crat<T>(-100, 6) * ir2;
  const T x6_5 = T(5) * x6_1;
  const T y6_1 = crat<T>(-11, 6) * yr;
  const T D47 = fma(y6_1, D31, fma(x6_5, D32, w6_5 * D20));
  const T z6_1 = crat<T>(-11, 6) * zr;
  const T D48 = fma(z6_1, D31, fma(x6_5, D33, w6_5 * D21));
  const T w6_4 = crat<T>(-60, 6) * ir2;
  const T w6_2 = crat<T>(-10, 6) * ir2;
  const T x6_4 = T(4) * x6_1;
  const T y6_2 = T(2) * y6_1;
  const T D49 = fma(y6_2, D32, fma(x6_4, D34, fma(w6_2, D19, w6_4 * D22)));
  const T D50 = fma(z6_1, D32, fma(y6_1, D33, fma(x6_4, D35, w6_4 * D23)));
  const T D51 = -(D46 + D49);
  const T w6_3 = crat<T>(-30, 6) * ir2;
  const T x6_3 = T(3) * x6_1;
  const T y6_3 = T(3) * y6_1;
  const T D52 = fma(y6_3, D34, fma(x6_3, D37, fma(w6_3, D20, w6_3 * D25)));
  const T D53 = fma(z6_1, D34, fma(y6_2, D35, fma(x6_3, D38, fma(w6_2, D21, w6_3 * D26))));
  const T D54 = -(D47 + D52);
  const T x6_2 = T(2) * x6_1;
  const T y6_4 = T(4) * y6_1;
  const T D55 = fma(y6_4, D37, fma(x6_2, D40, fma(w6_4, D22, w6_2 * D28)));
  const T D56 = fma(z6_1, D37, fma(y6_3, D38, fma(x6_2, D41, fma(w6_3, D23, w6_2 * D29))));
  const T D57 = -(D49 + D55);
  const T y6_5 = T(5) * y6_1;
  const T D58 = fma(y6_5, D40, fma(x6_1, D43, w6_5 * D25));
  const T D59 = fma(z6_1, D40, fma(y6_4, D41, fma(x6_1, D44, w6_4 * D26)));
  const T D60 = -(D52 + D58);
  const T y6_6 = T(6) * y6_1;
  const T D61 = fma(y6_6, D43, w6_6 * D28);
  const T D62 = fma(z6_1, D43, fma(y6_5, D44, w6_5 * D29));
  const T D63 = -(D55 + D61);
  { const T mk = Mb[0];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
    acc[25] = fma(D46, mk, acc[25]);
    acc[26] = fma(D47, mk, acc[26]);
    acc[27] = fma(D48, mk, acc[27]);
    acc[28] = fma(D49, mk, acc[28]);
    acc[29] = fma(D50, mk, acc[29]);
    acc[30] = fma(D52, mk, acc[30]);
    acc[31] = fma(D53, mk, acc[31]);
    acc[32] = fma(D55, mk, acc[32]);
    acc[33] = fma(D56, mk, acc[33]);
    acc[34] = fma(D58, mk, acc[34]);
    acc[35] = fma(D59, mk, acc[35]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
    acc[25] = fma(D47, mk, acc[25]);
    acc[26] = fma(D49, mk, acc[26]);
    acc[27] = fma(D50, mk, acc[27]);
    acc[28] = fma(D52, mk, acc[28]);
    acc[29] = fma(D53, mk, acc[29]);
    acc[30] = fma(D55, mk, acc[30]);
    acc[31] = fma(D56, mk, acc[31]);
    acc[32] = fma(D58, mk, acc[32]);
    acc[33] = fma(D59, mk, acc[33]);
    acc[34] = fma(D61, mk, acc[34]);
    acc[35] = fma(D62, mk, acc[35]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
    acc[25] = fma(D48, mk, acc[25]);
    acc[26] = fma(D50, mk, acc[26]);
    acc[27] = fma(D51, mk, acc[27]);
    acc[28] = fma(D53, mk, acc[28]);
    acc[29] = fma(D54, mk, acc[29]);
    acc[30] = fma(D56, mk, acc[30]);
    acc[31] = fma(D57, mk, acc[31]);
    acc[32] = fma(D59, mk, acc[32]);
    acc[33] = fma(D60, mk, acc[33]);
    acc[34] = fma(D62, mk, acc[34]);
    acc[35] = fma(D63, mk, acc[35]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
    acc[16] = fma(D46, mk, acc[16]);
    acc[17] = fma(D47, mk, acc[17]);
    acc[18] = fma(D48, mk, acc[18]);
    acc[19] = fma(D49, mk, acc[19]);
    acc[20] = fma(D50, mk, acc[20]);
    acc[21] = fma(D52, mk, acc[21]);
    acc[22] = fma(D53, mk, acc[22]);
    acc[23] = fma(D55, mk, acc[23]);
    acc[24] = fma(D56, mk, acc[24]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
    acc[16] = fma(D47, mk, acc[16]);
    acc[17] = fma(D49, mk, acc[17]);
    acc[18] = fma(D50, mk, acc[18]);
    acc[19] = fma(D52, mk, acc[19]);
    acc[20] = fma(D53, mk, acc[20]);
    acc[21] = fma(D55, mk, acc[21]);
    acc[22] = fma(D56, mk, acc[22]);
    acc[23] = fma(D58, mk, acc[23]);
    acc[24] = fma(D59, mk, acc[24]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
    acc[16] = fma(D48, mk, acc[16]);
    acc[17] = fma(D50, mk, acc[17]);
    acc[18] = fma(D51, mk, acc[18]);
    acc[19] = fma(D53, mk, acc[19]);
    acc[20] = fma(D54, mk, acc[20]);
    acc[21] = fma(D56, mk, acc[21]);
    acc[22] = fma(D57, mk, acc[22]);
    acc[23] = fma(D59, mk, acc[23]);
    acc[24] = fma(D60, mk, acc[24]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
    acc[16] = fma(D49, mk, acc[16]);
    acc[17] = fma(D52, mk, acc[17]);
    acc[18] = fma(D53, mk, acc[18]);
    acc[19] = fma(D55, mk, acc[19]);
    acc[20] = fma(D56, mk, acc[20]);
    acc[21] = fma(D58, mk, acc[21]);
    acc[22] = fma(D59, mk, acc[22]);
    acc[23] = fma(D61, mk, acc[23]);
    acc[24] = fma(D62, mk, acc[24]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
    acc[16] = fma(D50, mk, acc[16]);
    acc[17] = fma(D53, mk, acc[17]);
    acc[18] = fma(D54, mk, acc[18]);
    acc[19] = fma(D56, mk, acc[19]);
    acc[20] = fma(D57, mk, acc[20]);
    acc[21] = fma(D59, mk, acc[21]);
    acc[22] = fma(D60, mk, acc[22]);
    acc[23] = fma(D62, mk, acc[23]);
    acc[24] = fma(D63, mk, acc[24]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
    acc[9] = fma(D46, mk, acc[9]);
    acc[10] = fma(D47, mk, acc[10]);
    acc[11] = fma(D48, mk, acc[11]);
    acc[12] = fma(D49, mk, acc[12]);
    acc[13] = fma(D50, mk, acc[13]);
    acc[14] = fma(D52, mk, acc[14]);
    acc[15] = fma(D53, mk, acc[15]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
    acc[9] = fma(D47, mk, acc[9]);
    acc[10] = fma(D49, mk, acc[10]);
    acc[11] = fma(D50, mk, acc[11]);
    acc[12] = fma(D52, mk, acc[12]);
    acc[13] = fma(D53, mk, acc[13]);
    acc[14] = fma(D55, mk, acc[14]);
    acc[15] = fma(D56, mk, acc[15]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
    acc[9] = fma(D48, mk, acc[9]);
    acc[10] = fma(D50, mk, acc[10]);
    acc[11] = fma(D51, mk, acc[11]);
    acc[12] = fma(D53, mk, acc[12]);
    acc[13] = fma(D54, mk, acc[13]);
    acc[14] = fma(D56, mk, acc[14]);
    acc[15] = fma(D57, mk, acc[15]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
    acc[9] = fma(D49, mk, acc[9]);
    acc[10] = fma(D52, mk, acc[10]);
    acc[11] = fma(D53, mk, acc[11]);
    acc[12] = fma(D55, mk, acc[12]);
    acc[13] = fma(D56, mk, acc[13]);
    acc[14] = fma(D58, mk, acc[14]);
    acc[15] = fma(D59, mk, acc[15]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
    acc[9] = fma(D50, mk, acc[9]);
    acc[10] = fma(D53, mk, acc[10]);
    acc[11] = fma(D54, mk, acc[11]);
    acc[12] = fma(D56, mk, acc[12]);
    acc[13] = fma(D57, mk, acc[13]);
    acc[14] = fma(D59, mk, acc[14]);
    acc[15] = fma(D60, mk, acc[15]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
    acc[9] = fma(D52, mk, acc[9]);
    acc[10] = fma(D55, mk, acc[10]);
    acc[11] = fma(D56, mk, acc[11]);
    acc[12] = fma(D58, mk, acc[12]);
    acc[13] = fma(D59, mk, acc[13]);
    acc[14] = fma(D61, mk, acc[14]);
    acc[15] = fma(D62, mk, acc[15]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
    acc[9] = fma(D53, mk, acc[9]);
    acc[10] = fma(D56, mk, acc[10]);
    acc[11] = fma(D57, mk, acc[11]);
    acc[12] = fma(D59, mk, acc[12]);
    acc[13] = fma(D60, mk, acc[13]);
    acc[14] = fma(D62, mk, acc[14]);
    acc[15] = fma(D63, mk, acc[15]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
    acc[4] = fma(D46, mk, acc[4]);
    acc[5] = fma(D47, mk, acc[5]);
    acc[6] = fma(D48, mk, acc[6]);
    acc[7] = fma(D49, mk, acc[7]);
    acc[8] = fma(D50, mk, acc[8]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
    acc[4] = fma(D47, mk, acc[4]);
    acc[5] = fma(D49, mk, acc[5]);
    acc[6] = fma(D50, mk, acc[6]);
    acc[7] = fma(D52, mk, acc[7]);
    acc[8] = fma(D53, mk, acc[8]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
    acc[4] = fma(D48, mk, acc[4]);
    acc[5] = fma(D50, mk, acc[5]);
    acc[6] = fma(D51, mk, acc[6]);
    acc[7] = fma(D53, mk, acc[7]);
    acc[8] = fma(D54, mk, acc[8]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
    acc[4] = fma(D49, mk, acc[4]);
    acc[5] = fma(D52, mk, acc[5]);
    acc[6] = fma(D53, mk, acc[6]);
    acc[7] = fma(D55, mk, acc[7]);
    acc[8] = fma(D56, mk, acc[8]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
    acc[4] = fma(D50, mk, acc[4]);
    acc[5] = fma(D53, mk, acc[5]);
    acc[6] = fma(D54, mk, acc[6]);
    acc[7] = fma(D56, mk, acc[7]);
    acc[8] = fma(D57, mk, acc[8]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
    acc[4] = fma(D52, mk, acc[4]);
    acc[5] = fma(D55, mk, acc[5]);
    acc[6] = fma(D56, mk, acc[6]);
    acc[7] = fma(D58, mk, acc[7]);
    acc[8] = fma(D59, mk, acc[8]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
    acc[4] = fma(D53, mk, acc[4]);
    acc[5] = fma(D56, mk, acc[5]);
    acc[6] = fma(D57, mk, acc[6]);
    acc[7] = fma(D59, mk, acc[7]);
    acc[8] = fma(D60, mk, acc[8]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
    acc[4] = fma(D55, mk, acc[4]);
    acc[5] = fma(D58, mk, acc[5]);
    acc[6] = fma(D59, mk, acc[6]);
    acc[7] = fma(D61, mk, acc[7]);
    acc[8] = fma(D62, mk, acc[8]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
    acc[4] = fma(D56, mk, acc[4]);
    acc[5] = fma(D59, mk, acc[5]);
    acc[6] = fma(D60, mk, acc[6]);
    acc[7] = fma(D62, mk, acc[7]);
    acc[8] = fma(D63, mk, acc[8]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D31, mk, acc[0]);
    acc[1] = fma(D46, mk, acc[1]);
    acc[2] = fma(D47, mk, acc[2]);
    acc[3] = fma(D48, mk, acc[3]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D32, mk, acc[0]);
    acc[1] = fma(D47, mk, acc[1]);
    acc[2] = fma(D49, mk, acc[2]);
    acc[3] = fma(D50, mk, acc[3]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D33, mk, acc[0]);
    acc[1] = fma(D48, mk, acc[1]);
    acc[2] = fma(D50, mk, acc[2]);
    acc[3] = fma(D51, mk, acc[3]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D34, mk, acc[0]);
    acc[1] = fma(D49, mk, acc[1]);
    acc[2] = fma(D52, mk, acc[2]);
    acc[3] = fma(D53, mk, acc[3]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D35, mk, acc[0]);
    acc[1] = fma(D50, mk, acc[1]);
    acc[2] = fma(D53, mk, acc[2]);
    acc[3] = fma(D54, mk, acc[3]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D37, mk, acc[0]);
    acc[1] = fma(D52, mk, acc[1]);
    acc[2] = fma(D55, mk, acc[2]);
    acc[3] = fma(D56, mk, acc[3]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D38, mk, acc[0]);
    acc[1] = fma(D53, mk, acc[1]);
    acc[2] = fma(D56, mk, acc[2]);
    acc[3] = fma(D57, mk, acc[3]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D40, mk, acc[0]);
    acc[1] = fma(D55, mk, acc[1]);
    acc[2] = fma(D58, mk, acc[2]);
    acc[3] = fma(D59, mk, acc[3]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D41, mk, acc[0]);
    acc[1] = fma(D56, mk, acc[1]);
    acc[2] = fma(D59, mk, acc[2]);
    acc[3] = fma(D60, mk, acc[3]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D43, mk, acc[0]);
    acc[1] = fma(D58, mk, acc[1]);
    acc[2] = fma(D61, mk, acc[2]);
    acc[3] = fma(D62, mk, acc[3]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D44, mk, acc[0]);
    acc[1] = fma(D59, mk, acc[1]);
    acc[2] = fma(D62, mk, acc[2]);
    acc[3] = fma(D63, mk, acc[3]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D46, mk, acc[0]);
  }
  { const T mk = Mb[36];
    acc[0] = fma(D47, mk, acc[0]);
  }
  { const T mk = Mb[37];
    acc[0] = fma(D48, mk, acc[0]);
  }
  { const T mk = Mb[38];
    acc[0] = fma(D49, mk, acc[0]);
  }
  { const T mk = Mb[39];
    acc[0] = fma(D50, mk, acc[0]);
  }
  { const T mk = Mb[40];
    acc[0] = fma(D52, mk, acc[0]);
  }
  { const T mk = Mb[41];
    acc[0] = fma(D53, mk, acc[0]);
  }
  { const T mk = Mb[42];
    acc[0] = fma(D55, mk, acc[0]);
  }
  { const T mk = Mb[43];
    acc[0] = fma(D56, mk, acc[0]);
  }
  { const T mk = Mb[44];
    acc[0] = fma(D58, mk, acc[0]);
  }
  { const T mk = Mb[45];
    acc[0] = fma(D59, mk, acc[0]);
  }
  { const T mk = Mb[46];
    acc[0] = fma(D61, mk, acc[0]);
  }
  { const T mk = Mb[47];
    acc[0] = fma(D62, mk, acc[0]);
  }
}
template <typename T>
__device__ __forceinline__ void dtensor_m1_p6(T x, T y, T z, T* __restrict__ Dout) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  const T w6_6 = crat<T>(-150, 6) * ir2;
  const T x6_1 = crat<T>(-11, 6) * xr;
  const T x6_6 = T(6) * x6_1;
  const T D46 = fma(x6_6, D31, w6_6 * D19);
  const T w6_5 = crat<T>(-100, 6) * ir2;
  const T x6_5 = T(5) * x6_1;
  const T y6_1 = crat<T>(-11, 6) * yr;
  const T D47 = fma(y6_1, D31, fma(x6_5, D32, w6_5 * D20));
  const T z6_1 = crat<T>(-11, 6) * zr;
  const T D48 = fma(z6_1, D31, fma(x6_5, D33, w6_5 * D21));
  const T w6_4 = crat<T>(-60, 6) * ir2;
  const T w6_2 = crat<T>(-10, 6) * ir2;
  const T x6_4 = T(4) * x6_1;
  const T y6_2 = T(2) * y6_1;
  const T D49 = fma(y6_2, D32, fma(x6_4, D34, fma(w6_2, D19, w6_4 * D22)));
  const T D50 = fma(z6_1, D32, fma(y6_1, D33, fma(x6_4, D35, w6_4 * D23)));
  const T D51 = -(D46 + D49);
  const T w6_3 = crat<T>(-30, 6) * ir2;
  const T x6_3 = T(3) * x6_1;
  const T y6_3 = T(3) * y6_1;
  const T D52 = fma(y6_3, D34, fma(x6_3, D37, fma(w6_3, D20, w6_3 * D25)));
  const T D53 = fma(z6_1, D34, fma(y6_2, D35, fma(x6_3, D38, fma(w6_2, D21, w6_3 * D26))));
  const T D54 = -(D47 + D52);
  const T x6_2 = T(2) * x6_1;
  const T y6_4 = T(4) * y6_1;
  const T D55 = fma(y6_4, D37, fma(x6_2, D40, fma(w6_4, D22, w6_2 * D28)));
  const T D56 = fma(z6_1, D37, fma(y6_3, D38, fma(x6_2, D41, fma(w6_3, D23, w6_2 * D29))));
  const T D57 = -(D49 + D55);
  const T y6_5 = T(5) * y6_1;
  const T D58 = fma(y6_5, D40, fma(x6_1, D43, w6_5 * D25));
  const T D59 = fma(z6_1, D40, fma(y6_4, D41, fma(x6_1, D44, w6_4 * D26)));
  const T D60 = -(D52 + D58);
  const T y6_6 = T(6) * y6_1;
  const T D61 = fma(y6_6, D43, w6_6 * D28);
  const T D62 = fma(z6_1, D43, fma(y6_5, D44, w6_5 * D29));
  const T D63 = -(D55 + D61);
  Dout[0] = D0;
  Dout[1] = D1;
  Dout[2] = D2;
  Dout[3] = D3;
  Dout[4] = D4;
  Dout[5] = D5;
  Dout[6] = D6;
  Dout[7] = D7;
  Dout[8] = D8;
  Dout[9] = D9;
  Dout[10] = D10;
  Dout[11] = D11;
  Dout[12] = D12;
  Dout[13] = D13;
  Dout[14] = D14;
  Dout[15] = D15;
  Dout[16] = D16;
  Dout[17] = D17;
  Dout[18] = D18;
  Dout[19] = D19;
  Dout[20] = D20;
  Dout[21] = D21;
  Dout[22] = D22;
  Dout[23] = D23;
  Dout[24] = D24;
  Dout[25] = D25;
  Dout[26] = D26;
  Dout[27] = D27;
  Dout[28] = D28;
  Dout[29] = D29;
  Dout[30] = D30;
  Dout[31] = D31;
  Dout[32] = D32;
  Dout[33] = D33;
  Dout[34] = D34;
  Dout[35] = D35;
  Dout[36] = D36;
  Dout[37] = D37;
  Dout[38] = D38;
  Dout[39] = D39;
  Dout[40] = D40;
  Dout[41] = D41;
  Dout[42] = D42;
  Dout[43] = D43;
  Dout[44] = D44;
  Dout[45] = D45;
  Dout[46] = D46;
  Dout[47] = D47;
  Dout[48] = D48;
  Dout[49] = D49;
  Dout[50] = D50;
  Dout[51] = D51;
  Dout[52] = D52;
  Dout[53] = D53;
  Dout[54] = D54;
  Dout[55] = D55;
  Dout[56] = D56;
  Dout[57] = D57;
  Dout[58] = D58;
  Dout[59] = D59;
  Dout[60] = D60;
  Dout[61] = D61;
  Dout[62] = D62;
  Dout[63] = D63;
}
template <typename T>
__device__ __forceinline__ void m2l_m1_p6_pre(const T* __restrict__ Dt, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T D0 = Dt[0];
  const T D1 = Dt[1];
  const T D2 = Dt[2];
  const T D3 = Dt[3];
  const T D4 = Dt[4];
  const T D5 = Dt[5];
  const T D6 = Dt[6];
  const T D7 = Dt[7];
  const T D8 = Dt[8];
  const T D9 = Dt[9];
  const T D10 = Dt[10];
  const T D11 = Dt[11];
  const T D12 = Dt[12];
  const T D13 = Dt[13];
  const T D14 = Dt[14];
  const T D15 = Dt[15];
  const T D16 = Dt[16];
  const T D17 = Dt[17];
  const T D18 = Dt[18];
  const T D19 = Dt[19];
  const T D20 = Dt[20];
  const T D21 = Dt[21];
  const T D22 = Dt[22];
  const T D23 = Dt[23];
  const T D24 = Dt[24];
  const T D25 = Dt[25];
  const T D26 = Dt[26];
  const T D27 = Dt[27];
  const T D28 = Dt[28];
  const T D29 = Dt[29];
  const T D30 = Dt[30];
  const T D31 = Dt[31];
  const T D32 = Dt[32];
  const T D33 = Dt[33];
  const T D34 = Dt[34];
  const T D35 = Dt[35];
  const T D36 = Dt[36];
  const T D37 = Dt[37];
  const T D38 = Dt[38];
  const T D39 = Dt[39];
  const T D40 = Dt[40];
  const T D41 = Dt[41];
  const T D42 = Dt[42];
  const T D43 = Dt[43];
  const T D44 = Dt[44];
  const T D45 = Dt[45];
  const T D46 = Dt[46];
  const T D47 = Dt[47];
  const T D48 = Dt[48];
  const T D49 = Dt[49];
  const T D50 = Dt[50];
  const T D51 = Dt[51];
  const T D52 = Dt[52];
  const T D53 = Dt[53];
  const T D54 = Dt[54];
  const T D55 = Dt[55];
  const T D56 = Dt[56];
  const T D57 = Dt[57];
  const T D58 = Dt[58];
  const T D59 = Dt[59];
  const T D60 = Dt[60];
  const T D61 = Dt[61];
  const T D62 = Dt[62];
  const T D63 = Dt[63];
  { const T mk = Mb[0];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
    acc[25] = fma(D46, mk, acc[25]);
    acc[26] = fma(D47, mk, acc[26]);
    acc[27] = fma(D48, mk, acc[27]);
    acc[28] = fma(D49, mk, acc[28]);
    acc[29] = fma(D50, mk, acc[29]);
    acc[30] = fma(D52, mk, acc[30]);
    acc[31] = fma(D53, mk, acc[31]);
    acc[32] = fma(D55, mk, acc[32]);
    acc[33] = fma(D56, mk, acc[33]);
    acc[34] = fma(D58, mk, acc[34]);
    acc[35] = fma(D59, mk, acc[35]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
    acc[25] = fma(D47, mk, acc[25]);
    acc[26] = fma(D49, mk, acc[26]);
    acc[27] = fma(D50, mk, acc[27]);
    acc[28] = fma(D52, mk, acc[28]);
    acc[29] = fma(D53, mk, acc[29]);
    acc[30] = fma(D55, mk, acc[30]);
    acc[31] = fma(D56, mk, acc[31]);
    acc[32] = fma(D58, mk, acc[32]);
    acc[33] = fma(D59, mk, acc[33]);
    acc[34] = fma(D61, mk, acc[34]);
    acc[35] = fma(D62, mk, acc[35]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
    acc[25] = fma(D48, mk, acc[25]);
    acc[26] = fma(D50, mk, acc[26]);
    acc[27] = fma(D51, mk, acc[27]);
    acc[28] = fma(D53, mk, acc[28]);
    acc[29] = fma(D54, mk, acc[29]);
    acc[30] = fma(D56, mk, acc[30]);
    acc[31] = fma(D57, mk, acc[31]);
    acc[32] = fma(D59, mk, acc[32]);
    acc[33] = fma(D60, mk, acc[33]);
    acc[34] = fma(D62, mk, acc[34]);
    acc[35] = fma(D63, mk, acc[35]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
    acc[16] = fma(D46, mk, acc[16]);
    acc[17] = fma(D47, mk, acc[17]);
    acc[18] = fma(D48, mk, acc[18]);
    acc[19] = fma(D49, mk, acc[19]);
    acc[20] = fma(D50, mk, acc[20]);
    acc[21] = fma(D52, mk, acc[21]);
    acc[22] = fma(D53, mk, acc[22]);
    acc[23] = fma(D55, mk, acc[23]);
    acc[24] = fma(D56, mk, acc[24]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
    acc[16] = fma(D47, mk, acc[16]);
    acc[17] = fma(D49, mk, acc[17]);
    acc[18] = fma(D50, mk, acc[18]);
    acc[19] = fma(D52, mk, acc[19]);
    acc[20] = fma(D53, mk, acc[20]);
    acc[21] = fma(D55, mk, acc[21]);
    acc[22] = fma(D56, mk, acc[22]);
    acc[23] = fma(D58, mk, acc[23]);
    acc[24] = fma(D59, mk, acc[24]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
    acc[16] = fma(D48, mk, acc[16]);
    acc[17] = fma(D50, mk, acc[17]);
    acc[18] = fma(D51, mk, acc[18]);
    acc[19] = fma(D53, mk, acc[19]);
    acc[20] = fma(D54, mk, acc[20]);
    acc[21] = fma(D56, mk, acc[21]);
    acc[22] = fma(D57, mk, acc[22]);
    acc[23] = fma(D59, mk, acc[23]);
    acc[24] = fma(D60, mk, acc[24]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
    acc[16] = fma(D49, mk, acc[16]);
    acc[17] = fma(D52, mk, acc[17]);
    acc[18] = fma(D53, mk, acc[18]);
    acc[19] = fma(D55, mk, acc[19]);
    acc[20] = fma(D56, mk, acc[20]);
    acc[21] = fma(D58, mk, acc[21]);
    acc[22] = fma(D59, mk, acc[22]);
    acc[23] = fma(D61, mk, acc[23]);
    acc[24] = fma(D62, mk, acc[24]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
    acc[16] = fma(D50, mk, acc[16]);
    acc[17] = fma(D53, mk, acc[17]);
    acc[18] = fma(D54, mk, acc[18]);
    acc[19] = fma(D56, mk, acc[19]);
    acc[20] = fma(D57, mk, acc[20]);
    acc[21] = fma(D59, mk, acc[21]);
    acc[22] = fma(D60, mk, acc[22]);
    acc[23] = fma(D62, mk, acc[23]);
    acc[24] = fma(D63, mk, acc[24]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
    acc[9] = fma(D46, mk, acc[9]);
    acc[10] = fma(D47, mk, acc[10]);
    acc[11] = fma(D48, mk, acc[11]);
    acc[12] = fma(D49, mk, acc[12]);
    acc[13] = fma(D50, mk, acc[13]);
    acc[14] = fma(D52, mk, acc[14]);
    acc[15] = fma(D53, mk, acc[15]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
    acc[9] = fma(D47, mk, acc[9]);
    acc[10] = fma(D49, mk, acc[10]);
    acc[11] = fma(D50, mk, acc[11]);
    acc[12] = fma(D52, mk, acc[12]);
    acc[13] = fma(D53, mk, acc[13]);
    acc[14] = fma(D55, mk, acc[14]);
    acc[15] = fma(D56, mk, acc[15]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
    acc[9] = fma(D48, mk, acc[9]);
    acc[10] = fma(D50, mk, acc[10]);
    acc[11] = fma(D51, mk, acc[11]);
    acc[12] = fma(D53, mk, acc[12]);
    acc[13] = fma(D54, mk, acc[13]);
    acc[14] = fma(D56, mk, acc[14]);
    acc[15] = fma(D57, mk, acc[15]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
    acc[9] = fma(D49, mk, acc[9]);
    acc[10] = fma(D52, mk, acc[10]);
    acc[11] = fma(D53, mk, acc[11]);
    acc[12] = fma(D55, mk, acc[12]);
    acc[13] = fma(D56, mk, acc[13]);
    acc[14] = fma(D58, mk, acc[14]);
    acc[15] = fma(D59, mk, acc[15]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
    acc[9] = fma(D50, mk, acc[9]);
    acc[10] = fma(D53, mk, acc[10]);
    acc[11] = fma(D54, mk, acc[11]);
    acc[12] = fma(D56, mk, acc[12]);
    acc[13] = fma(D57, mk, acc[13]);
    acc[14] = fma(D59, mk, acc[14]);
    acc[15] = fma(D60, mk, acc[15]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
    acc[9] = fma(D52, mk, acc[9]);
    acc[10] = fma(D55, mk, acc[10]);
    acc[11] = fma(D56, mk, acc[11]);
    acc[12] = fma(D58, mk, acc[12]);
    acc[13] = fma(D59, mk, acc[13]);
    acc[14] = fma(D61, mk, acc[14]);
    acc[15] = fma(D62, mk, acc[15]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
    acc[9] = fma(D53, mk, acc[9]);
    acc[10] = fma(D56, mk, acc[10]);
    acc[11] = fma(D57, mk, acc[11]);
    acc[12] = fma(D59, mk, acc[12]);
    acc[13] = fma(D60, mk, acc[13]);
    acc[14] = fma(D62, mk, acc[14]);
    acc[15] = fma(D63, mk, acc[15]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
    acc[4] = fma(D46, mk, acc[4]);
    acc[5] = fma(D47, mk, acc[5]);
    acc[6] = fma(D48, mk, acc[6]);
    acc[7] = fma(D49, mk, acc[7]);
    acc[8] = fma(D50, mk, acc[8]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
    acc[4] = fma(D47, mk, acc[4]);
    acc[5] = fma(D49, mk, acc[5]);
    acc[6] = fma(D50, mk, acc[6]);
    acc[7] = fma(D52, mk, acc[7]);
    acc[8] = fma(D53, mk, acc[8]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
    acc[4] = fma(D48, mk, acc[4]);
    acc[5] = fma(D50, mk, acc[5]);
    acc[6] = fma(D51, mk, acc[6]);
    acc[7] = fma(D53, mk, acc[7]);
    acc[8] = fma(D54, mk, acc[8]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
    acc[4] = fma(D49, mk, acc[4]);
    acc[5] = fma(D52, mk, acc[5]);
    acc[6] = fma(D53, mk, acc[6]);
    acc[7] = fma(D55, mk, acc[7]);
    acc[8] = fma(D56, mk, acc[8]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
    acc[4] = fma(D50, mk, acc[4]);
    acc[5] = fma(D53, mk, acc[5]);
    acc[6] = fma(D54, mk, acc[6]);
    acc[7] = fma(D56, mk, acc[7]);
    acc[8] = fma(D57, mk, acc[8]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
    acc[4] = fma(D52, mk, acc[4]);
    acc[5] = fma(D55, mk, acc[5]);
    acc[6] = fma(D56, mk, acc[6]);
    acc[7] = fma(D58, mk, acc[7]);
    acc[8] = fma(D59, mk, acc[8]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
    acc[4] = fma(D53, mk, acc[4]);
    acc[5] = fma(D56, mk, acc[5]);
    acc[6] = fma(D57, mk, acc[6]);
    acc[7] = fma(D59, mk, acc[7]);
    acc[8] = fma(D60, mk, acc[8]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
    acc[4] = fma(D55, mk, acc[4]);
    acc[5] = fma(D58, mk, acc[5]);
    acc[6] = fma(D59, mk, acc[6]);
    acc[7] = fma(D61, mk, acc[7]);
    acc[8] = fma(D62, mk, acc[8]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
    acc[4] = fma(D56, mk, acc[4]);
    acc[5] = fma(D59, mk, acc[5]);
    acc[6] = fma(D60, mk, acc[6]);
    acc[7] = fma(D62, mk, acc[7]);
    acc[8] = fma(D63, mk, acc[8]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D31, mk, acc[0]);
    acc[1] = fma(D46, mk, acc[1]);
    acc[2] = fma(D47, mk, acc[2]);
    acc[3] = fma(D48, mk, acc[3]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D32, mk, acc[0]);
    acc[1] = fma(D47, mk, acc[1]);
    acc[2] = fma(D49, mk, acc[2]);
    acc[3] = fma(D50, mk, acc[3]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D33, mk, acc[0]);
    acc[1] = fma(D48, mk, acc[1]);
    acc[2] = fma(D50, mk, acc[2]);
    acc[3] = fma(D51, mk, acc[3]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D34, mk, acc[0]);
    acc[1] = fma(D49, mk, acc[1]);
    acc[2] = fma(D52, mk, acc[2]);
    acc[3] = fma(D53, mk, acc[3]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D35, mk, acc[0]);
    acc[1] = fma(D50, mk, acc[1]);
    acc[2] = fma(D53, mk, acc[2]);
    acc[3] = fma(D54, mk, acc[3]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D37, mk, acc[0]);
    acc[1] = fma(D52, mk, acc[1]);
    acc[2] = fma(D55, mk, acc[2]);
    acc[3] = fma(D56, mk, acc[3]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D38, mk, acc[0]);
    acc[1] = fma(D53, mk, acc[1]);
    acc[2] = fma(D56, mk, acc[2]);
    acc[3] = fma(D57, mk, acc[3]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D40, mk, acc[0]);
    acc[1] = fma(D55, mk, acc[1]);
    acc[2] = fma(D58, mk, acc[2]);
    acc[3] = fma(D59, mk, acc[3]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D41, mk, acc[0]);
    acc[1] = fma(D56, mk, acc[1]);
    acc[2] = fma(D59, mk, acc[2]);
    acc[3] = fma(D60, mk, acc[3]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D43, mk, acc[0]);
    acc[1] = fma(D58, mk, acc[1]);
    acc[2] = fma(D61, mk, acc[2]);
    acc[3] = fma(D62, mk, acc[3]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D44, mk, acc[0]);
    acc[1] = fma(D59, mk, acc[1]);
    acc[2] = fma(D62, mk, acc[2]);
    acc[3] = fma(D63, mk, acc[3]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D46, mk, acc[0]);
  }
  { const T mk = Mb[36];
    acc[0] = fma(D47, mk, acc[0]);
  }
  { const T mk = Mb[37];
    acc[0] = fma(D48, mk, acc[0]);
  }
  { const T mk = Mb[38];
    acc[0] = fma(D49, mk, acc[0]);
  }
  { const T mk = Mb[39];
    acc[0] = fma(D50, mk, acc[0]);
  }
  { const T mk = Mb[40];
    acc[0] = fma(D52, mk, acc[0]);
  }
  { const T mk = Mb[41];
    acc[0] = fma(D53, mk, acc[0]);
  }
  { const T mk = Mb[42];
    acc[0] = fma(D55, mk, acc[0]);
  }
  { const T mk = Mb[43];
    acc[0] = fma(D56, mk, acc[0]);
  }
  { const T mk = Mb[44];
    acc[0] = fma(D58, mk, acc[0]);
  }
  { const T mk = Mb[45];
    acc[0] = fma(D59, mk, acc[0]);
  }
  { const T mk = Mb[46];
    acc[0] = fma(D61, mk, acc[0]);
  }
  { const T mk = Mb[47];
    acc[0] = fma(D62, mk, acc[0]);
  }
}
static __constant__ unsigned char m2l_w_m1_p6[483] = {
  1, 4, 5, 6, 10, 11, 12, 13, 14, 19, 20, 21, 22, 23, 25, 26, 31, 32, 33, 34, 35, 37, 38, 40, 41, 46, 47, 48, 49, 50, 52, 53, 55, 56, 58, 59, 2, 5, 7, 8, 11, 13, 14, 16, 17, 20, 22, 23, 25, 26, 28, 29, 32, 34, 35, 37, 38, 40, 41, 43, 44, 47, 49, 50, 52, 53, 55, 56, 58, 59, 61, 62, 3, 6, 8, 9, 12, 14, 15, 17, 18, 21, 23, 24, 26, 27, 29, 30, 33, 35, 36, 38, 39, 41, 42, 44, 45, 48, 50, 51, 53, 54, 56, 57, 59, 60, 62, 63, 4, 10, 11, 12, 19, 20, 21, 22, 23, 31, 32, 33, 34, 35, 37, 38, 46, 47, 48, 49, 50, 52, 53, 55, 56, 5, 11, 13, 14, 20, 22, 23, 25, 26, 32, 34, 35, 37, 38, 40, 41, 47, 49, 50, 52, 53, 55, 56, 58, 59, 6, 12, 14, 15, 21, 23, 24, 26, 27, 33, 35, 36, 38, 39, 41, 42, 48, 50, 51, 53, 54, 56, 57, 59, 60, 7, 13, 16, 17, 22, 25, 26, 28, 29, 34, 37, 38, 40, 41, 43, 44, 49, 52, 53, 55, 56, 58, 59, 61, 62, 8, 14, 17, 18, 23, 26, 27, 29, 30, 35, 38, 39, 41, 42, 44, 45, 50, 53, 54, 56, 57, 59, 60, 62, 63, 10, 19, 20, 21, 31, 32, 33, 34, 35, 46, 47, 48, 49, 50, 52, 53, 11, 20, 22, 23, 32, 34, 35, 37, 38, 47, 49, 50, 52, 53, 55, 56, 12, 21, 23, 24, 33, 35, 36, 38, 39, 48, 50, 51, 53, 54, 56, 57, 13, 22, 25, 26, 34, 37, 38, 40, 41, 49, 52, 53, 55, 56, 58, 59, 14, 23, 26, 27, 35, 38, 39, 41, 42, 50, 53, 54, 56, 57, 59, 60, 16, 25, 28, 29, 37, 40, 41, 43, 44, 52, 55, 56, 58, 59, 61, 62, 17, 26, 29, 30, 38, 41, 42, 44, 45, 53, 56, 57, 59, 60, 62, 63, 19, 31, 32, 33, 46, 47, 48, 49, 50, 20, 32, 34, 35, 47, 49, 50, 52, 53, 21, 33, 35, 36, 48, 50, 51, 53, 54, 22, 34, 37, 38, 49, 52, 53, 55, 56, 23, 35, 38, 39, 50, 53, 54, 56, 57, 25, 37, 40, 41, 52, 55, 56, 58, 59, 26, 38, 41, 42, 53, 56, 57, 59, 60, 28, 40, 43, 44, 55, 58, 59, 61, 62, 29, 41, 44, 45, 56, 59, 60, 62, 63, 31, 46, 47, 48, 32, 47, 49, 50, 33, 48, 50, 51, 34, 49, 52, 53, 35, 50, 53, 54, 37, 52, 55, 56, 38, 53, 56, 57, 40, 55, 58, 59, 41, 56, 59, 60, 43, 58, 61, 62, 44, 59, 62, 63, 46, 47, 48, 49, 50, 52, 53, 55, 56, 58, 59, 61, 62};
static __device__ const signed char m2l_fold_m1_p6[48][6][2] = {
  {{0, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {8, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {8, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{9, 1}, {14, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{10, 1}, {17, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{11, 1}, {18, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{12, 1}, {14, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{15, 1}, {17, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{16, 1}, {18, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{19, 1}, {24, -1}, {33, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{20, 1}, {27, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{21, 1}, {28, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{22, 1}, {24, -1}, {31, -1}, {33, 2}, {0, 0}, {0, 0}},
  {{23, 1}, {32, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{25, 1}, {27, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{26, 1}, {28, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{29, 1}, {31, -1}, {33, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{30, 1}, {32, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{34, 1}, {39, -1}, {48, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{35, 1}, {42, -1}, {53, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{36, 1}, {43, -1}, {54, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{37, 1}, {39, -1}, {46, -1}, {48, 2}, {0, 0}, {0, 0}},
  {{38, 1}, {47, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{40, 1}, {42, -1}, {51, -1}, {53, 2}, {0, 0}, {0, 0}},
  {{41, 1}, {43, -1}, {52, -1}, {54, 2}, {0, 0}, {0, 0}},
  {{44, 1}, {46, -1}, {48, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{45, 1}, {47, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{49, 1}, {51, -1}, {53, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{50, 1}, {52, -1}, {54, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{55, 1}, {60, -1}, {69, 1}, {82, -1}, {0, 0}, {0, 0}},
  {{56, 1}, {63, -1}, {74, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{57, 1}, {64, -1}, {75, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{58, 1}, {60, -1}, {67, -1}, {69, 2}, {80, 1}, {82, -3}},
  {{59, 1}, {68, -1}, {81, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{61, 1}, {63, -1}, {72, -1}, {74, 2}, {0, 0}, {0, 0}},
  {{62, 1}, {64, -1}, {73, -1}, {75, 2}, {0, 0}, {0, 0}},
  {{65, 1}, {67, -1}, {69, 1}, {78, -1}, {80, 2}, {82, -3}},
  {{66, 1}, {68, -1}, {79, -1}, {81, 2}, {0, 0}, {0, 0}},
  {{70, 1}, {72, -1}, {74, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{71, 1}, {73, -1}, {75, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{76, 1}, {78, -1}, {80, 1}, {82, -1}, {0, 0}, {0, 0}},
  {{77, 1}, {79, -1}, {81, 1}, {0, 0}, {0, 0}, {0, 0}},
};
static __device__ const signed char m2l_unfold_m1_p6[56][3][2] = {
  {{0, 1}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}},
  {{7, -1}, {4, -1}, {0, 0}},
  {{9, 1}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}},
  {{11, 1}, {0, 0}, {0, 0}},
  {{12, 1}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}},
  {{12, -1}, {9, -1}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}},
  {{15, 1}, {0, 0}, {0, 0}},
  {{14, -1}, {10, -1}, {0, 0}},
  {{15, -1}, {11, -1}, {0, 0}},
  {{16, 1}, {0, 0}, {0, 0}},
  {{17, 1}, {0, 0}, {0, 0}},
  {{18, 1}, {0, 0}, {0, 0}},
  {{19, 1}, {0, 0}, {0, 0}},
  {{20, 1}, {0, 0}, {0, 0}},
  {{19, -1}, {16, -1}, {0, 0}},
  {{21, 1}, {0, 0}, {0, 0}},
  {{22, 1}, {0, 0}, {0, 0}},
  {{21, -1}, {17, -1}, {0, 0}},
  {{22, -1}, {18, -1}, {0, 0}},
  {{23, 1}, {0, 0}, {0, 0}},
  {{24, 1}, {0, 0}, {0, 0}},
  {{23, -1}, {19, -1}, {0, 0}},
  {{24, -1}, {20, -1}, {0, 0}},
  {{23, 1}, {19, 2}, {16, 1}},
  {{25, 1}, {0, 0}, {0, 0}},
  {{26, 1}, {0, 0}, {0, 0}},
  {{27, 1}, {0, 0}, {0, 0}},
  {{28, 1}, {0, 0}, {0, 0}},
  {{29, 1}, {0, 0}, {0, 0}},
  {{28, -1}, {25, -1}, {0, 0}},
  {{30, 1}, {0, 0}, {0, 0}},
  {{31, 1}, {0, 0}, {0, 0}},
  {{30, -1}, {26, -1}, {0, 0}},
  {{31, -1}, {27, -1}, {0, 0}},
  {{32, 1}, {0, 0}, {0, 0}},
  {{33, 1}, {0, 0}, {0, 0}},
  {{32, -1}, {28, -1}, {0, 0}},
  {{33, -1}, {29, -1}, {0, 0}},
  {{32, 1}, {28, 2}, {25, 1}},
  {{34, 1}, {0, 0}, {0, 0}},
  {{35, 1}, {0, 0}, {0, 0}},
  {{34, -1}, {30, -1}, {0, 0}},
  {{35, -1}, {31, -1}, {0, 0}},
  {{34, 1}, {30, 2}, {26, 1}},
  {{35, 1}, {31, 2}, {27, 1}},
};

// M2L between reduced coefficients, source order 0, expansion order 5: 36 multipole, 36 local, 46 tensor entries, 301 terms
template <typename T>
__device__ __forceinline__ void m2l_m0_p5(T x, T y, T z, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  { const T mk = Mb[0];
    acc[0] = fma(D0, mk, acc[0]);
    acc[1] = fma(D1, mk, acc[1]);
    acc[2] = fma(D2, mk, acc[2]);
    acc[3] = fma(D3, mk, acc[3]);
    acc[4] = fma(D4, mk, acc[4]);
    acc[5] = fma(D5, mk, acc[5]);
    acc[6] = fma(D6, mk, acc[6]);
    acc[7] = fma(D7, mk, acc[7]);
    acc[8] = fma(D8, mk, acc[8]);
    acc[9] = fma(D10, mk, acc[9]);
    acc[10] = fma(D11, mk, acc[10]);
    acc[11] = fma(D12, mk, acc[11]);
    acc[12] = fma(D13, mk, acc[12]);
    acc[13] = fma(D14, mk, acc[13]);
    acc[14] = fma(D16, mk, acc[14]);
    acc[15] = fma(D17, mk, acc[15]);
    acc[16] = fma(D19, mk, acc[16]);
    acc[17] = fma(D20, mk, acc[17]);
    acc[18] = fma(D21, mk, acc[18]);
    acc[19] = fma(D22, mk, acc[19]);
    acc[20] = fma(D23, mk, acc[20]);
    acc[21] = fma(D25, mk, acc[21]);
    acc[22] = fma(D26, mk, acc[22]);
    acc[23] = fma(D28, mk, acc[23]);
    acc[24] = fma(D29, mk, acc[24]);
    acc[25] = fma(D31, mk, acc[25]);
    acc[26] = fma(D32, mk, acc[26]);
    acc[27] = fma(D33, mk, acc[27]);
    acc[28] = fma(D34, mk, acc[28]);
    acc[29] = fma(D35, mk, acc[29]);
    acc[30] = fma(D37, mk, acc[30]);
    acc[31] = fma(D38, mk, acc[31]);
    acc[32] = fma(D40, mk, acc[32]);
    acc[33] = fma(D41, mk, acc[33]);
    acc[34] = fma(D43, mk, acc[34]);
    acc[35] = fma(D44, mk, acc[35]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D31, mk, acc[0]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D32, mk, acc[0]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D33, mk, acc[0]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D34, mk, acc[0]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D35, mk, acc[0]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D37, mk, acc[0]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D38, mk, acc[0]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D40, mk, acc[0]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D41, mk, acc[0]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D43, mk, acc[0]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D44, mk, acc[0]);
  }
}
template <typename T>
__device__ __forceinline__ void dtensor_m0_p5(T x, T y, T z, T* __restrict__ Dout) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  Dout[0] = D0;
  Dout[1] = D1;
  Dout[2] = D2;
  Dout[3] = D3;
  Dout[4] = D4;
  Dout[5] = D5;
  Dout[6] = D6;
  Dout[7] = D7;
  Dout[8] = D8;
  Dout[9] = D9;
  Dout[10] = D10;
  Dout[11] = D11;
  Dout[12] = D12;
  Dout[13] = D13;
  Dout[14] = D14;
  Dout[15] = D15;
  Dout[16] = D16;
  Dout[17] = D17;
  Dout[18] = D18;
  Dout[19] = D19;
  Dout[20] = D20;
  Dout[21] = D21;
  Dout[22] = D22;
  Dout[23] = D23;
  Dout[24] = D24;
  Dout[25] = D25;
  Dout[26] = D26;
  Dout[27] = D27;
  Dout[28] = D28;
  Dout[29] = D29;
  Dout[30] = D30;
  Dout[31] = D31;
  Dout[32] = D32;
  Dout[33] = D33;
  Dout[34] = D34;
  Dout[35] = D35;
  Dout[36] = D36;
  Dout[37] = D37;
  Dout[38] = D38;
  Dout[39] = D39;
  Dout[40] = D40;
  Dout[41] = D41;
  Dout[42] = D42;
  Dout[43] = D43;
  Dout[44] = D44;
  Dout[45] = D45;
}
template <typename T>
__device__ __forceinline__ void m2l_m0_p5_pre(const T* __restrict__ Dt, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T D0 = Dt[0];
  const T D1 = Dt[1];
  const T D2 = Dt[2];
  const T D3 = Dt[3];
  const T D4 = Dt[4];
  const T D5 = Dt[5];
  const T D6 = Dt[6];
  const T D7 = Dt[7];
  const T D8 = Dt[8];
  const T D9 = Dt[9];
  const T D10 = Dt[10];
  const T D11 = Dt[11];
  const T D12 = Dt[12];
  const T D13 = Dt[13];
  const T D14 = Dt[14];
  const T D15 = Dt[15];
  const T D16 = Dt[16];
  const T D17 = Dt[17];
  const T D18 = Dt[18];
  const T D19 = Dt[19];
  const T D20 = Dt[20];
  const T D21 = Dt[21];
  const T D22 = Dt[22];
  const T D23 = Dt[23];
  const T D24 = Dt[24];
  const T D25 = Dt[25];
  const T D26 = Dt[26];
  const T D27 = Dt[27];
  const T D28 = Dt[28];
  const T D29 = Dt[29];
  const T D30 = Dt[30];
  const T D31 = Dt[31];
  const T D32 = Dt[32];
  const T D33 = Dt[33];
  const T D34 = Dt[34];
  const T D35 = Dt[35];
  const T D36 = Dt[36];
  const T D37 = Dt[37];
  const T D38 = Dt[38];
  const T D39 = Dt[39];
  const T D40 = Dt[40];
  const T D41 = Dt[41];
  const T D42 = Dt[42];
  const T D43 = Dt[43];
  const T D44 = Dt[44];
  const T D45 = Dt[45];
  { const T mk = Mb[0];
    acc[0] = fma(D0, mk, acc[0]);
    acc[1] = fma(D1, mk, acc[1]);
    acc[2] = fma(D2, mk, acc[2]);
    acc[3] = fma(D3, mk, acc[3]);
    acc[4] = fma(D4, mk, acc[4]);
    acc[5] = fma(D5, mk, acc[5]);
    acc[6] = fma(D6, mk, acc[6]);
    acc[7] = fma(D7, mk, acc[7]);
    acc[8] = fma(D8, mk, acc[8]);
    acc[9] = fma(D10, mk, acc[9]);
    acc[10] = fma(D11, mk, acc[10]);
    acc[11] = fma(D12, mk, acc[11]);
    acc[12] = fma(D13, mk, acc[12]);
    acc[13] = fma(D14, mk, acc[13]);
    acc[14] = fma(D16, mk, acc[14]);
    acc[15] = fma(D17, mk, acc[15]);
    acc[16] = fma(D19, mk, acc[16]);
    acc[17] = fma(D20, mk, acc[17]);
    acc[18] = fma(D21, mk, acc[18]);
    acc[19] = fma(D22, mk, acc[19]);
    acc[20] = fma(D23, mk, acc[20]);
    acc[21] = fma(D25, mk, acc[21]);
    acc[22] = fma(D26, mk, acc[22]);
    acc[23] = fma(D28, mk, acc[23]);
    acc[24] = fma(D29, mk, acc[24]);
    acc[25] = fma(D31, mk, acc[25]);
    acc[26] = fma(D32, mk, acc[26]);
    acc[27] = fma(D33, mk, acc[27]);
    acc[28] = fma(D34, mk, acc[28]);
    acc[29] = fma(D35, mk, acc[29]);
    acc[30] = fma(D37, mk, acc[30]);
    acc[31] = fma(D38, mk, acc[31]);
    acc[32] = fma(D40, mk, acc[32]);
    acc[33] = fma(D41, mk, acc[33]);
    acc[34] = fma(D43, mk, acc[34]);
    acc[35] = fma(D44, mk, acc[35]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D31, mk, acc[0]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D32, mk, acc[0]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D33, mk, acc[0]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D34, mk, acc[0]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D35, mk, acc[0]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D37, mk, acc[0]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D38, mk, acc[0]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D40, mk, acc[0]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D41, mk, acc[0]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D43, mk, acc[0]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D44, mk, acc[0]);
  }
}
static __constant__ unsigned char m2l_w_m0_p5[301] = {
  0, 1, 2, 3, 4, 5, 6, 7, 8, 10, 11, 12, 13, 14, 16, 17, 19, 20, 21, 22, 23, 25, 26, 28, 29, 31, 32, 33, 34, 35, 37, 38, 40, 41, 43, 44, 1, 4, 5, 6, 10, 11, 12, 13, 14, 19, 20, 21, 22, 23, 25, 26, 31, 32, 33, 34, 35, 37, 38, 40, 41, 2, 5, 7, 8, 11, 13, 14, 16, 17, 20, 22, 23, 25, 26, 28, 29, 32, 34, 35, 37, 38, 40, 41, 43, 44, 3, 6, 8, 9, 12, 14, 15, 17, 18, 21, 23, 24, 26, 27, 29, 30, 33, 35, 36, 38, 39, 41, 42, 44, 45, 4, 10, 11, 12, 19, 20, 21, 22, 23, 31, 32, 33, 34, 35, 37, 38, 5, 11, 13, 14, 20, 22, 23, 25, 26, 32, 34, 35, 37, 38, 40, 41, 6, 12, 14, 15, 21, 23, 24, 26, 27, 33, 35, 36, 38, 39, 41, 42, 7, 13, 16, 17, 22, 25, 26, 28, 29, 34, 37, 38, 40, 41, 43, 44, 8, 14, 17, 18, 23, 26, 27, 29, 30, 35, 38, 39, 41, 42, 44, 45, 10, 19, 20, 21, 31, 32, 33, 34, 35, 11, 20, 22, 23, 32, 34, 35, 37, 38, 12, 21, 23, 24, 33, 35, 36, 38, 39, 13, 22, 25, 26, 34, 37, 38, 40, 41, 14, 23, 26, 27, 35, 38, 39, 41, 42, 16, 25, 28, 29, 37, 40, 41, 43, 44, 17, 26, 29, 30, 38, 41, 42, 44, 45, 19, 31, 32, 33, 20, 32, 34, 35, 21, 33, 35, 36, 22, 34, 37, 38, 23, 35, 38, 39, 25, 37, 40, 41, 26, 38, 41, 42, 28, 40, 43, 44, 29, 41, 44, 45, 31, 32, 33, 34, 35, 37, 38, 40, 41, 43, 44};
static __device__ const signed char m2l_fold_m0_p5[36][4][2] = {
  {{0, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{4, 1}, {9, -1}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{7, 1}, {9, -1}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{10, 1}, {15, -1}, {0, 0}, {0, 0}},
  {{11, 1}, {18, -1}, {0, 0}, {0, 0}},
  {{12, 1}, {19, -1}, {0, 0}, {0, 0}},
  {{13, 1}, {15, -1}, {0, 0}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{16, 1}, {18, -1}, {0, 0}, {0, 0}},
  {{17, 1}, {19, -1}, {0, 0}, {0, 0}},
  {{20, 1}, {25, -1}, {34, 1}, {0, 0}},
  {{21, 1}, {28, -1}, {0, 0}, {0, 0}},
  {{22, 1}, {29, -1}, {0, 0}, {0, 0}},
  {{23, 1}, {25, -1}, {32, -1}, {34, 2}},
  {{24, 1}, {33, -1}, {0, 0}, {0, 0}},
  {{26, 1}, {28, -1}, {0, 0}, {0, 0}},
  {{27, 1}, {29, -1}, {0, 0}, {0, 0}},
  {{30, 1}, {32, -1}, {34, 1}, {0, 0}},
  {{31, 1}, {33, -1}, {0, 0}, {0, 0}},
  {{35, 1}, {40, -1}, {49, 1}, {0, 0}},
  {{36, 1}, {43, -1}, {54, 1}, {0, 0}},
  {{37, 1}, {44, -1}, {55, 1}, {0, 0}},
  {{38, 1}, {40, -1}, {47, -1}, {49, 2}},
  {{39, 1}, {48, -1}, {0, 0}, {0, 0}},
  {{41, 1}, {43, -1}, {52, -1}, {54, 2}},
  {{42, 1}, {44, -1}, {53, -1}, {55, 2}},
  {{45, 1}, {47, -1}, {49, 1}, {0, 0}},
  {{46, 1}, {48, -1}, {0, 0}, {0, 0}},
  {{50, 1}, {52, -1}, {54, 1}, {0, 0}},
  {{51, 1}, {53, -1}, {55, 1}, {0, 0}},
};
static __device__ const signed char m2l_unfold_m0_p5[56][3][2] = {
  {{0, 1}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}},
  {{7, -1}, {4, -1}, {0, 0}},
  {{9, 1}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}},
  {{11, 1}, {0, 0}, {0, 0}},
  {{12, 1}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}},
  {{12, -1}, {9, -1}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}},
  {{15, 1}, {0, 0}, {0, 0}},
  {{14, -1}, {10, -1}, {0, 0}},
  {{15, -1}, {11, -1}, {0, 0}},
  {{16, 1}, {0, 0}, {0, 0}},
  {{17, 1}, {0, 0}, {0, 0}},
  {{18, 1}, {0, 0}, {0, 0}},
  {{19, 1}, {0, 0}, {0, 0}},
  {{20, 1}, {0, 0}, {0, 0}},
  {{19, -1}, {16, -1}, {0, 0}},
  {{21, 1}, {0, 0}, {0, 0}},
  {{22, 1}, {0, 0}, {0, 0}},
  {{21, -1}, {17, -1}, {0, 0}},
  {{22, -1}, {18, -1}, {0, 0}},
  {{23, 1}, {0, 0}, {0, 0}},
  {{24, 1}, {0, 0}, {0, 0}},
  {{23, -1}, {19, -1}, {0, 0}},
  {{24, -1}, {20, -1}, {0, 0}},
  {{23, 1}, {19, 2}, {16, 1}},
  {{25, 1}, {0, 0}, {0, 0}},
  {{26, 1}, {0, 0}, {0, 0}},
  {{27, 1}, {0, 0}, {0, 0}},
  {{28, 1}, {0, 0}, {0, 0}},
  {{29, 1}, {0, 0}, {0, 0}},
  {{28, -1}, {25, -1}, {0, 0}},
  {{30, 1}, {0, 0}, {0, 0}},
  {{31, 1}, {0, 0}, {0, 0}},
  {{30, -1}, {26, -1}, {0, 0}},
  {{31, -1}, {27, -1}, {0, 0}},
  {{32, 1}, {0, 0}, {0, 0}},
  {{33, 1}, {0, 0}, {0, 0}},
  {{32, -1}, {28, -1}, {0, 0}},
  {{33, -1}, {29, -1}, {0, 0}},
  {{32, 1}, {28, 2}, {25, 1}},
  {{34, 1}, {0, 0}, {0, 0}},
  {{35, 1}, {0, 0}, {0, 0}},
  {{34, -1}, {30, -1}, {0, 0}},
  {{35, -1}, {31, -1}, {0, 0}},
  {{34, 1}, {30, 2}, {26, 1}},
  {{35, 1}, {31, 2}, {27, 1}},
};

// M2L between reduced coefficients, source order 0, expansion order 6: 49 multipole, 49 local, 64 tensor entries, 532 terms
template <typename T>
__device__ __forceinline__ void m2l_m0_p6(T x, T y, T z, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  const T w6_6 = crat<T>(-150, 6) * ir2;
  const T x6_1 = crat<T>(-11, 6) * xr;
  const T x6_6 = T(6) * x6_1;
  const T D46 = fma(x6_6, D31, w6_6 * D19);
  const T w6_5 = crat<T>(-100, 6) * ir2;
  const T x6_5 = T(5) * x6_1;
  const T y6_1 = crat<T>(-11, 6) * yr;
  const T D47 = fma(y6_1, D31, fma(x6_5, D32, w6_5 * D20));
  const T z6_1 = crat<T>(-11, 6) * zr;
  const T D48 = fma(z6_1, D31, fma(x6_5, D33, w6_5 * D21));
  const T w6_4 = crat<T>(-60, 6) * ir2;
  const T w6_2 = crat<T>(-10, 6) * ir2;
  const T x6_4 = T(4) * x6_1;
  const T y6_2 = T(2) * y6_1;
  const T D49 = fma(y6_2, D32, fma(x6_4, D34, fma(w6_2, D19, w6_4 * D22)));
  const T D50 = fma(z6_1, D32, fma(y6_1, D33, fma(x6_4, D35, w6_4 * D23)));
  const T D51 = -(D46 + D49);
  const T w6_3 = crat<T>(-30, 6) * ir2;
  const T x6_3 = T(3) * x6_1;
  const T y6_3 = T(3) * y6_1;
  const T D52 = fma(y6_3, D34, fma(x6_3, D37, fma(w6_3, D20, w6_3 * D25)));
  const T D53 = fma(z6_1, D34, fma(y6_2, D35, fma(x6_3, D38, fma(w6_2, D21, w6_3 * D26))));
  const T D54 = -(D47 + D52);
  const T x6_2 = T(2) * x6_1;
  const T y6_4 = T(4) * y6_1;
  const T D55 = fma(y6_4, D37, fma(x6_2, D40, fma(w6_4, D22, w6_2 * D28)));
  const T D56 = fma(z6_1, D37, fma(y6_3, D38, fma(x6_2, D41, fma(w6_3, D23, w6_2 * D29))));
  const T D57 = -(D49 + D55);
  const T y6_5 = T(5) * y6_1;
  const T D58 = fma(y6_5, D40, fma(x6_1, D43, w6_5 * D25));
  const T D59 = fma(z6_1, D40, fma(y6_4, D41, fma(x6_1, D44, w6_4 * D26)));
  const T D60 = -(D52 + D58);
  const T y6_6 = T(6) * y6_1;
  const T D61 = fma(y6_6, D43, w6_6 * D28);
  const T D62 = fma(z6_1, D43, fma(y6_5, D44, w6_5 * D29));
  const T D63 = -(D55 + D61);
  { const T mk = Mb[0];
    acc[0] = fma(D0, mk, acc[0]);
    acc[1] = fma(D1, mk, acc[1]);
    acc[2] = fma(D2, mk, acc[2]);
    acc[3] = fma(D3, mk, acc[3]);
    acc[4] = fma(D4, mk, acc[4]);
    acc[5] = fma(D5, mk, acc[5]);
    acc[6] = fma(D6, mk, acc[6]);
    acc[7] = fma(D7, mk, acc[7]);
    acc[8] = fma(D8, mk, acc[8]);
    acc[9] = fma(D10, mk, acc[9]);
    acc[10] = fma(D11, mk, acc[10]);
    acc[11] = fma(D12, mk, acc[11]);
    acc[12] = fma(D13, mk, acc[12]);
    acc[13] = fma(D14, mk, acc[13]);
    acc[14] = fma(D16, mk, acc[14]);
    acc[15] = fma(D17, mk, acc[15]);
    acc[16] = fma(D19, mk, acc[16]);
    acc[17] = fma(D20, mk, acc[17]);
    acc[18] = fma(D21, mk, acc[18]);
    acc[19] = fma(D22, mk, acc[19]);
    acc[20] = fma(D23, mk, acc[20]);
    acc[21] = fma(D25, mk, acc[21]);
    acc[22] = fma(D26, mk, acc[22]);
    acc[23] = fma(D28, mk, acc[23]);
    acc[24] = fma(D29, mk, acc[24]);
    acc[25] = fma(D31, mk, acc[25]);
    acc[26] = fma(D32, mk, acc[26]);
    acc[27] = fma(D33, mk, acc[27]);
    acc[28] = fma(D34, mk, acc[28]);
    acc[29] = fma(D35, mk, acc[29]);
    acc[30] = fma(D37, mk, acc[30]);
    acc[31] = fma(D38, mk, acc[31]);
    acc[32] = fma(D40, mk, acc[32]);
    acc[33] = fma(D41, mk, acc[33]);
    acc[34] = fma(D43, mk, acc[34]);
    acc[35] = fma(D44, mk, acc[35]);
    acc[36] = fma(D46, mk, acc[36]);
    acc[37] = fma(D47, mk, acc[37]);
    acc[38] = fma(D48, mk, acc[38]);
    acc[39] = fma(D49, mk, acc[39]);
    acc[40] = fma(D50, mk, acc[40]);
    acc[41] = fma(D52, mk, acc[41]);
    acc[42] = fma(D53, mk, acc[42]);
    acc[43] = fma(D55, mk, acc[43]);
    acc[44] = fma(D56, mk, acc[44]);
    acc[45] = fma(D58, mk, acc[45]);
    acc[46] = fma(D59, mk, acc[46]);
    acc[47] = fma(D61, mk, acc[47]);
    acc[48] = fma(D62, mk, acc[48]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
    acc[25] = fma(D46, mk, acc[25]);
    acc[26] = fma(D47, mk, acc[26]);
    acc[27] = fma(D48, mk, acc[27]);
    acc[28] = fma(D49, mk, acc[28]);
    acc[29] = fma(D50, mk, acc[29]);
    acc[30] = fma(D52, mk, acc[30]);
    acc[31] = fma(D53, mk, acc[31]);
    acc[32] = fma(D55, mk, acc[32]);
    acc[33] = fma(D56, mk, acc[33]);
    acc[34] = fma(D58, mk, acc[34]);
    acc[35] = fma(D59, mk, acc[35]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
    acc[25] = fma(D47, mk, acc[25]);
    acc[26] = fma(D49, mk, acc[26]);
    acc[27] = fma(D50, mk, acc[27]);
    acc[28] = fma(D52, mk, acc[28]);
    acc[29] = fma(D53, mk, acc[29]);
    acc[30] = fma(D55, mk, acc[30]);
    acc[31] = fma(D56, mk, acc[31]);
    acc[32] = fma(D58, mk, acc[32]);
    acc[33] = fma(D59, mk, acc[33]);
    acc[34] = fma(D61, mk, acc[34]);
    acc[35] = fma(D62, mk, acc[35]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
    acc[25] = fma(D48, mk, acc[25]);
    acc[26] = fma(D50, mk, acc[26]);
    acc[27] = fma(D51, mk, acc[27]);
    acc[28] = fma(D53, mk, acc[28]);
    acc[29] = fma(D54, mk, acc[29]);
    acc[30] = fma(D56, mk, acc[30]);
    acc[31] = fma(D57, mk, acc[31]);
    acc[32] = fma(D59, mk, acc[32]);
    acc[33] = fma(D60, mk, acc[33]);
    acc[34] = fma(D62, mk, acc[34]);
    acc[35] = fma(D63, mk, acc[35]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
    acc[16] = fma(D46, mk, acc[16]);
    acc[17] = fma(D47, mk, acc[17]);
    acc[18] = fma(D48, mk, acc[18]);
    acc[19] = fma(D49, mk, acc[19]);
    acc[20] = fma(D50, mk, acc[20]);
    acc[21] = fma(D52, mk, acc[21]);
    acc[22] = fma(D53, mk, acc[22]);
    acc[23] = fma(D55, mk, acc[23]);
    acc[24] = fma(D56, mk, acc[24]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
    acc[16] = fma(D47, mk, acc[16]);
    acc[17] = fma(D49, mk, acc[17]);
    acc[18] = fma(D50, mk, acc[18]);
    acc[19] = fma(D52, mk, acc[19]);
    acc[20] = fma(D53, mk, acc[20]);
    acc[21] = fma(D55, mk, acc[21]);
    acc[22] = fma(D56, mk, acc[22]);
    acc[23] = fma(D58, mk, acc[23]);
    acc[24] = fma(D59, mk, acc[24]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
    acc[16] = fma(D48, mk, acc[16]);
    acc[17] = fma(D50, mk, acc[17]);
    acc[18] = fma(D51, mk, acc[18]);
    acc[19] = fma(D53, mk, acc[19]);
    acc[20] = fma(D54, mk, acc[20]);
    acc[21] = fma(D56, mk, acc[21]);
    acc[22] = fma(D57, mk, acc[22]);
    acc[23] = fma(D59, mk, acc[23]);
    acc[24] = fma(D60, mk, acc[24]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
    acc[16] = fma(D49, mk, acc[16]);
    acc[17] = fma(D52, mk, acc[17]);
    acc[18] = fma(D53, mk, acc[18]);
    acc[19] = fma(D55, mk, acc[19]);
    acc[20] = fma(D56, mk, acc[20]);
    acc[21] = fma(D58, mk, acc[21]);
    acc[22] = fma(D59, mk, acc[22]);
    acc[23] = fma(D61, mk, acc[23]);
    acc[24] = fma(D62, mk, acc[24]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
    acc[16] = fma(D50, mk, acc[16]);
    acc[17] = fma(D53, mk, acc[17]);
    acc[18] = fma(D54, mk, acc[18]);
    acc[19] = fma(D56, mk, acc[19]);
    acc[20] = fma(D57, mk, acc[20]);
    acc[21] = fma(D59, mk, acc[21]);
    acc[22] = fma(D60, mk, acc[22]);
    acc[23] = fma(D62, mk, acc[23]);
    acc[24] = fma(D63, mk, acc[24]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
    acc[9] = fma(D46, mk, acc[9]);
    acc[10] = fma(D47, mk, acc[10]);
    acc[11] = fma(D48, mk, acc[11]);
    acc[12] = fma(D49, mk, acc[12]);
    acc[13] = fma(D50, mk, acc[13]);
    acc[14] = fma(D52, mk, acc[14]);
    acc[15] = fma(D53, mk, acc[15]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
    acc[9] = fma(D47, mk, acc[9]);
    acc[10] = fma(D49, mk, acc[10]);
    acc[11] = fma(D50, mk, acc[11]);
    acc[12] = fma(D52, mk, acc[12]);
    acc[13] = fma(D53, mk, acc[13]);
    acc[14] = fma(D55, mk, acc[14]);
    acc[15] = fma(D56, mk, acc[15]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
    acc[9] = fma(D48, mk, acc[9]);
    acc[10] = fma(D50, mk, acc[10]);
    acc[11] = fma(D51, mk, acc[11]);
    acc[12] = fma(D53, mk, acc[12]);
    acc[13] = fma(D54, mk, acc[13]);
    acc[14] = fma(D56, mk, acc[14]);
    acc[15] = fma(D57, mk, acc[15]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
    acc[9] = fma(D49, mk, acc[9]);
    acc[10] = fma(D52, mk, acc[10]);
    acc[11] = fma(D53, mk, acc[11]);
    acc[12] = fma(D55, mk, acc[12]);
    acc[13] = fma(D56, mk, acc[13]);
    acc[14] = fma(D58, mk, acc[14]);
    acc[15] = fma(D59, mk, acc[15]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
    acc[9] = fma(D50, mk, acc[9]);
    acc[10] = fma(D53, mk, acc[10]);
    acc[11] = fma(D54, mk, acc[11]);
    acc[12] = fma(D56, mk, acc[12]);
    acc[13] = fma(D57, mk, acc[13]);
    acc[14] = fma(D59, mk, acc[14]);
    acc[15] = fma(D60, mk, acc[15]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
    acc[9] = fma(D52, mk, acc[9]);
    acc[10] = fma(D55, mk, acc[10]);
    acc[11] = fma(D56, mk, acc[11]);
    acc[12] = fma(D58, mk, acc[12]);
    acc[13] = fma(D59, mk, acc[13]);
    acc[14] = fma(D61, mk, acc[14]);
    acc[15] = fma(D62, mk, acc[15]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
    acc[9] = fma(D53, mk, acc[9]);
    acc[10] = fma(D56, mk, acc[10]);
    acc[11] = fma(D57, mk, acc[11]);
    acc[12] = fma(D59, mk, acc[12]);
    acc[13] = fma(D60, mk, acc[13]);
    acc[14] = fma(D62, mk, acc[14]);
    acc[15] = fma(D63, mk, acc[15]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
    acc[4] = fma(D46, mk, acc[4]);
    acc[5] = fma(D47, mk, acc[5]);
    acc[6] = fma(D48, mk, acc[6]);
    acc[7] = fma(D49, mk, acc[7]);
    acc[8] = fma(D50, mk, acc[8]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
    acc[4] = fma(D47, mk, acc[4]);
    acc[5] = fma(D49, mk, acc[5]);
    acc[6] = fma(D50, mk, acc[6]);
    acc[7] = fma(D52, mk, acc[7]);
    acc[8] = fma(D53, mk, acc[8]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
    acc[4] = fma(D48, mk, acc[4]);
    acc[5] = fma(D50, mk, acc[5]);
    acc[6] = fma(D51, mk, acc[6]);
    acc[7] = fma(D53, mk, acc[7]);
    acc[8] = fma(D54, mk, acc[8]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
    acc[4] = fma(D49, mk, acc[4]);
    acc[5] = fma(D52, mk, acc[5]);
    acc[6] = fma(D53, mk, acc[6]);
    acc[7] = fma(D55, mk, acc[7]);
    acc[8] = fma(D56, mk, acc[8]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
    acc[4] = fma(D50, mk, acc[4]);
    acc[5] = fma(D53, mk, acc[5]);
    acc[6] = fma(D54, mk, acc[6]);
    acc[7] = fma(D56, mk, acc[7]);
    acc[8] = fma(D57, mk, acc[8]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
    acc[4] = fma(D52, mk, acc[4]);
    acc[5] = fma(D55, mk, acc[5]);
    acc[6] = fma(D56, mk, acc[6]);
    acc[7] = fma(D58, mk, acc[7]);
    acc[8] = fma(D59, mk, acc[8]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
    acc[4] = fma(D53, mk, acc[4]);
    acc[5] = fma(D56, mk, acc[5]);
    acc[6] = fma(D57, mk, acc[6]);
    acc[7] = fma(D59, mk, acc[7]);
    acc[8] = fma(D60, mk, acc[8]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
    acc[4] = fma(D55, mk, acc[4]);
    acc[5] = fma(D58, mk, acc[5]);
    acc[6] = fma(D59, mk, acc[6]);
    acc[7] = fma(D61, mk, acc[7]);
    acc[8] = fma(D62, mk, acc[8]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
    acc[4] = fma(D56, mk, acc[4]);
    acc[5] = fma(D59, mk, acc[5]);
    acc[6] = fma(D60, mk, acc[6]);
    acc[7] = fma(D62, mk, acc[7]);
    acc[8] = fma(D63, mk, acc[8]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D31, mk, acc[0]);
    acc[1] = fma(D46, mk, acc[1]);
    acc[2] = fma(D47, mk, acc[2]);
    acc[3] = fma(D48, mk, acc[3]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D32, mk, acc[0]);
    acc[1] = fma(D47, mk, acc[1]);
    acc[2] = fma(D49, mk, acc[2]);
    acc[3] = fma(D50, mk, acc[3]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D33, mk, acc[0]);
    acc[1] = fma(D48, mk, acc[1]);
    acc[2] = fma(D50, mk, acc[2]);
    acc[3] = fma(D51, mk, acc[3]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D34, mk, acc[0]);
    acc[1] = fma(D49, mk, acc[1]);
    acc[2] = fma(D52, mk, acc[2]);
    acc[3] = fma(D53, mk, acc[3]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D35, mk, acc[0]);
    acc[1] = fma(D50, mk, acc[1]);
    acc[2] = fma(D53, mk, acc[2]);
    acc[3] = fma(D54, mk, acc[3]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D37, mk, acc[0]);
    acc[1] = fma(D52, mk, acc[1]);
    acc[2] = fma(D55, mk, acc[2]);
    acc[3] = fma(D56, mk, acc[3]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D38, mk, acc[0]);
    acc[1] = fma(D53, mk, acc[1]);
    acc[2] = fma(D56, mk, acc[2]);
    acc[3] = fma(D57, mk, acc[3]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D40, mk, acc[0]);
    acc[1] = fma(D55, mk, acc[1]);
    acc[2] = fma(D58, mk, acc[2]);
    acc[3] = fma(D59, mk, acc[3]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D41, mk, acc[0]);
    acc[1] = fma(D56, mk, acc[1]);
    acc[2] = fma(D59, mk, acc[2]);
    acc[3] = fma(D60, mk, acc[3]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D43, mk, acc[0]);
    acc[1] = fma(D58, mk, acc[1]);
    acc[2] = fma(D61, mk, acc[2]);
    acc[3] = fma(D62, mk, acc[3]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D44, mk, acc[0]);
    acc[1] = fma(D59, mk, acc[1]);
    acc[2] = fma(D62, mk, acc[2]);
    acc[3] = fma(D63, mk, acc[3]);
  }
  { const T mk = Mb[36];
    acc[0] = fma(D46, mk, acc[0]);
  }
  { const T mk = Mb[37];
    acc[0] = fma(D47, mk, acc[0]);
  }
  { const T mk = Mb[38];
    acc[0] = fma(D48, mk, acc[0]);
  }
  { const T mk = Mb[39];
    acc[0] = fma(D49, mk, acc[0]);
  }
  { const T mk = Mb[40];
    acc[0] = fma(D50, mk, acc[0]);
  }
  { const T mk = Mb[41];
    acc[0] = fma(D52, mk, acc[0]);
  }
  { const T mk = Mb[42];
    acc[0] = fma(D53, mk, acc[0]);
  }
  { const T mk = Mb[43];
    acc[0] = fma(D55, mk, acc[0]);
  }
  { const T mk = Mb[44];
    acc[0] = fma(D56, mk, acc[0]);
  }
  { const T mk = Mb[45];
    acc[0] = fma(D58, mk, acc[0]);
  }
  { const T mk = Mb[46];
    acc[0] = fma(D59, mk, acc[0]);
  }
  { const T mk = Mb[47];
    acc[0] = fma(D61, mk, acc[0]);
  }
  { const T mk = Mb[48];
    acc[0] = fma(D62, mk, acc[0]);
  }
}
template <typename T>
__device__ __forceinline__ void dtensor_m0_p6(T x, T y, T z, T* __restrict__ Dout) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  const T w6_6 = crat<T>(-150, 6) * ir2;
  const T x6_1 = crat<T>(-11, 6) * xr;
  const T x6_6 = T(6) * x6_1;
  const T D46 = fma(x6_6, D31, w6_6 * D19);
  const T w6_5 = crat<T>(-100, 6) * ir2;
  const T x6_5 = T(5) * x6_1;
  const T y6_1 = crat<T>(-11, 6) * yr;
  const T D47 = fma(y6_1, D31, fma(x6_5, D32, w6_5 * D20));
  const T z6_1 = crat<T>(-11, 6) * zr;
  const T D48 = fma(z6_1, D31, fma(x6_5, D33, w6_5 * D21));
  const T w6_4 = crat<T>(-60, 6) * ir2;
  const T w6_2 = crat<T>(-10, 6) * ir2;
  const T x6_4 = T(4) * x6_1;
  const T y6_2 = T(2) * y6_1;
  const T D49 = fma(y6_2, D32, fma(x6_4, D34, fma(w6_2, D19, w6_4 * D22)));
  const T D50 = fma(z6_1, D32, fma(y6_1, D33, fma(x6_4, D35, w6_4 * D23)));
  const T D51 = -(D46 + D49);
  const T w6_3 = crat<T>(-30, 6) * ir2;
  const T x6_3 = T(3) * x6_1;
  const T y6_3 = T(3) * y6_1;
  const T D52 = fma(y6_3, D34, fma(x6_3, D37, fma(w6_3, D20, w6_3 * D25)));
  const T D53 = fma(z6_1, D34, fma(y6_2, D35, fma(x6_3, D38, fma(w6_2, D21, w6_3 * D26))));
  const T D54 = -(D47 + D52);
  const T x6_2 = T(2) * x6_1;
  const T y6_4 = T(4) * y6_1;
  const T D55 = fma(y6_4, D37, fma(x6_2, D40, fma(w6_4, D22, w6_2 * D28)));
  const T D56 = fma(z6_1, D37, fma(y6_3, D38, fma(x6_2, D41, fma(w6_3, D23, w6_2 * D29))));
  const T D57 = -(D49 + D55);
  const T y6_5 = T(5) * y6_1;
  const T D58 = fma(y6_5, D40, fma(x6_1, D43, w6_5 * D25));
  const T D59 = fma(z6_1, D40, fma(y6_4, D41, fma(x6_1, D44, w6_4 * D26)));
  const T D60 = -(D52 + D58);
  const T y6_6 = T(6) * y6_1;
  const T D61 = fma(y6_6, D43, w6_6 * D28);
  const T D62 = fma(z6_1, D43, fma(y6_5, D44, w6_5 * D29));
  const T D63 = -(D55 + D61);
  Dout[0] = D0;
  Dout[1] = D1;
  Dout[2] = D2;
  Dout[3] = D3;
  Dout[4] = D4;
  Dout[5] = D5;
  Dout[6] = D6;
  Dout[7] = D7;
  Dout[8] = D8;
  Dout[9] = D9;
  Dout[10] = D10;
  Dout[11] = D11;
  Dout[12] = D12;
  Dout[13] = D13;
  Dout[14] = D14;
  Dout[15] = D15;
  Dout[16] = D16;
  Dout[17] = D17;
  Dout[18] = D18;
  Dout[19] = D19;
  Dout[20] = D20;
  Dout[21] = D21;
  Dout[22] = D22;
  Dout[23] = D23;
  Dout[24] = D24;
  Dout[25] = D25;
  Dout[26] = D26;
  Dout[27] = D27;
  Dout[28] = D28;
  Dout[29] = D29;
  Dout[30] = D30;
  Dout[31] = D31;
  Dout[32] = D32;
  Dout[33] = D33;
  Dout[34] = D34;
  Dout[35] = D35;
  Dout[36] = D36;
  Dout[37] = D37;
  Dout[38] = D38;
  Dout[39] = D39;
  Dout[40] = D40;
  Dout[41] = D41;
  Dout[42] = D42;
  Dout[43] = D43;
  Dout[44] = D44;
  Dout[45] = D45;
  Dout[46] = D46;
  Dout[47] = D47;
  Dout[48] = D48;
  Dout[49] = D49;
  Dout[50] = D50;
  Dout[51] = D51;
  Dout[52] = D52;
  Dout[53] = D53;
  Dout[54] = D54;
  Dout[55] = D55;
  Dout[56] = D56;
  Dout[57] = D57;
  Dout[58] = D58;
  Dout[59] = D59;
  Dout[60] = D60;
  Dout[61] = D61;
  Dout[62] = D62;
  Dout[63] = D63;
}
template <typename T>
__device__ __forceinline__ void m2l_m0_p6_pre(const T* __restrict__ Dt, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T D0 = Dt[0];
  const T D1 = Dt[1];
  const T D2 = Dt[2];
  const T D3 = Dt[3];
  const T D4 = Dt[4];
  const T D5 = Dt[5];
  const T D6 = Dt[6];
  const T D7 = Dt[7];
  const T D8 = Dt[8];
  const T D9 = Dt[9];
  const T D10 = Dt[10];
  const T D11 = Dt[11];
  const T D12 = Dt[12];
  const T D13 = Dt[13];
  const T D14 = Dt[14];
  const T D15 = Dt[15];
  const T D16 = Dt[16];
  const T D17 = Dt[17];
  const T D18 = Dt[18];
  const T D19 = Dt[19];
  const T D20 = Dt[20];
  const T D21 = Dt[21];
  const T D22 = Dt[22];
  const T D23 = Dt[23];
  const T D24 = Dt[24];
  const T D25 = Dt[25];
  const T D26 = Dt[26];
  const T D27 = Dt[27];
  const T D28 = Dt[28];
  const T D29 = Dt[29];
  const T D30 = Dt[30];
  const T D31 = Dt[31];
  const T D32 = Dt[32];
  const T D33 = Dt[33];
  const T D34 = Dt[34];
  const T D35 = Dt[35];
  const T D36 = Dt[36];
  const T D37 = Dt[37];
  const T D38 = Dt[38];
  const T D39 = Dt[39];
  const T D40 = Dt[40];
  const T D41 = Dt[41];
  const T D42 = Dt[42];
  const T D43 = Dt[43];
  const T D44 = Dt[44];
  const T D45 = Dt[45];
  const T D46 = Dt[46];
  const T D47 = Dt[47];
  const T D48 = Dt[48];
  const T D49 = Dt[49];
  const T D50 = Dt[50];
  const T D51 = Dt[51];
  const T D52 = Dt[52];
  const T D53 = Dt[53];
  const T D54 = Dt[54];
  const T D55 = Dt[55];
  const T D56 = Dt[56];
  const T D57 = Dt[57];
  const T D58 = Dt[58];
  const T D59 = Dt[59];
  const T D60 = Dt[60];
  const T D61 = Dt[61];
  const T D62 = Dt[62];
  const T D63 = Dt[63];
  { const T mk = Mb[0];
    acc[0] = fma(D0, mk, acc[0]);
    acc[1] = fma(D1, mk, acc[1]);
    acc[2] = fma(D2, mk, acc[2]);
    acc[3] = fma(D3, mk, acc[3]);
    acc[4] = fma(D4, mk, acc[4]);
    acc[5] = fma(D5, mk, acc[5]);
    acc[6] = fma(D6, mk, acc[6]);
    acc[7] = fma(D7, mk, acc[7]);
    acc[8] = fma(D8, mk, acc[8]);
    acc[9] = fma(D10, mk, acc[9]);
    acc[10] = fma(D11, mk, acc[10]);
    acc[11] = fma(D12, mk, acc[11]);
    acc[12] = fma(D13, mk, acc[12]);
    acc[13] = fma(D14, mk, acc[13]);
    acc[14] = fma(D16, mk, acc[14]);
    acc[15] = fma(D17, mk, acc[15]);
    acc[16] = fma(D19, mk, acc[16]);
    acc[17] = fma(D20, mk, acc[17]);
    acc[18] = fma(D21, mk, acc[18]);
    acc[19] = fma(D22, mk, acc[19]);
    acc[20] = fma(D23, mk, acc[20]);
    acc[21] = fma(D25, mk, acc[21]);
    acc[22] = fma(D26, mk, acc[22]);
    acc[23] = fma(D28, mk, acc[23]);
    acc[24] = fma(D29, mk, acc[24]);
    acc[25] = fma(D31, mk, acc[25]);
    acc[26] = fma(D32, mk, acc[26]);
    acc[27] = fma(D33, mk, acc[27]);
    acc[28] = fma(D34, mk, acc[28]);
    acc[29] = fma(D35, mk, acc[29]);
    acc[30] = fma(D37, mk, acc[30]);
    acc[31] = fma(D38, mk, acc[31]);
    acc[32] = fma(D40, mk, acc[32]);
    acc[33] = fma(D41, mk, acc[33]);
    acc[34] = fma(D43, mk, acc[34]);
    acc[35] = fma(D44, mk, acc[35]);
    acc[36] = fma(D46, mk, acc[36]);
    acc[37] = fma(D47, mk, acc[37]);
    acc[38] = fma(D48, mk, acc[38]);
    acc[39] = fma(D49, mk, acc[39]);
    acc[40] = fma(D50, mk, acc[40]);
    acc[41] = fma(D52, mk, acc[41]);
    acc[42] = fma(D53, mk, acc[42]);
    acc[43] = fma(D55, mk, acc[43]);
    acc[44] = fma(D56, mk, acc[44]);
    acc[45] = fma(D58, mk, acc[45]);
    acc[46] = fma(D59, mk, acc[46]);
    acc[47] = fma(D61, mk, acc[47]);
    acc[48] = fma(D62, mk, acc[48]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D1, mk, acc[0]);
    acc[1] = fma(D4, mk, acc[1]);
    acc[2] = fma(D5, mk, acc[2]);
    acc[3] = fma(D6, mk, acc[3]);
    acc[4] = fma(D10, mk, acc[4]);
    acc[5] = fma(D11, mk, acc[5]);
    acc[6] = fma(D12, mk, acc[6]);
    acc[7] = fma(D13, mk, acc[7]);
    acc[8] = fma(D14, mk, acc[8]);
    acc[9] = fma(D19, mk, acc[9]);
    acc[10] = fma(D20, mk, acc[10]);
    acc[11] = fma(D21, mk, acc[11]);
    acc[12] = fma(D22, mk, acc[12]);
    acc[13] = fma(D23, mk, acc[13]);
    acc[14] = fma(D25, mk, acc[14]);
    acc[15] = fma(D26, mk, acc[15]);
    acc[16] = fma(D31, mk, acc[16]);
    acc[17] = fma(D32, mk, acc[17]);
    acc[18] = fma(D33, mk, acc[18]);
    acc[19] = fma(D34, mk, acc[19]);
    acc[20] = fma(D35, mk, acc[20]);
    acc[21] = fma(D37, mk, acc[21]);
    acc[22] = fma(D38, mk, acc[22]);
    acc[23] = fma(D40, mk, acc[23]);
    acc[24] = fma(D41, mk, acc[24]);
    acc[25] = fma(D46, mk, acc[25]);
    acc[26] = fma(D47, mk, acc[26]);
    acc[27] = fma(D48, mk, acc[27]);
    acc[28] = fma(D49, mk, acc[28]);
    acc[29] = fma(D50, mk, acc[29]);
    acc[30] = fma(D52, mk, acc[30]);
    acc[31] = fma(D53, mk, acc[31]);
    acc[32] = fma(D55, mk, acc[32]);
    acc[33] = fma(D56, mk, acc[33]);
    acc[34] = fma(D58, mk, acc[34]);
    acc[35] = fma(D59, mk, acc[35]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D2, mk, acc[0]);
    acc[1] = fma(D5, mk, acc[1]);
    acc[2] = fma(D7, mk, acc[2]);
    acc[3] = fma(D8, mk, acc[3]);
    acc[4] = fma(D11, mk, acc[4]);
    acc[5] = fma(D13, mk, acc[5]);
    acc[6] = fma(D14, mk, acc[6]);
    acc[7] = fma(D16, mk, acc[7]);
    acc[8] = fma(D17, mk, acc[8]);
    acc[9] = fma(D20, mk, acc[9]);
    acc[10] = fma(D22, mk, acc[10]);
    acc[11] = fma(D23, mk, acc[11]);
    acc[12] = fma(D25, mk, acc[12]);
    acc[13] = fma(D26, mk, acc[13]);
    acc[14] = fma(D28, mk, acc[14]);
    acc[15] = fma(D29, mk, acc[15]);
    acc[16] = fma(D32, mk, acc[16]);
    acc[17] = fma(D34, mk, acc[17]);
    acc[18] = fma(D35, mk, acc[18]);
    acc[19] = fma(D37, mk, acc[19]);
    acc[20] = fma(D38, mk, acc[20]);
    acc[21] = fma(D40, mk, acc[21]);
    acc[22] = fma(D41, mk, acc[22]);
    acc[23] = fma(D43, mk, acc[23]);
    acc[24] = fma(D44, mk, acc[24]);
    acc[25] = fma(D47, mk, acc[25]);
    acc[26] = fma(D49, mk, acc[26]);
    acc[27] = fma(D50, mk, acc[27]);
    acc[28] = fma(D52, mk, acc[28]);
    acc[29] = fma(D53, mk, acc[29]);
    acc[30] = fma(D55, mk, acc[30]);
    acc[31] = fma(D56, mk, acc[31]);
    acc[32] = fma(D58, mk, acc[32]);
    acc[33] = fma(D59, mk, acc[33]);
    acc[34] = fma(D61, mk, acc[34]);
    acc[35] = fma(D62, mk, acc[35]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D3, mk, acc[0]);
    acc[1] = fma(D6, mk, acc[1]);
    acc[2] = fma(D8, mk, acc[2]);
    acc[3] = fma(D9, mk, acc[3]);
    acc[4] = fma(D12, mk, acc[4]);
    acc[5] = fma(D14, mk, acc[5]);
    acc[6] = fma(D15, mk, acc[6]);
    acc[7] = fma(D17, mk, acc[7]);
    acc[8] = fma(D18, mk, acc[8]);
    acc[9] = fma(D21, mk, acc[9]);
    acc[10] = fma(D23, mk, acc[10]);
    acc[11] = fma(D24, mk, acc[11]);
    acc[12] = fma(D26, mk, acc[12]);
    acc[13] = fma(D27, mk, acc[13]);
    acc[14] = fma(D29, mk, acc[14]);
    acc[15] = fma(D30, mk, acc[15]);
    acc[16] = fma(D33, mk, acc[16]);
    acc[17] = fma(D35, mk, acc[17]);
    acc[18] = fma(D36, mk, acc[18]);
    acc[19] = fma(D38, mk, acc[19]);
    acc[20] = fma(D39, mk, acc[20]);
    acc[21] = fma(D41, mk, acc[21]);
    acc[22] = fma(D42, mk, acc[22]);
    acc[23] = fma(D44, mk, acc[23]);
    acc[24] = fma(D45, mk, acc[24]);
    acc[25] = fma(D48, mk, acc[25]);
    acc[26] = fma(D50, mk, acc[26]);
    acc[27] = fma(D51, mk, acc[27]);
    acc[28] = fma(D53, mk, acc[28]);
    acc[29] = fma(D54, mk, acc[29]);
    acc[30] = fma(D56, mk, acc[30]);
    acc[31] = fma(D57, mk, acc[31]);
    acc[32] = fma(D59, mk, acc[32]);
    acc[33] = fma(D60, mk, acc[33]);
    acc[34] = fma(D62, mk, acc[34]);
    acc[35] = fma(D63, mk, acc[35]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
    acc[16] = fma(D46, mk, acc[16]);
    acc[17] = fma(D47, mk, acc[17]);
    acc[18] = fma(D48, mk, acc[18]);
    acc[19] = fma(D49, mk, acc[19]);
    acc[20] = fma(D50, mk, acc[20]);
    acc[21] = fma(D52, mk, acc[21]);
    acc[22] = fma(D53, mk, acc[22]);
    acc[23] = fma(D55, mk, acc[23]);
    acc[24] = fma(D56, mk, acc[24]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
    acc[16] = fma(D47, mk, acc[16]);
    acc[17] = fma(D49, mk, acc[17]);
    acc[18] = fma(D50, mk, acc[18]);
    acc[19] = fma(D52, mk, acc[19]);
    acc[20] = fma(D53, mk, acc[20]);
    acc[21] = fma(D55, mk, acc[21]);
    acc[22] = fma(D56, mk, acc[22]);
    acc[23] = fma(D58, mk, acc[23]);
    acc[24] = fma(D59, mk, acc[24]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
    acc[16] = fma(D48, mk, acc[16]);
    acc[17] = fma(D50, mk, acc[17]);
    acc[18] = fma(D51, mk, acc[18]);
    acc[19] = fma(D53, mk, acc[19]);
    acc[20] = fma(D54, mk, acc[20]);
    acc[21] = fma(D56, mk, acc[21]);
    acc[22] = fma(D57, mk, acc[22]);
    acc[23] = fma(D59, mk, acc[23]);
    acc[24] = fma(D60, mk, acc[24]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
    acc[16] = fma(D49, mk, acc[16]);
    acc[17] = fma(D52, mk, acc[17]);
    acc[18] = fma(D53, mk, acc[18]);
    acc[19] = fma(D55, mk, acc[19]);
    acc[20] = fma(D56, mk, acc[20]);
    acc[21] = fma(D58, mk, acc[21]);
    acc[22] = fma(D59, mk, acc[22]);
    acc[23] = fma(D61, mk, acc[23]);
    acc[24] = fma(D62, mk, acc[24]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
    acc[16] = fma(D50, mk, acc[16]);
    acc[17] = fma(D53, mk, acc[17]);
    acc[18] = fma(D54, mk, acc[18]);
    acc[19] = fma(D56, mk, acc[19]);
    acc[20] = fma(D57, mk, acc[20]);
    acc[21] = fma(D59, mk, acc[21]);
    acc[22] = fma(D60, mk, acc[22]);
    acc[23] = fma(D62, mk, acc[23]);
    acc[24] = fma(D63, mk, acc[24]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
    acc[9] = fma(D46, mk, acc[9]);
    acc[10] = fma(D47, mk, acc[10]);
    acc[11] = fma(D48, mk, acc[11]);
    acc[12] = fma(D49, mk, acc[12]);
    acc[13] = fma(D50, mk, acc[13]);
    acc[14] = fma(D52, mk, acc[14]);
    acc[15] = fma(D53, mk, acc[15]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
    acc[9] = fma(D47, mk, acc[9]);
    acc[10] = fma(D49, mk, acc[10]);
    acc[11] = fma(D50, mk, acc[11]);
    acc[12] = fma(D52, mk, acc[12]);
    acc[13] = fma(D53, mk, acc[13]);
    acc[14] = fma(D55, mk, acc[14]);
    acc[15] = fma(D56, mk, acc[15]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
    acc[9] = fma(D48, mk, acc[9]);
    acc[10] = fma(D50, mk, acc[10]);
    acc[11] = fma(D51, mk, acc[11]);
    acc[12] = fma(D53, mk, acc[12]);
    acc[13] = fma(D54, mk, acc[13]);
    acc[14] = fma(D56, mk, acc[14]);
    acc[15] = fma(D57, mk, acc[15]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
    acc[9] = fma(D49, mk, acc[9]);
    acc[10] = fma(D52, mk, acc[10]);
    acc[11] = fma(D53, mk, acc[11]);
    acc[12] = fma(D55, mk, acc[12]);
    acc[13] = fma(D56, mk, acc[13]);
    acc[14] = fma(D58, mk, acc[14]);
    acc[15] = fma(D59, mk, acc[15]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
    acc[9] = fma(D50, mk, acc[9]);
    acc[10] = fma(D53, mk, acc[10]);
    acc[11] = fma(D54, mk, acc[11]);
    acc[12] = fma(D56, mk, acc[12]);
    acc[13] = fma(D57, mk, acc[13]);
    acc[14] = fma(D59, mk, acc[14]);
    acc[15] = fma(D60, mk, acc[15]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
    acc[9] = fma(D52, mk, acc[9]);
    acc[10] = fma(D55, mk, acc[10]);
    acc[11] = fma(D56, mk, acc[11]);
    acc[12] = fma(D58, mk, acc[12]);
    acc[13] = fma(D59, mk, acc[13]);
    acc[14] = fma(D61, mk, acc[14]);
    acc[15] = fma(D62, mk, acc[15]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
    acc[9] = fma(D53, mk, acc[9]);
    acc[10] = fma(D56, mk, acc[10]);
    acc[11] = fma(D57, mk, acc[11]);
    acc[12] = fma(D59, mk, acc[12]);
    acc[13] = fma(D60, mk, acc[13]);
    acc[14] = fma(D62, mk, acc[14]);
    acc[15] = fma(D63, mk, acc[15]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
    acc[4] = fma(D46, mk, acc[4]);
    acc[5] = fma(D47, mk, acc[5]);
    acc[6] = fma(D48, mk, acc[6]);
    acc[7] = fma(D49, mk, acc[7]);
    acc[8] = fma(D50, mk, acc[8]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
    acc[4] = fma(D47, mk, acc[4]);
    acc[5] = fma(D49, mk, acc[5]);
    acc[6] = fma(D50, mk, acc[6]);
    acc[7] = fma(D52, mk, acc[7]);
    acc[8] = fma(D53, mk, acc[8]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
    acc[4] = fma(D48, mk, acc[4]);
    acc[5] = fma(D50, mk, acc[5]);
    acc[6] = fma(D51, mk, acc[6]);
    acc[7] = fma(D53, mk, acc[7]);
    acc[8] = fma(D54, mk, acc[8]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
    acc[4] = fma(D49, mk, acc[4]);
    acc[5] = fma(D52, mk, acc[5]);
    acc[6] = fma(D53, mk, acc[6]);
    acc[7] = fma(D55, mk, acc[7]);
    acc[8] = fma(D56, mk, acc[8]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
    acc[4] = fma(D50, mk, acc[4]);
    acc[5] = fma(D53, mk, acc[5]);
    acc[6] = fma(D54, mk, acc[6]);
    acc[7] = fma(D56, mk, acc[7]);
    acc[8] = fma(D57, mk, acc[8]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
    acc[4] = fma(D52, mk, acc[4]);
    acc[5] = fma(D55, mk, acc[5]);
    acc[6] = fma(D56, mk, acc[6]);
    acc[7] = fma(D58, mk, acc[7]);
    acc[8] = fma(D59, mk, acc[8]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
    acc[4] = fma(D53, mk, acc[4]);
    acc[5] = fma(D56, mk, acc[5]);
    acc[6] = fma(D57, mk, acc[6]);
    acc[7] = fma(D59, mk, acc[7]);
    acc[8] = fma(D60, mk, acc[8]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
    acc[4] = fma(D55, mk, acc[4]);
    acc[5] = fma(D58, mk, acc[5]);
    acc[6] = fma(D59, mk, acc[6]);
    acc[7] = fma(D61, mk, acc[7]);
    acc[8] = fma(D62, mk, acc[8]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
    acc[4] = fma(D56, mk, acc[4]);
    acc[5] = fma(D59, mk, acc[5]);
    acc[6] = fma(D60, mk, acc[6]);
    acc[7] = fma(D62, mk, acc[7]);
    acc[8] = fma(D63, mk, acc[8]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D31, mk, acc[0]);
    acc[1] = fma(D46, mk, acc[1]);
    acc[2] = fma(D47, mk, acc[2]);
    acc[3] = fma(D48, mk, acc[3]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D32, mk, acc[0]);
    acc[1] = fma(D47, mk, acc[1]);
    acc[2] = fma(D49, mk, acc[2]);
    acc[3] = fma(D50, mk, acc[3]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D33, mk, acc[0]);
    acc[1] = fma(D48, mk, acc[1]);
    acc[2] = fma(D50, mk, acc[2]);
    acc[3] = fma(D51, mk, acc[3]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D34, mk, acc[0]);
    acc[1] = fma(D49, mk, acc[1]);
    acc[2] = fma(D52, mk, acc[2]);
    acc[3] = fma(D53, mk, acc[3]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D35, mk, acc[0]);
    acc[1] = fma(D50, mk, acc[1]);
    acc[2] = fma(D53, mk, acc[2]);
    acc[3] = fma(D54, mk, acc[3]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D37, mk, acc[0]);
    acc[1] = fma(D52, mk, acc[1]);
    acc[2] = fma(D55, mk, acc[2]);
    acc[3] = fma(D56, mk, acc[3]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D38, mk, acc[0]);
    acc[1] = fma(D53, mk, acc[1]);
    acc[2] = fma(D56, mk, acc[2]);
    acc[3] = fma(D57, mk, acc[3]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D40, mk, acc[0]);
    acc[1] = fma(D55, mk, acc[1]);
    acc[2] = fma(D58, mk, acc[2]);
    acc[3] = fma(D59, mk, acc[3]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D41, mk, acc[0]);
    acc[1] = fma(D56, mk, acc[1]);
    acc[2] = fma(D59, mk, acc[2]);
    acc[3] = fma(D60, mk, acc[3]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D43, mk, acc[0]);
    acc[1] = fma(D58, mk, acc[1]);
    acc[2] = fma(D61, mk, acc[2]);
    acc[3] = fma(D62, mk, acc[3]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D44, mk, acc[0]);
    acc[1] = fma(D59, mk, acc[1]);
    acc[2] = fma(D62, mk, acc[2]);
    acc[3] = fma(D63, mk, acc[3]);
  }
  { const T mk = Mb[36];
    acc[0] = fma(D46, mk, acc[0]);
  }
  { const T mk = Mb[37];
    acc[0] = fma(D47, mk, acc[0]);
  }
  { const T mk = Mb[38];
    acc[0] = fma(D48, mk, acc[0]);
  }
  { const T mk = Mb[39];
    acc[0] = fma(D49, mk, acc[0]);
  }
  { const T mk = Mb[40];
    acc[0] = fma(D50, mk, acc[0]);
  }
  { const T mk = Mb[41];
    acc[0] = fma(D52, mk, acc[0]);
  }
  { const T mk = Mb[42];
    acc[0] = fma(D53, mk, acc[0]);
  }
  { const T mk = Mb[43];
    acc[0] = fma(D55, mk, acc[0]);
  }
  { const T mk = Mb[44];
    acc[0] = fma(D56, mk, acc[0]);
  }
  { const T mk = Mb[45];
    acc[0] = fma(D58, mk, acc[0]);
  }
  { const T mk = Mb[46];
    acc[0] = fma(D59, mk, acc[0]);
  }
  { const T mk = Mb[47];
    acc[0] = fma(D61, mk, acc[0]);
  }
  { const T mk = Mb[48];
    acc[0] = fma(D62, mk, acc[0]);
  }
}
static __constant__ unsigned char m2l_w_m0_p6[532] = {
  0, 1, 2, 3, 4, 5, 6, 7, 8, 10, 11, 12, 13, 14, 16, 17, 19, 20, 21, 22, 23, 25, 26, 28, 29, 31, 32, 33, 34, 35, 37, 38, 40, 41, 43, 44, 46, 47, 48, 49, 50, 52, 53, 55, 56, 58, 59, 61, 62, 1, 4, 5, 6, 10, 11, 12, 13, 14, 19, 20, 21, 22, 23, 25, 26, 31, 32, 33, 34, 35, 37, 38, 40, 41, 46, 47, 48, 49, 50, 52, 53, 55, 56, 58, 59, 2, 5, 7, 8, 11, 13, 14, 16, 17, 20, 22, 23, 25, 26, 28, 29, 32, 34, 35, 37, 38, 40, 41, 43, 44, 47, 49, 50, 52, 53, 55, 56, 58, 59, 61, 62, 3, 6, 8, 9, 12, 14, 15, 17, 18, 21, 23, 24, 26, 27, 29, 30, 33, 35, 36, 38, 39, 41, 42, 44, 45, 48, 50, 51, 53, 54, 56, 57, 59, 60, 62, 63, 4, 10, 11, 12, 19, 20, 21, 22, 23, 31, 32, 33, 34, 35, 37, 38, 46, 47, 48, 49, 50, 52, 53, 55, 56, 5, 11, 13, 14, 20, 22, 23, 25, 26, 32, 34, 35, 37, 38, 40, 41, 47, 49, 50, 52, 53, 55, 56, 58, 59, 6, 12, 14, 15, 21, 23, 24, 26, 27, 33, 35, 36, 38, 39, 41, 42, 48, 50, 51, 53, 54, 56, 57, 59, 60, 7, 13, 16, 17, 22, 25, 26, 28, 29, 34, 37, 38, 40, 41, 43, 44, 49, 52, 53, 55, 56, 58, 59, 61, 62, 8, 14, 17, 18, 23, 26, 27, 29, 30, 35, 38, 39, 41, 42, 44, 45, 50, 53, 54, 56, 57, 59, 60, 62, 63, 10, 19, 20, 21, 31, 32, 33, 34, 35, 46, 47, 48, 49, 50, 52, 53, 11, 20, 22, 23, 32, 34, 35, 37, 38, 47, 49, 50, 52, 53, 55, 56, 12, 21, 23, 24, 33, 35, 36, 38, 39, 48, 50, 51, 53, 54, 56, 57, 13, 22, 25, 26, 34, 37, 38, 40, 41, 49, 52, 53, 55, 56, 58, 59, 14, 23, 26, 27, 35, 38, 39, 41, 42, 50, 53, 54, 56, 57, 59, 60, 16, 25, 28, 29, 37, 40, 41, 43, 44, 52, 55, 56, 58, 59, 61, 62, 17, 26, 29, 30, 38, 41, 42, 44, 45, 53, 56, 57, 59, 60, 62, 63, 19, 31, 32, 33, 46, 47, 48, 49, 50, 20, 32, 34, 35, 47, 49, 50, 52, 53, 21, 33, 35, 36, 48, 50, 51, 53, 54, 22, 34, 37, 38, 49, 52, 53, 55, 56, 23, 35, 38, 39, 50, 53, 54, 56, 57, 25, 37, 40, 41, 52, 55, 56, 58, 59, 26, 38, 41, 42, 53, 56, 57, 59, 60, 28, 40, 43, 44, 55, 58, 59, 61, 62, 29, 41, 44, 45, 56, 59, 60, 62, 63, 31, 46, 47, 48, 32, 47, 49, 50, 33, 48, 50, 51, 34, 49, 52, 53, 35, 50, 53, 54, 37, 52, 55, 56, 38, 53, 56, 57, 40, 55, 58, 59, 41, 56, 59, 60, 43, 58, 61, 62, 44, 59, 62, 63, 46, 47, 48, 49, 50, 52, 53, 55, 56, 58, 59, 61, 62};
static __device__ const signed char m2l_fold_m0_p6[49][6][2] = {
  {{0, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{4, 1}, {9, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{7, 1}, {9, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{10, 1}, {15, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{11, 1}, {18, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{12, 1}, {19, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{13, 1}, {15, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{16, 1}, {18, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{17, 1}, {19, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{20, 1}, {25, -1}, {34, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{21, 1}, {28, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{22, 1}, {29, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{23, 1}, {25, -1}, {32, -1}, {34, 2}, {0, 0}, {0, 0}},
  {{24, 1}, {33, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{26, 1}, {28, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{27, 1}, {29, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{30, 1}, {32, -1}, {34, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{31, 1}, {33, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{35, 1}, {40, -1}, {49, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{36, 1}, {43, -1}, {54, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{37, 1}, {44, -1}, {55, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{38, 1}, {40, -1}, {47, -1}, {49, 2}, {0, 0}, {0, 0}},
  {{39, 1}, {48, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{41, 1}, {43, -1}, {52, -1}, {54, 2}, {0, 0}, {0, 0}},
  {{42, 1}, {44, -1}, {53, -1}, {55, 2}, {0, 0}, {0, 0}},
  {{45, 1}, {47, -1}, {49, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{46, 1}, {48, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{50, 1}, {52, -1}, {54, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{51, 1}, {53, -1}, {55, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{56, 1}, {61, -1}, {70, 1}, {83, -1}, {0, 0}, {0, 0}},
  {{57, 1}, {64, -1}, {75, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{58, 1}, {65, -1}, {76, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{59, 1}, {61, -1}, {68, -1}, {70, 2}, {81, 1}, {83, -3}},
  {{60, 1}, {69, -1}, {82, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{62, 1}, {64, -1}, {73, -1}, {75, 2}, {0, 0}, {0, 0}},
  {{63, 1}, {65, -1}, {74, -1}, {76, 2}, {0, 0}, {0, 0}},
  {{66, 1}, {68, -1}, {70, 1}, {79, -1}, {81, 2}, {83, -3}},
  {{67, 1}, {69, -1}, {80, -1}, {82, 2}, {0, 0}, {0, 0}},
  {{71, 1}, {73, -1}, {75, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{72, 1}, {74, -1}, {76, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{77, 1}, {79, -1}, {81, 1}, {83, -1}, {0, 0}, {0, 0}},
  {{78, 1}, {80, -1}, {82, 1}, {0, 0}, {0, 0}, {0, 0}},
};
static __device__ const signed char m2l_unfold_m0_p6[84][4][2] = {
  {{0, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{7, -1}, {4, -1}, {0, 0}, {0, 0}},
  {{9, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{11, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{12, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{12, -1}, {9, -1}, {0, 0}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{15, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{14, -1}, {10, -1}, {0, 0}, {0, 0}},
  {{15, -1}, {11, -1}, {0, 0}, {0, 0}},
  {{16, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{17, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{18, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{19, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{20, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{19, -1}, {16, -1}, {0, 0}, {0, 0}},
  {{21, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{22, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{21, -1}, {17, -1}, {0, 0}, {0, 0}},
  {{22, -1}, {18, -1}, {0, 0}, {0, 0}},
  {{23, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{24, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{23, -1}, {19, -1}, {0, 0}, {0, 0}},
  {{24, -1}, {20, -1}, {0, 0}, {0, 0}},
  {{23, 1}, {19, 2}, {16, 1}, {0, 0}},
  {{25, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{26, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{27, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{28, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{29, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{28, -1}, {25, -1}, {0, 0}, {0, 0}},
  {{30, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{31, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{30, -1}, {26, -1}, {0, 0}, {0, 0}},
  {{31, -1}, {27, -1}, {0, 0}, {0, 0}},
  {{32, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{33, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{32, -1}, {28, -1}, {0, 0}, {0, 0}},
  {{33, -1}, {29, -1}, {0, 0}, {0, 0}},
  {{32, 1}, {28, 2}, {25, 1}, {0, 0}},
  {{34, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{35, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{34, -1}, {30, -1}, {0, 0}, {0, 0}},
  {{35, -1}, {31, -1}, {0, 0}, {0, 0}},
  {{34, 1}, {30, 2}, {26, 1}, {0, 0}},
  {{35, 1}, {31, 2}, {27, 1}, {0, 0}},
  {{36, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{37, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{38, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{39, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{40, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{39, -1}, {36, -1}, {0, 0}, {0, 0}},
  {{41, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{42, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{41, -1}, {37, -1}, {0, 0}, {0, 0}},
  {{42, -1}, {38, -1}, {0, 0}, {0, 0}},
  {{43, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{44, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{43, -1}, {39, -1}, {0, 0}, {0, 0}},
  {{44, -1}, {40, -1}, {0, 0}, {0, 0}},
  {{43, 1}, {39, 2}, {36, 1}, {0, 0}},
  {{45, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{46, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{45, -1}, {41, -1}, {0, 0}, {0, 0}},
  {{46, -1}, {42, -1}, {0, 0}, {0, 0}},
  {{45, 1}, {41, 2}, {37, 1}, {0, 0}},
  {{46, 1}, {42, 2}, {38, 1}, {0, 0}},
  {{47, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{48, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{47, -1}, {43, -1}, {0, 0}, {0, 0}},
  {{48, -1}, {44, -1}, {0, 0}, {0, 0}},
  {{47, 1}, {43, 2}, {39, 1}, {0, 0}},
  {{48, 1}, {44, 2}, {40, 1}, {0, 0}},
  {{47, -1}, {43, -3}, {39, -3}, {36, -1}},
};

// M2L between reduced coefficients, source order 2, expansion order 5: 32 multipole, 16 local, 46 tensor entries, 190 terms
template <typename T>
__device__ __forceinline__ void m2l_m2_p5(T x, T y, T z, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  { const T mk = Mb[0];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D31, mk, acc[0]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D32, mk, acc[0]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D33, mk, acc[0]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D34, mk, acc[0]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D35, mk, acc[0]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D37, mk, acc[0]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D38, mk, acc[0]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D40, mk, acc[0]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D41, mk, acc[0]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D43, mk, acc[0]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D44, mk, acc[0]);
  }
}
template <typename T>
__device__ __forceinline__ void dtensor_m2_p5(T x, T y, T z, T* __restrict__ Dout) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  Dout[0] = D0;
  Dout[1] = D1;
  Dout[2] = D2;
  Dout[3] = D3;
  Dout[4] = D4;
  Dout[5] = D5;
  Dout[6] = D6;
  Dout[7] = D7;
  Dout[8] = D8;
  Dout[9] = D9;
  Dout[10] = D10;
  Dout[11] = D11;
  Dout[12] = D12;
  Dout[13] = D13;
  Dout[14] = D14;
  Dout[15] = D15;
  Dout[16] = D16;
  Dout[17] = D17;
  Dout[18] = D18;
  Dout[19] = D19;
  Dout[20] = D20;
  Dout[21] = D21;
  Dout[22] = D22;
  Dout[23] = D23;
  Dout[24] = D24;
  Dout[25] = D25;
  Dout[26] = D26;
  Dout[27] = D27;
  Dout[28] = D28;
  Dout[29] = D29;
  Dout[30] = D30;
  Dout[31] = D31;
  Dout[32] = D32;
  Dout[33] = D33;
  Dout[34] = D34;
  Dout[35] = D35;
  Dout[36] = D36;
  Dout[37] = D37;
  Dout[38] = D38;
  Dout[39] = D39;
  Dout[40] = D40;
  Dout[41] = D41;
  Dout[42] = D42;
  Dout[43] = D43;
  Dout[44] = D44;
  Dout[45] = D45;
}
template <typename T>
__device__ __forceinline__ void m2l_m2_p5_pre(const T* __restrict__ Dt, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T D0 = Dt[0];
  const T D1 = Dt[1];
  const T D2 = Dt[2];
  const T D3 = Dt[3];
  const T D4 = Dt[4];
  const T D5 = Dt[5];
  const T D6 = Dt[6];
  const T D7 = Dt[7];
  const T D8 = Dt[8];
  const T D9 = Dt[9];
  const T D10 = Dt[10];
  const T D11 = Dt[11];
  const T D12 = Dt[12];
  const T D13 = Dt[13];
  const T D14 = Dt[14];
  const T D15 = Dt[15];
  const T D16 = Dt[16];
  const T D17 = Dt[17];
  const T D18 = Dt[18];
  const T D19 = Dt[19];
  const T D20 = Dt[20];
  const T D21 = Dt[21];
  const T D22 = Dt[22];
  const T D23 = Dt[23];
  const T D24 = Dt[24];
  const T D25 = Dt[25];
  const T D26 = Dt[26];
  const T D27 = Dt[27];
  const T D28 = Dt[28];
  const T D29 = Dt[29];
  const T D30 = Dt[30];
  const T D31 = Dt[31];
  const T D32 = Dt[32];
  const T D33 = Dt[33];
  const T D34 = Dt[34];
  const T D35 = Dt[35];
  const T D36 = Dt[36];
  const T D37 = Dt[37];
  const T D38 = Dt[38];
  const T D39 = Dt[39];
  const T D40 = Dt[40];
  const T D41 = Dt[41];
  const T D42 = Dt[42];
  const T D43 = Dt[43];
  const T D44 = Dt[44];
  const T D45 = Dt[45];
  { const T mk = Mb[0];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D31, mk, acc[0]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D32, mk, acc[0]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D33, mk, acc[0]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D34, mk, acc[0]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D35, mk, acc[0]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D37, mk, acc[0]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D38, mk, acc[0]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D40, mk, acc[0]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D41, mk, acc[0]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D43, mk, acc[0]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D44, mk, acc[0]);
  }
}
static __constant__ unsigned char m2l_w_m2_p5[190] = {
  4, 10, 11, 12, 19, 20, 21, 22, 23, 31, 32, 33, 34, 35, 37, 38, 5, 11, 13, 14, 20, 22, 23, 25, 26, 32, 34, 35, 37, 38, 40, 41, 6, 12, 14, 15, 21, 23, 24, 26, 27, 33, 35, 36, 38, 39, 41, 42, 7, 13, 16, 17, 22, 25, 26, 28, 29, 34, 37, 38, 40, 41, 43, 44, 8, 14, 17, 18, 23, 26, 27, 29, 30, 35, 38, 39, 41, 42, 44, 45, 10, 19, 20, 21, 31, 32, 33, 34, 35, 11, 20, 22, 23, 32, 34, 35, 37, 38, 12, 21, 23, 24, 33, 35, 36, 38, 39, 13, 22, 25, 26, 34, 37, 38, 40, 41, 14, 23, 26, 27, 35, 38, 39, 41, 42, 16, 25, 28, 29, 37, 40, 41, 43, 44, 17, 26, 29, 30, 38, 41, 42, 44, 45, 19, 31, 32, 33, 20, 32, 34, 35, 21, 33, 35, 36, 22, 34, 37, 38, 23, 35, 38, 39, 25, 37, 40, 41, 26, 38, 41, 42, 28, 40, 43, 44, 29, 41, 44, 45, 31, 32, 33, 34, 35, 37, 38, 40, 41, 43, 44};
static __device__ const signed char m2l_fold_m2_p5[32][4][2] = {
  {{0, 1}, {5, -1}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {5, -1}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {11, -1}, {0, 0}, {0, 0}},
  {{7, 1}, {14, -1}, {0, 0}, {0, 0}},
  {{8, 1}, {15, -1}, {0, 0}, {0, 0}},
  {{9, 1}, {11, -1}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{12, 1}, {14, -1}, {0, 0}, {0, 0}},
  {{13, 1}, {15, -1}, {0, 0}, {0, 0}},
  {{16, 1}, {21, -1}, {30, 1}, {0, 0}},
  {{17, 1}, {24, -1}, {0, 0}, {0, 0}},
  {{18, 1}, {25, -1}, {0, 0}, {0, 0}},
  {{19, 1}, {21, -1}, {28, -1}, {30, 2}},
  {{20, 1}, {29, -1}, {0, 0}, {0, 0}},
  {{22, 1}, {24, -1}, {0, 0}, {0, 0}},
  {{23, 1}, {25, -1}, {0, 0}, {0, 0}},
  {{26, 1}, {28, -1}, {30, 1}, {0, 0}},
  {{27, 1}, {29, -1}, {0, 0}, {0, 0}},
  {{31, 1}, {36, -1}, {45, 1}, {0, 0}},
  {{32, 1}, {39, -1}, {50, 1}, {0, 0}},
  {{33, 1}, {40, -1}, {51, 1}, {0, 0}},
  {{34, 1}, {36, -1}, {43, -1}, {45, 2}},
  {{35, 1}, {44, -1}, {0, 0}, {0, 0}},
  {{37, 1}, {39, -1}, {48, -1}, {50, 2}},
  {{38, 1}, {40, -1}, {49, -1}, {51, 2}},
  {{41, 1}, {43, -1}, {45, 1}, {0, 0}},
  {{42, 1}, {44, -1}, {0, 0}, {0, 0}},
  {{46, 1}, {48, -1}, {50, 1}, {0, 0}},
  {{47, 1}, {49, -1}, {51, 1}, {0, 0}},
};
static __device__ const signed char m2l_unfold_m2_p5[20][2][2] = {
  {{0, 1}, {0, 0}},
  {{1, 1}, {0, 0}},
  {{2, 1}, {0, 0}},
  {{3, 1}, {0, 0}},
  {{4, 1}, {0, 0}},
  {{5, 1}, {0, 0}},
  {{6, 1}, {0, 0}},
  {{7, 1}, {0, 0}},
  {{8, 1}, {0, 0}},
  {{7, -1}, {4, -1}},
  {{9, 1}, {0, 0}},
  {{10, 1}, {0, 0}},
  {{11, 1}, {0, 0}},
  {{12, 1}, {0, 0}},
  {{13, 1}, {0, 0}},
  {{12, -1}, {9, -1}},
  {{14, 1}, {0, 0}},
  {{15, 1}, {0, 0}},
  {{14, -1}, {10, -1}},
  {{15, -1}, {11, -1}},
};

// M2L between reduced coefficients, source order 2, expansion order 6: 45 multipole, 25 local, 64 tensor entries, 375 terms
template <typename T>
__device__ __forceinline__ void m2l_m2_p6(T x, T y, T z, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  const T w6_6 = crat<T>(-150, 6) * ir2;
  const T x6_1 = crat<T>(-11, 6) * xr;
  const T x6_6 = T(6) * x6_1;
  const T D46 = fma(x6_6, D31, w6_6 * D19);
  const T w6_5 = crat<T>(-100, 6) * ir2;
  const T x6_5 = T(5) * x6_1;
  const T y6_1 = crat<T>(-11, 6) * yr;
  const T D47 = fma(y6_1, D31, fma(x6_5, D32, w6_5 * D20));
  const T z6_1 = crat<T>(-11, 6) * zr;
  const T D48 = fma(z6_1, D31, fma(x6_5, D33, w6_5 * D21));
  const T w6_4 = crat<T>(-60, 6) * ir2;
  const T w6_2 = crat<T>(-10, 6) * ir2;
  const T x6_4 = T(4) * x6_1;
  const T y6_2 = T(2) * y6_1;
  const T D49 = fma(y6_2, D32, fma(x6_4, D34, fma(w6_2, D19, w6_4 * D22)));
  const T D50 = fma(z6_1, D32, fma(y6_1, D33, fma(x6_4, D35, w6_4 * D23)));
  const T D51 = -(D46 + D49);
  const T w6_3 = crat<T>(-30, 6) * ir2;
  const T x6_3 = T(3) * x6_1;
  const T y6_3 = T(3) * y6_1;
  const T D52 = fma(y6_3, D34, fma(x6_3, D37, fma(w6_3, D20, w6_3 * D25)));
  const T D53 = fma(z6_1, D34, fma(y6_2, D35, fma(x6_3, D38, fma(w6_2, D21, w6_3 * D26))));
  const T D54 = -(D47 + D52);
  const T x6_2 = T(2) * x6_1;
  const T y6_4 = T(4) * y6_1;
  const T D55 = fma(y6_4, D37, fma(x6_2, D40, fma(w6_4, D22, w6_2 * D28)));
  const T D56 = fma(z6_1, D37, fma(y6_3, D38, fma(x6_2, D41, fma(w6_3, D23, w6_2 * D29))));
  const T D57 = -(D49 + D55);
  const T y6_5 = T(5) * y6_1;
  const T D58 = fma(y6_5, D40, fma(x6_1, D43, w6_5 * D25));
  const T D59 = fma(z6_1, D40, fma(y6_4, D41, fma(x6_1, D44, w6_4 * D26)));
  const T D60 = -(D52 + D58);
  const T y6_6 = T(6) * y6_1;
  const T D61 = fma(y6_6, D43, w6_6 * D28);
  const T D62 = fma(z6_1, D43, fma(y6_5, D44, w6_5 * D29));
  const T D63 = -(D55 + D61);
  { const T mk = Mb[0];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
    acc[16] = fma(D46, mk, acc[16]);
    acc[17] = fma(D47, mk, acc[17]);
    acc[18] = fma(D48, mk, acc[18]);
    acc[19] = fma(D49, mk, acc[19]);
    acc[20] = fma(D50, mk, acc[20]);
    acc[21] = fma(D52, mk, acc[21]);
    acc[22] = fma(D53, mk, acc[22]);
    acc[23] = fma(D55, mk, acc[23]);
    acc[24] = fma(D56, mk, acc[24]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
    acc[16] = fma(D47, mk, acc[16]);
    acc[17] = fma(D49, mk, acc[17]);
    acc[18] = fma(D50, mk, acc[18]);
    acc[19] = fma(D52, mk, acc[19]);
    acc[20] = fma(D53, mk, acc[20]);
    acc[21] = fma(D55, mk, acc[21]);
    acc[22] = fma(D56, mk, acc[22]);
    acc[23] = fma(D58, mk, acc[23]);
    acc[24] = fma(D59, mk, acc[24]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
    acc[16] = fma(D48, mk, acc[16]);
    acc[17] = fma(D50, mk, acc[17]);
    acc[18] = fma(D51, mk, acc[18]);
    acc[19] = fma(D53, mk, acc[19]);
    acc[20] = fma(D54, mk, acc[20]);
    acc[21] = fma(D56, mk, acc[21]);
    acc[22] = fma(D57, mk, acc[22]);
    acc[23] = fma(D59, mk, acc[23]);
    acc[24] = fma(D60, mk, acc[24]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
    acc[16] = fma(D49, mk, acc[16]);
    acc[17] = fma(D52, mk, acc[17]);
    acc[18] = fma(D53, mk, acc[18]);
    acc[19] = fma(D55, mk, acc[19]);
    acc[20] = fma(D56, mk, acc[20]);
    acc[21] = fma(D58, mk, acc[21]);
    acc[22] = fma(D59, mk, acc[22]);
    acc[23] = fma(D61, mk, acc[23]);
    acc[24] = fma(D62, mk, acc[24]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
    acc[16] = fma(D50, mk, acc[16]);
    acc[17] = fma(D53, mk, acc[17]);
    acc[18] = fma(D54, mk, acc[18]);
    acc[19] = fma(D56, mk, acc[19]);
    acc[20] = fma(D57, mk, acc[20]);
    acc[21] = fma(D59, mk, acc[21]);
    acc[22] = fma(D60, mk, acc[22]);
    acc[23] = fma(D62, mk, acc[23]);
    acc[24] = fma(D63, mk, acc[24]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
    acc[9] = fma(D46, mk, acc[9]);
    acc[10] = fma(D47, mk, acc[10]);
    acc[11] = fma(D48, mk, acc[11]);
    acc[12] = fma(D49, mk, acc[12]);
    acc[13] = fma(D50, mk, acc[13]);
    acc[14] = fma(D52, mk, acc[14]);
    acc[15] = fma(D53, mk, acc[15]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
    acc[9] = fma(D47, mk, acc[9]);
    acc[10] = fma(D49, mk, acc[10]);
    acc[11] = fma(D50, mk, acc[11]);
    acc[12] = fma(D52, mk, acc[12]);
    acc[13] = fma(D53, mk, acc[13]);
    acc[14] = fma(D55, mk, acc[14]);
    acc[15] = fma(D56, mk, acc[15]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
    acc[9] = fma(D48, mk, acc[9]);
    acc[10] = fma(D50, mk, acc[10]);
    acc[11] = fma(D51, mk, acc[11]);
    acc[12] = fma(D53, mk, acc[12]);
    acc[13] = fma(D54, mk, acc[13]);
    acc[14] = fma(D56, mk, acc[14]);
    acc[15] = fma(D57, mk, acc[15]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
    acc[9] = fma(D49, mk, acc[9]);
    acc[10] = fma(D52, mk, acc[10]);
    acc[11] = fma(D53, mk, acc[11]);
    acc[12] = fma(D55, mk, acc[12]);
    acc[13] = fma(D56, mk, acc[13]);
    acc[14] = fma(D58, mk, acc[14]);
    acc[15] = fma(D59, mk, acc[15]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
    acc[9] = fma(D50, mk, acc[9]);
    acc[10] = fma(D53, mk, acc[10]);
    acc[11] = fma(D54, mk, acc[11]);
    acc[12] = fma(D56, mk, acc[12]);
    acc[13] = fma(D57, mk, acc[13]);
    acc[14] = fma(D59, mk, acc[14]);
    acc[15] = fma(D60, mk, acc[15]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
    acc[9] = fma(D52, mk, acc[9]);
    acc[10] = fma(D55, mk, acc[10]);
    acc[11] = fma(D56, mk, acc[11]);
    acc[12] = fma(D58, mk, acc[12]);
    acc[13] = fma(D59, mk, acc[13]);
    acc[14] = fma(D61, mk, acc[14]);
    acc[15] = fma(D62, mk, acc[15]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
    acc[9] = fma(D53, mk, acc[9]);
    acc[10] = fma(D56, mk, acc[10]);
    acc[11] = fma(D57, mk, acc[11]);
    acc[12] = fma(D59, mk, acc[12]);
    acc[13] = fma(D60, mk, acc[13]);
    acc[14] = fma(D62, mk, acc[14]);
    acc[15] = fma(D63, mk, acc[15]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
    acc[4] = fma(D46, mk, acc[4]);
    acc[5] = fma(D47, mk, acc[5]);
    acc[6] = fma(D48, mk, acc[6]);
    acc[7] = fma(D49, mk, acc[7]);
    acc[8] = fma(D50, mk, acc[8]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
    acc[4] = fma(D47, mk, acc[4]);
    acc[5] = fma(D49, mk, acc[5]);
    acc[6] = fma(D50, mk, acc[6]);
    acc[7] = fma(D52, mk, acc[7]);
    acc[8] = fma(D53, mk, acc[8]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
    acc[4] = fma(D48, mk, acc[4]);
    acc[5] = fma(D50, mk, acc[5]);
    acc[6] = fma(D51, mk, acc[6]);
    acc[7] = fma(D53, mk, acc[7]);
    acc[8] = fma(D54, mk, acc[8]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
    acc[4] = fma(D49, mk, acc[4]);
    acc[5] = fma(D52, mk, acc[5]);
    acc[6] = fma(D53, mk, acc[6]);
    acc[7] = fma(D55, mk, acc[7]);
    acc[8] = fma(D56, mk, acc[8]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
    acc[4] = fma(D50, mk, acc[4]);
    acc[5] = fma(D53, mk, acc[5]);
    acc[6] = fma(D54, mk, acc[6]);
    acc[7] = fma(D56, mk, acc[7]);
    acc[8] = fma(D57, mk, acc[8]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
    acc[4] = fma(D52, mk, acc[4]);
    acc[5] = fma(D55, mk, acc[5]);
    acc[6] = fma(D56, mk, acc[6]);
    acc[7] = fma(D58, mk, acc[7]);
    acc[8] = fma(D59, mk, acc[8]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
    acc[4] = fma(D53, mk, acc[4]);
    acc[5] = fma(D56, mk, acc[5]);
    acc[6] = fma(D57, mk, acc[6]);
    acc[7] = fma(D59, mk, acc[7]);
    acc[8] = fma(D60, mk, acc[8]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
    acc[4] = fma(D55, mk, acc[4]);
    acc[5] = fma(D58, mk, acc[5]);
    acc[6] = fma(D59, mk, acc[6]);
    acc[7] = fma(D61, mk, acc[7]);
    acc[8] = fma(D62, mk, acc[8]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
    acc[4] = fma(D56, mk, acc[4]);
    acc[5] = fma(D59, mk, acc[5]);
    acc[6] = fma(D60, mk, acc[6]);
    acc[7] = fma(D62, mk, acc[7]);
    acc[8] = fma(D63, mk, acc[8]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D31, mk, acc[0]);
    acc[1] = fma(D46, mk, acc[1]);
    acc[2] = fma(D47, mk, acc[2]);
    acc[3] = fma(D48, mk, acc[3]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D32, mk, acc[0]);
    acc[1] = fma(D47, mk, acc[1]);
    acc[2] = fma(D49, mk, acc[2]);
    acc[3] = fma(D50, mk, acc[3]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D33, mk, acc[0]);
    acc[1] = fma(D48, mk, acc[1]);
    acc[2] = fma(D50, mk, acc[2]);
    acc[3] = fma(D51, mk, acc[3]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D34, mk, acc[0]);
    acc[1] = fma(D49, mk, acc[1]);
    acc[2] = fma(D52, mk, acc[2]);
    acc[3] = fma(D53, mk, acc[3]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D35, mk, acc[0]);
    acc[1] = fma(D50, mk, acc[1]);
    acc[2] = fma(D53, mk, acc[2]);
    acc[3] = fma(D54, mk, acc[3]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D37, mk, acc[0]);
    acc[1] = fma(D52, mk, acc[1]);
    acc[2] = fma(D55, mk, acc[2]);
    acc[3] = fma(D56, mk, acc[3]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D38, mk, acc[0]);
    acc[1] = fma(D53, mk, acc[1]);
    acc[2] = fma(D56, mk, acc[2]);
    acc[3] = fma(D57, mk, acc[3]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D40, mk, acc[0]);
    acc[1] = fma(D55, mk, acc[1]);
    acc[2] = fma(D58, mk, acc[2]);
    acc[3] = fma(D59, mk, acc[3]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D41, mk, acc[0]);
    acc[1] = fma(D56, mk, acc[1]);
    acc[2] = fma(D59, mk, acc[2]);
    acc[3] = fma(D60, mk, acc[3]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D43, mk, acc[0]);
    acc[1] = fma(D58, mk, acc[1]);
    acc[2] = fma(D61, mk, acc[2]);
    acc[3] = fma(D62, mk, acc[3]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D44, mk, acc[0]);
    acc[1] = fma(D59, mk, acc[1]);
    acc[2] = fma(D62, mk, acc[2]);
    acc[3] = fma(D63, mk, acc[3]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D46, mk, acc[0]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D47, mk, acc[0]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D48, mk, acc[0]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D49, mk, acc[0]);
  }
  { const T mk = Mb[36];
    acc[0] = fma(D50, mk, acc[0]);
  }
  { const T mk = Mb[37];
    acc[0] = fma(D52, mk, acc[0]);
  }
  { const T mk = Mb[38];
    acc[0] = fma(D53, mk, acc[0]);
  }
  { const T mk = Mb[39];
    acc[0] = fma(D55, mk, acc[0]);
  }
  { const T mk = Mb[40];
    acc[0] = fma(D56, mk, acc[0]);
  }
  { const T mk = Mb[41];
    acc[0] = fma(D58, mk, acc[0]);
  }
  { const T mk = Mb[42];
    acc[0] = fma(D59, mk, acc[0]);
  }
  { const T mk = Mb[43];
    acc[0] = fma(D61, mk, acc[0]);
  }
  { const T mk = Mb[44];
    acc[0] = fma(D62, mk, acc[0]);
  }
}
template <typename T>
__device__ __forceinline__ void dtensor_m2_p6(T x, T y, T z, T* __restrict__ Dout) {
  const T r2 = x * x + y * y + z * z;
  const T ir2 = T(1) / r2;
  const T D0 = rsqrt_t(r2);
  const T xr = x * ir2;
  const T yr = y * ir2;
  const T zr = z * ir2;
  const T x1_1 = crat<T>(-1, 1) * xr;
  const T D1 = x1_1 * D0;
  const T y1_1 = crat<T>(-1, 1) * yr;
  const T D2 = y1_1 * D0;
  const T z1_1 = crat<T>(-1, 1) * zr;
  const T D3 = z1_1 * D0;
  const T w2_2 = crat<T>(-2, 2) * ir2;
  const T x2_1 = crat<T>(-3, 2) * xr;
  const T x2_2 = T(2) * x2_1;
  const T D4 = fma(x2_2, D1, w2_2 * D0);
  const T y2_1 = crat<T>(-3, 2) * yr;
  const T D5 = fma(y2_1, D1, x2_1 * D2);
  const T z2_1 = crat<T>(-3, 2) * zr;
  const T D6 = fma(z2_1, D1, x2_1 * D3);
  const T y2_2 = T(2) * y2_1;
  const T D7 = fma(y2_2, D2, w2_2 * D0);
  const T D8 = fma(z2_1, D2, y2_1 * D3);
  const T D9 = -(D4 + D7);
  const T w3_3 = crat<T>(-12, 3) * ir2;
  const T x3_1 = crat<T>(-5, 3) * xr;
  const T x3_3 = T(3) * x3_1;
  const T D10 = fma(x3_3, D4, w3_3 * D1);
  const T w3_2 = crat<T>(-4, 3) * ir2;
  const T x3_2 = T(2) * x3_1;
  const T y3_1 = crat<T>(-5, 3) * yr;
  const T D11 = fma(y3_1, D4, fma(x3_2, D5, w3_2 * D2));
  const T z3_1 = crat<T>(-5, 3) * zr;
  const T D12 = fma(z3_1, D4, fma(x3_2, D6, w3_2 * D3));
  const T y3_2 = T(2) * y3_1;
  const T D13 = fma(y3_2, D5, fma(x3_1, D7, w3_2 * D1));
  const T D14 = fma(z3_1, D5, fma(y3_1, D6, x3_1 * D8));
  const T D15 = -(D10 + D13);
  const T y3_3 = T(3) * y3_1;
  const T D16 = fma(y3_3, D7, w3_3 * D2);
  const T D17 = fma(z3_1, D7, fma(y3_2, D8, w3_2 * D3));
  const T D18 = -(D11 + D16);
  const T w4_4 = crat<T>(-36, 4) * ir2;
  const T x4_1 = crat<T>(-7, 4) * xr;
  const T x4_4 = T(4) * x4_1;
  const T D19 = fma(x4_4, D10, w4_4 * D4);
  const T w4_3 = crat<T>(-18, 4) * ir2;
  const T x4_3 = T(3) * x4_1;
  const T y4_1 = crat<T>(-7, 4) * yr;
  const T D20 = fma(y4_1, D10, fma(x4_3, D11, w4_3 * D5));
  const T z4_1 = crat<T>(-7, 4) * zr;
  const T D21 = fma(z4_1, D10, fma(x4_3, D12, w4_3 * D6));
  const T w4_2 = crat<T>(-6, 4) * ir2;
  const T x4_2 = T(2) * x4_1;
  const T y4_2 = T(2) * y4_1;
  const T D22 = fma(y4_2, D11, fma(x4_2, D13, fma(w4_2, D4, w4_2 * D7)));
  const T D23 = fma(z4_1, D11, fma(y4_1, D12, fma(x4_2, D14, w4_2 * D8)));
  const T D24 = -(D19 + D22);
  const T y4_3 = T(3) * y4_1;
  const T D25 = fma(y4_3, D13, fma(x4_1, D16, w4_3 * D5));
  const T D26 = fma(z4_1, D13, fma(y4_2, D14, fma(x4_1, D17, w4_2 * D6)));
  const T D27 = -(D20 + D25);
  const T y4_4 = T(4) * y4_1;
  const T D28 = fma(y4_4, D16, w4_4 * D7);
  const T D29 = fma(z4_1, D16, fma(y4_3, D17, w4_3 * D8));
  const T D30 = -(D22 + D28);
  const T w5_5 = crat<T>(-80, 5) * ir2;
  const T x5_1 = crat<T>(-9, 5) * xr;
  const T x5_5 = T(5) * x5_1;
  const T D31 = fma(x5_5, D19, w5_5 * D10);
  const T w5_4 = crat<T>(-48, 5) * ir2;
  const T x5_4 = T(4) * x5_1;
  const T y5_1 = crat<T>(-9, 5) * yr;
  const T D32 = fma(y5_1, D19, fma(x5_4, D20, w5_4 * D11));
  const T z5_1 = crat<T>(-9, 5) * zr;
  const T D33 = fma(z5_1, D19, fma(x5_4, D21, w5_4 * D12));
  const T w5_3 = crat<T>(-24, 5) * ir2;
  const T w5_2 = crat<T>(-8, 5) * ir2;
  const T x5_3 = T(3) * x5_1;
  const T y5_2 = T(2) * y5_1;
  const T D34 = fma(y5_2, D20, fma(x5_3, D22, fma(w5_2, D10, w5_3 * D13)));
  const T D35 = fma(z5_1, D20, fma(y5_1, D21, fma(x5_3, D23, w5_3 * D14)));
  const T D36 = -(D31 + D34);
  const T x5_2 = T(2) * x5_1;
  const T y5_3 = T(3) * y5_1;
  const T D37 = fma(y5_3, D22, fma(x5_2, D25, fma(w5_3, D11, w5_2 * D16)));
  const T D38 = fma(z5_1, D22, fma(y5_2, D23, fma(x5_2, D26, fma(w5_2, D12, w5_2 * D17))));
  const T D39 = -(D32 + D37);
  const T y5_4 = T(4) * y5_1;
  const T D40 = fma(y5_4, D25, fma(x5_1, D28, w5_4 * D13));
  const T D41 = fma(z5_1, D25, fma(y5_3, D26, fma(x5_1, D29, w5_3 * D14)));
  const T D42 = -(D34 + D40);
  const T y5_5 = T(5) * y5_1;
  const T D43 = fma(y5_5, D28, w5_5 * D16);
  const T D44 = fma(z5_1, D28, fma(y5_4, D29, w5_4 * D17));
  const T D45 = -(D37 + D43);
  const T w6_6 = crat<T>(-150, 6) * ir2;
  const T x6_1 = crat<T>(-11, 6) * xr;
  const T x6_6 = T(6) * x6_1;
  const T D46 = fma(x6_6, D31, w6_6 * D19);
  const T w6_5 = crat<T>(-100, 6) * ir2;
  const T x6_5 = T(5) * x6_1;
  const T y6_1 = crat<T>(-11, 6) * yr;
  const T D47 = fma(y6_1, D31, fma(x6_5, D32, w6_5 * D20));
  const T z6_1 = crat<T>(-11, 6) * zr;
  const T D48 = fma(z6_1, D31, fma(x6_5, D33, w6_5 * D21));
  const T w6_4 = crat<T>(-60, 6) * ir2;
  const T w6_2 = crat<T>(-10, 6) * ir2;
  const T x6_4 = T(4) * x6_1;
  const T y6_2 = T(2) * y6_1;
  const T D49 = fma(y6_2, D32, fma(x6_4, D34, fma(w6_2, D19, w6_4 * D22)));
  const T D50 = fma(z6_1, D32, fma(y6_1, D33, fma(x6_4, D35, w6_4 * D23)));
  const T D51 = -(D46 + D49);
  const T w6_3 = crat<T>(-30, 6) * ir2;
  const T x6_3 = T(3) * x6_1;
  const T y6_3 = T(3) * y6_1;
  const T D52 = fma(y6_3, D34, fma(x6_3, D37, fma(w6_3, D20, w6_3 * D25)));
  const T D53 = fma(z6_1, D34, fma(y6_2, D35, fma(x6_3, D38, fma(w6_2, D21, w6_3 * D26))));
  const T D54 = -(D47 + D52);
  const T x6_2 = T(2) * x6_1;
  const T y6_4 = T(4) * y6_1;
  const T D55 = fma(y6_4, D37, fma(x6_2, D40, fma(w6_4, D22, w6_2 * D28)));
  const T D56 = fma(z6_1, D37, fma(y6_3, D38, fma(x6_2, D41, fma(w6_3, D23, w6_2 * D29))));
  const T D57 = -(D49 + D55);
  const T y6_5 = T(5) * y6_1;
  const T D58 = fma(y6_5, D40, fma(x6_1, D43, w6_5 * D25));
  const T D59 = fma(z6_1, D40, fma(y6_4, D41, fma(x6_1, D44, w6_4 * D26)));
  const T D60 = -(D52 + D58);
  const T y6_6 = T(6) * y6_1;
  const T D61 = fma(y6_6, D43, w6_6 * D28);
  const T D62 = fma(z6_1, D43, fma(y6_5, D44, w6_5 * D29));
  const T D63 = -(D55 + D61);
  Dout[0] = D0;
  Dout[1] = D1;
  Dout[2] = D2;
  Dout[3] = D3;
  Dout[4] = D4;
  Dout[5] = D5;
  Dout[6] = D6;
  Dout[7] = D7;
  Dout[8] = D8;
  Dout[9] = D9;
  Dout[10] = D10;
  Dout[11] = D11;
  Dout[12] = D12;
  Dout[13] = D13;
  Dout[14] = D14;
  Dout[15] = D15;
  Dout[16] = D16;
  Dout[17] = D17;
  Dout[18] = D18;
  Dout[19] = D19;
  Dout[20] = D20;
  Dout[21] = D21;
  Dout[22] = D22;
  Dout[23] = D23;
  Dout[24] = D24;
  Dout[25] = D25;
  Dout[26] = D26;
  Dout[27] = D27;
  Dout[28] = D28;
  Dout[29] = D29;
  Dout[30] = D30;
  Dout[31] = D31;
  Dout[32] = D32;
  Dout[33] = D33;
  Dout[34] = D34;
  Dout[35] = D35;
  Dout[36] = D36;
  Dout[37] = D37;
  Dout[38] = D38;
  Dout[39] = D39;
  Dout[40] = D40;
  Dout[41] = D41;
  Dout[42] = D42;
  Dout[43] = D43;
  Dout[44] = D44;
  Dout[45] = D45;
  Dout[46] = D46;
  Dout[47] = D47;
  Dout[48] = D48;
  Dout[49] = D49;
  Dout[50] = D50;
  Dout[51] = D51;
  Dout[52] = D52;
  Dout[53] = D53;
  Dout[54] = D54;
  Dout[55] = D55;
  Dout[56] = D56;
  Dout[57] = D57;
  Dout[58] = D58;
  Dout[59] = D59;
  Dout[60] = D60;
  Dout[61] = D61;
  Dout[62] = D62;
  Dout[63] = D63;
}
template <typename T>
__device__ __forceinline__ void m2l_m2_p6_pre(const T* __restrict__ Dt, const T* __restrict__ Mb, T* __restrict__ acc) {
  const T D0 = Dt[0];
  const T D1 = Dt[1];
  const T D2 = Dt[2];
  const T D3 = Dt[3];
  const T D4 = Dt[4];
  const T D5 = Dt[5];
  const T D6 = Dt[6];
  const T D7 = Dt[7];
  const T D8 = Dt[8];
  const T D9 = Dt[9];
  const T D10 = Dt[10];
  const T D11 = Dt[11];
  const T D12 = Dt[12];
  const T D13 = Dt[13];
  const T D14 = Dt[14];
  const T D15 = Dt[15];
  const T D16 = Dt[16];
  const T D17 = Dt[17];
  const T D18 = Dt[18];
  const T D19 = Dt[19];
  const T D20 = Dt[20];
  const T D21 = Dt[21];
  const T D22 = Dt[22];
  const T D23 = Dt[23];
  const T D24 = Dt[24];
  const T D25 = Dt[25];
  const T D26 = Dt[26];
  const T D27 = Dt[27];
  const T D28 = Dt[28];
  const T D29 = Dt[29];
  const T D30 = Dt[30];
  const T D31 = Dt[31];
  const T D32 = Dt[32];
  const T D33 = Dt[33];
  const T D34 = Dt[34];
  const T D35 = Dt[35];
  const T D36 = Dt[36];
  const T D37 = Dt[37];
  const T D38 = Dt[38];
  const T D39 = Dt[39];
  const T D40 = Dt[40];
  const T D41 = Dt[41];
  const T D42 = Dt[42];
  const T D43 = Dt[43];
  const T D44 = Dt[44];
  const T D45 = Dt[45];
  const T D46 = Dt[46];
  const T D47 = Dt[47];
  const T D48 = Dt[48];
  const T D49 = Dt[49];
  const T D50 = Dt[50];
  const T D51 = Dt[51];
  const T D52 = Dt[52];
  const T D53 = Dt[53];
  const T D54 = Dt[54];
  const T D55 = Dt[55];
  const T D56 = Dt[56];
  const T D57 = Dt[57];
  const T D58 = Dt[58];
  const T D59 = Dt[59];
  const T D60 = Dt[60];
  const T D61 = Dt[61];
  const T D62 = Dt[62];
  const T D63 = Dt[63];
  { const T mk = Mb[0];
    acc[0] = fma(D4, mk, acc[0]);
    acc[1] = fma(D10, mk, acc[1]);
    acc[2] = fma(D11, mk, acc[2]);
    acc[3] = fma(D12, mk, acc[3]);
    acc[4] = fma(D19, mk, acc[4]);
    acc[5] = fma(D20, mk, acc[5]);
    acc[6] = fma(D21, mk, acc[6]);
    acc[7] = fma(D22, mk, acc[7]);
    acc[8] = fma(D23, mk, acc[8]);
    acc[9] = fma(D31, mk, acc[9]);
    acc[10] = fma(D32, mk, acc[10]);
    acc[11] = fma(D33, mk, acc[11]);
    acc[12] = fma(D34, mk, acc[12]);
    acc[13] = fma(D35, mk, acc[13]);
    acc[14] = fma(D37, mk, acc[14]);
    acc[15] = fma(D38, mk, acc[15]);
    acc[16] = fma(D46, mk, acc[16]);
    acc[17] = fma(D47, mk, acc[17]);
    acc[18] = fma(D48, mk, acc[18]);
    acc[19] = fma(D49, mk, acc[19]);
    acc[20] = fma(D50, mk, acc[20]);
    acc[21] = fma(D52, mk, acc[21]);
    acc[22] = fma(D53, mk, acc[22]);
    acc[23] = fma(D55, mk, acc[23]);
    acc[24] = fma(D56, mk, acc[24]);
  }
  { const T mk = Mb[1];
    acc[0] = fma(D5, mk, acc[0]);
    acc[1] = fma(D11, mk, acc[1]);
    acc[2] = fma(D13, mk, acc[2]);
    acc[3] = fma(D14, mk, acc[3]);
    acc[4] = fma(D20, mk, acc[4]);
    acc[5] = fma(D22, mk, acc[5]);
    acc[6] = fma(D23, mk, acc[6]);
    acc[7] = fma(D25, mk, acc[7]);
    acc[8] = fma(D26, mk, acc[8]);
    acc[9] = fma(D32, mk, acc[9]);
    acc[10] = fma(D34, mk, acc[10]);
    acc[11] = fma(D35, mk, acc[11]);
    acc[12] = fma(D37, mk, acc[12]);
    acc[13] = fma(D38, mk, acc[13]);
    acc[14] = fma(D40, mk, acc[14]);
    acc[15] = fma(D41, mk, acc[15]);
    acc[16] = fma(D47, mk, acc[16]);
    acc[17] = fma(D49, mk, acc[17]);
    acc[18] = fma(D50, mk, acc[18]);
    acc[19] = fma(D52, mk, acc[19]);
    acc[20] = fma(D53, mk, acc[20]);
    acc[21] = fma(D55, mk, acc[21]);
    acc[22] = fma(D56, mk, acc[22]);
    acc[23] = fma(D58, mk, acc[23]);
    acc[24] = fma(D59, mk, acc[24]);
  }
  { const T mk = Mb[2];
    acc[0] = fma(D6, mk, acc[0]);
    acc[1] = fma(D12, mk, acc[1]);
    acc[2] = fma(D14, mk, acc[2]);
    acc[3] = fma(D15, mk, acc[3]);
    acc[4] = fma(D21, mk, acc[4]);
    acc[5] = fma(D23, mk, acc[5]);
    acc[6] = fma(D24, mk, acc[6]);
    acc[7] = fma(D26, mk, acc[7]);
    acc[8] = fma(D27, mk, acc[8]);
    acc[9] = fma(D33, mk, acc[9]);
    acc[10] = fma(D35, mk, acc[10]);
    acc[11] = fma(D36, mk, acc[11]);
    acc[12] = fma(D38, mk, acc[12]);
    acc[13] = fma(D39, mk, acc[13]);
    acc[14] = fma(D41, mk, acc[14]);
    acc[15] = fma(D42, mk, acc[15]);
    acc[16] = fma(D48, mk, acc[16]);
    acc[17] = fma(D50, mk, acc[17]);
    acc[18] = fma(D51, mk, acc[18]);
    acc[19] = fma(D53, mk, acc[19]);
    acc[20] = fma(D54, mk, acc[20]);
    acc[21] = fma(D56, mk, acc[21]);
    acc[22] = fma(D57, mk, acc[22]);
    acc[23] = fma(D59, mk, acc[23]);
    acc[24] = fma(D60, mk, acc[24]);
  }
  { const T mk = Mb[3];
    acc[0] = fma(D7, mk, acc[0]);
    acc[1] = fma(D13, mk, acc[1]);
    acc[2] = fma(D16, mk, acc[2]);
    acc[3] = fma(D17, mk, acc[3]);
    acc[4] = fma(D22, mk, acc[4]);
    acc[5] = fma(D25, mk, acc[5]);
    acc[6] = fma(D26, mk, acc[6]);
    acc[7] = fma(D28, mk, acc[7]);
    acc[8] = fma(D29, mk, acc[8]);
    acc[9] = fma(D34, mk, acc[9]);
    acc[10] = fma(D37, mk, acc[10]);
    acc[11] = fma(D38, mk, acc[11]);
    acc[12] = fma(D40, mk, acc[12]);
    acc[13] = fma(D41, mk, acc[13]);
    acc[14] = fma(D43, mk, acc[14]);
    acc[15] = fma(D44, mk, acc[15]);
    acc[16] = fma(D49, mk, acc[16]);
    acc[17] = fma(D52, mk, acc[17]);
    acc[18] = fma(D53, mk, acc[18]);
    acc[19] = fma(D55, mk, acc[19]);
    acc[20] = fma(D56, mk, acc[20]);
    acc[21] = fma(D58, mk, acc[21]);
    acc[22] = fma(D59, mk, acc[22]);
    acc[23] = fma(D61, mk, acc[23]);
    acc[24] = fma(D62, mk, acc[24]);
  }
  { const T mk = Mb[4];
    acc[0] = fma(D8, mk, acc[0]);
    acc[1] = fma(D14, mk, acc[1]);
    acc[2] = fma(D17, mk, acc[2]);
    acc[3] = fma(D18, mk, acc[3]);
    acc[4] = fma(D23, mk, acc[4]);
    acc[5] = fma(D26, mk, acc[5]);
    acc[6] = fma(D27, mk, acc[6]);
    acc[7] = fma(D29, mk, acc[7]);
    acc[8] = fma(D30, mk, acc[8]);
    acc[9] = fma(D35, mk, acc[9]);
    acc[10] = fma(D38, mk, acc[10]);
    acc[11] = fma(D39, mk, acc[11]);
    acc[12] = fma(D41, mk, acc[12]);
    acc[13] = fma(D42, mk, acc[13]);
    acc[14] = fma(D44, mk, acc[14]);
    acc[15] = fma(D45, mk, acc[15]);
    acc[16] = fma(D50, mk, acc[16]);
    acc[17] = fma(D53, mk, acc[17]);
    acc[18] = fma(D54, mk, acc[18]);
    acc[19] = fma(D56, mk, acc[19]);
    acc[20] = fma(D57, mk, acc[20]);
    acc[21] = fma(D59, mk, acc[21]);
    acc[22] = fma(D60, mk, acc[22]);
    acc[23] = fma(D62, mk, acc[23]);
    acc[24] = fma(D63, mk, acc[24]);
  }
  { const T mk = Mb[5];
    acc[0] = fma(D10, mk, acc[0]);
    acc[1] = fma(D19, mk, acc[1]);
    acc[2] = fma(D20, mk, acc[2]);
    acc[3] = fma(D21, mk, acc[3]);
    acc[4] = fma(D31, mk, acc[4]);
    acc[5] = fma(D32, mk, acc[5]);
    acc[6] = fma(D33, mk, acc[6]);
    acc[7] = fma(D34, mk, acc[7]);
    acc[8] = fma(D35, mk, acc[8]);
    acc[9] = fma(D46, mk, acc[9]);
    acc[10] = fma(D47, mk, acc[10]);
    acc[11] = fma(D48, mk, acc[11]);
    acc[12] = fma(D49, mk, acc[12]);
    acc[13] = fma(D50, mk, acc[13]);
    acc[14] = fma(D52, mk, acc[14]);
    acc[15] = fma(D53, mk, acc[15]);
  }
  { const T mk = Mb[6];
    acc[0] = fma(D11, mk, acc[0]);
    acc[1] = fma(D20, mk, acc[1]);
    acc[2] = fma(D22, mk, acc[2]);
    acc[3] = fma(D23, mk, acc[3]);
    acc[4] = fma(D32, mk, acc[4]);
    acc[5] = fma(D34, mk, acc[5]);
    acc[6] = fma(D35, mk, acc[6]);
    acc[7] = fma(D37, mk, acc[7]);
    acc[8] = fma(D38, mk, acc[8]);
    acc[9] = fma(D47, mk, acc[9]);
    acc[10] = fma(D49, mk, acc[10]);
    acc[11] = fma(D50, mk, acc[11]);
    acc[12] = fma(D52, mk, acc[12]);
    acc[13] = fma(D53, mk, acc[13]);
    acc[14] = fma(D55, mk, acc[14]);
    acc[15] = fma(D56, mk, acc[15]);
  }
  { const T mk = Mb[7];
    acc[0] = fma(D12, mk, acc[0]);
    acc[1] = fma(D21, mk, acc[1]);
    acc[2] = fma(D23, mk, acc[2]);
    acc[3] = fma(D24, mk, acc[3]);
    acc[4] = fma(D33, mk, acc[4]);
    acc[5] = fma(D35, mk, acc[5]);
    acc[6] = fma(D36, mk, acc[6]);
    acc[7] = fma(D38, mk, acc[7]);
    acc[8] = fma(D39, mk, acc[8]);
    acc[9] = fma(D48, mk, acc[9]);
    acc[10] = fma(D50, mk, acc[10]);
    acc[11] = fma(D51, mk, acc[11]);
    acc[12] = fma(D53, mk, acc[12]);
    acc[13] = fma(D54, mk, acc[13]);
    acc[14] = fma(D56, mk, acc[14]);
    acc[15] = fma(D57, mk, acc[15]);
  }
  { const T mk = Mb[8];
    acc[0] = fma(D13, mk, acc[0]);
    acc[1] = fma(D22, mk, acc[1]);
    acc[2] = fma(D25, mk, acc[2]);
    acc[3] = fma(D26, mk, acc[3]);
    acc[4] = fma(D34, mk, acc[4]);
    acc[5] = fma(D37, mk, acc[5]);
    acc[6] = fma(D38, mk, acc[6]);
    acc[7] = fma(D40, mk, acc[7]);
    acc[8] = fma(D41, mk, acc[8]);
    acc[9] = fma(D49, mk, acc[9]);
    acc[10] = fma(D52, mk, acc[10]);
    acc[11] = fma(D53, mk, acc[11]);
    acc[12] = fma(D55, mk, acc[12]);
    acc[13] = fma(D56, mk, acc[13]);
    acc[14] = fma(D58, mk, acc[14]);
    acc[15] = fma(D59, mk, acc[15]);
  }
  { const T mk = Mb[9];
    acc[0] = fma(D14, mk, acc[0]);
    acc[1] = fma(D23, mk, acc[1]);
    acc[2] = fma(D26, mk, acc[2]);
    acc[3] = fma(D27, mk, acc[3]);
    acc[4] = fma(D35, mk, acc[4]);
    acc[5] = fma(D38, mk, acc[5]);
    acc[6] = fma(D39, mk, acc[6]);
    acc[7] = fma(D41, mk, acc[7]);
    acc[8] = fma(D42, mk, acc[8]);
    acc[9] = fma(D50, mk, acc[9]);
    acc[10] = fma(D53, mk, acc[10]);
    acc[11] = fma(D54, mk, acc[11]);
    acc[12] = fma(D56, mk, acc[12]);
    acc[13] = fma(D57, mk, acc[13]);
    acc[14] = fma(D59, mk, acc[14]);
    acc[15] = fma(D60, mk, acc[15]);
  }
  { const T mk = Mb[10];
    acc[0] = fma(D16, mk, acc[0]);
    acc[1] = fma(D25, mk, acc[1]);
    acc[2] = fma(D28, mk, acc[2]);
    acc[3] = fma(D29, mk, acc[3]);
    acc[4] = fma(D37, mk, acc[4]);
    acc[5] = fma(D40, mk, acc[5]);
    acc[6] = fma(D41, mk, acc[6]);
    acc[7] = fma(D43, mk, acc[7]);
    acc[8] = fma(D44, mk, acc[8]);
    acc[9] = fma(D52, mk, acc[9]);
    acc[10] = fma(D55, mk, acc[10]);
    acc[11] = fma(D56, mk, acc[11]);
    acc[12] = fma(D58, mk, acc[12]);
    acc[13] = fma(D59, mk, acc[13]);
    acc[14] = fma(D61, mk, acc[14]);
    acc[15] = fma(D62, mk, acc[15]);
  }
  { const T mk = Mb[11];
    acc[0] = fma(D17, mk, acc[0]);
    acc[1] = fma(D26, mk, acc[1]);
    acc[2] = fma(D29, mk, acc[2]);
    acc[3] = fma(D30, mk, acc[3]);
    acc[4] = fma(D38, mk, acc[4]);
    acc[5] = fma(D41, mk, acc[5]);
    acc[6] = fma(D42, mk, acc[6]);
    acc[7] = fma(D44, mk, acc[7]);
    acc[8] = fma(D45, mk, acc[8]);
    acc[9] = fma(D53, mk, acc[9]);
    acc[10] = fma(D56, mk, acc[10]);
    acc[11] = fma(D57, mk, acc[11]);
    acc[12] = fma(D59, mk, acc[12]);
    acc[13] = fma(D60, mk, acc[13]);
    acc[14] = fma(D62, mk, acc[14]);
    acc[15] = fma(D63, mk, acc[15]);
  }
  { const T mk = Mb[12];
    acc[0] = fma(D19, mk, acc[0]);
    acc[1] = fma(D31, mk, acc[1]);
    acc[2] = fma(D32, mk, acc[2]);
    acc[3] = fma(D33, mk, acc[3]);
    acc[4] = fma(D46, mk, acc[4]);
    acc[5] = fma(D47, mk, acc[5]);
    acc[6] = fma(D48, mk, acc[6]);
    acc[7] = fma(D49, mk, acc[7]);
    acc[8] = fma(D50, mk, acc[8]);
  }
  { const T mk = Mb[13];
    acc[0] = fma(D20, mk, acc[0]);
    acc[1] = fma(D32, mk, acc[1]);
    acc[2] = fma(D34, mk, acc[2]);
    acc[3] = fma(D35, mk, acc[3]);
    acc[4] = fma(D47, mk, acc[4]);
    acc[5] = fma(D49, mk, acc[5]);
    acc[6] = fma(D50, mk, acc[6]);
    acc[7] = fma(D52, mk, acc[7]);
    acc[8] = fma(D53, mk, acc[8]);
  }
  { const T mk = Mb[14];
    acc[0] = fma(D21, mk, acc[0]);
    acc[1] = fma(D33, mk, acc[1]);
    acc[2] = fma(D35, mk, acc[2]);
    acc[3] = fma(D36, mk, acc[3]);
    acc[4] = fma(D48, mk, acc[4]);
    acc[5] = fma(D50, mk, acc[5]);
    acc[6] = fma(D51, mk, acc[6]);
    acc[7] = fma(D53, mk, acc[7]);
    acc[8] = fma(D54, mk, acc[8]);
  }
  { const T mk = Mb[15];
    acc[0] = fma(D22, mk, acc[0]);
    acc[1] = fma(D34, mk, acc[1]);
    acc[2] = fma(D37, mk, acc[2]);
    acc[3] = fma(D38, mk, acc[3]);
    acc[4] = fma(D49, mk, acc[4]);
    acc[5] = fma(D52, mk, acc[5]);
    acc[6] = fma(D53, mk, acc[6]);
    acc[7] = fma(D55, mk, acc[7]);
    acc[8] = fma(D56, mk, acc[8]);
  }
  { const T mk = Mb[16];
    acc[0] = fma(D23, mk, acc[0]);
    acc[1] = fma(D35, mk, acc[1]);
    acc[2] = fma(D38, mk, acc[2]);
    acc[3] = fma(D39, mk, acc[3]);
    acc[4] = fma(D50, mk, acc[4]);
    acc[5] = fma(D53, mk, acc[5]);
    acc[6] = fma(D54, mk, acc[6]);
    acc[7] = fma(D56, mk, acc[7]);
    acc[8] = fma(D57, mk, acc[8]);
  }
  { const T mk = Mb[17];
    acc[0] = fma(D25, mk, acc[0]);
    acc[1] = fma(D37, mk, acc[1]);
    acc[2] = fma(D40, mk, acc[2]);
    acc[3] = fma(D41, mk, acc[3]);
    acc[4] = fma(D52, mk, acc[4]);
    acc[5] = fma(D55, mk, acc[5]);
    acc[6] = fma(D56, mk, acc[6]);
    acc[7] = fma(D58, mk, acc[7]);
    acc[8] = fma(D59, mk, acc[8]);
  }
  { const T mk = Mb[18];
    acc[0] = fma(D26, mk, acc[0]);
    acc[1] = fma(D38, mk, acc[1]);
    acc[2] = fma(D41, mk, acc[2]);
    acc[3] = fma(D42, mk, acc[3]);
    acc[4] = fma(D53, mk, acc[4]);
    acc[5] = fma(D56, mk, acc[5]);
    acc[6] = fma(D57, mk, acc[6]);
    acc[7] = fma(D59, mk, acc[7]);
    acc[8] = fma(D60, mk, acc[8]);
  }
  { const T mk = Mb[19];
    acc[0] = fma(D28, mk, acc[0]);
    acc[1] = fma(D40, mk, acc[1]);
    acc[2] = fma(D43, mk, acc[2]);
    acc[3] = fma(D44, mk, acc[3]);
    acc[4] = fma(D55, mk, acc[4]);
    acc[5] = fma(D58, mk, acc[5]);
    acc[6] = fma(D59, mk, acc[6]);
    acc[7] = fma(D61, mk, acc[7]);
    acc[8] = fma(D62, mk, acc[8]);
  }
  { const T mk = Mb[20];
    acc[0] = fma(D29, mk, acc[0]);
    acc[1] = fma(D41, mk, acc[1]);
    acc[2] = fma(D44, mk, acc[2]);
    acc[3] = fma(D45, mk, acc[3]);
    acc[4] = fma(D56, mk, acc[4]);
    acc[5] = fma(D59, mk, acc[5]);
    acc[6] = fma(D60, mk, acc[6]);
    acc[7] = fma(D62, mk, acc[7]);
    acc[8] = fma(D63, mk, acc[8]);
  }
  { const T mk = Mb[21];
    acc[0] = fma(D31, mk, acc[0]);
    acc[1] = fma(D46, mk, acc[1]);
    acc[2] = fma(D47, mk, acc[2]);
    acc[3] = fma(D48, mk, acc[3]);
  }
  { const T mk = Mb[22];
    acc[0] = fma(D32, mk, acc[0]);
    acc[1] = fma(D47, mk, acc[1]);
    acc[2] = fma(D49, mk, acc[2]);
    acc[3] = fma(D50, mk, acc[3]);
  }
  { const T mk = Mb[23];
    acc[0] = fma(D33, mk, acc[0]);
    acc[1] = fma(D48, mk, acc[1]);
    acc[2] = fma(D50, mk, acc[2]);
    acc[3] = fma(D51, mk, acc[3]);
  }
  { const T mk = Mb[24];
    acc[0] = fma(D34, mk, acc[0]);
    acc[1] = fma(D49, mk, acc[1]);
    acc[2] = fma(D52, mk, acc[2]);
    acc[3] = fma(D53, mk, acc[3]);
  }
  { const T mk = Mb[25];
    acc[0] = fma(D35, mk, acc[0]);
    acc[1] = fma(D50, mk, acc[1]);
    acc[2] = fma(D53, mk, acc[2]);
    acc[3] = fma(D54, mk, acc[3]);
  }
  { const T mk = Mb[26];
    acc[0] = fma(D37, mk, acc[0]);
    acc[1] = fma(D52, mk, acc[1]);
    acc[2] = fma(D55, mk, acc[2]);
    acc[3] = fma(D56, mk, acc[3]);
  }
  { const T mk = Mb[27];
    acc[0] = fma(D38, mk, acc[0]);
    acc[1] = fma(D53, mk, acc[1]);
    acc[2] = fma(D56, mk, acc[2]);
    acc[3] = fma(D57, mk, acc[3]);
  }
  { const T mk = Mb[28];
    acc[0] = fma(D40, mk, acc[0]);
    acc[1] = fma(D55, mk, acc[1]);
    acc[2] = fma(D58, mk, acc[2]);
    acc[3] = fma(D59, mk, acc[3]);
  }
  { const T mk = Mb[29];
    acc[0] = fma(D41, mk, acc[0]);
    acc[1] = fma(D56, mk, acc[1]);
    acc[2] = fma(D59, mk, acc[2]);
    acc[3] = fma(D60, mk, acc[3]);
  }
  { const T mk = Mb[30];
    acc[0] = fma(D43, mk, acc[0]);
    acc[1] = fma(D58, mk, acc[1]);
    acc[2] = fma(D61, mk, acc[2]);
    acc[3] = fma(D62, mk, acc[3]);
  }
  { const T mk = Mb[31];
    acc[0] = fma(D44, mk, acc[0]);
    acc[1] = fma(D59, mk, acc[1]);
    acc[2] = fma(D62, mk, acc[2]);
    acc[3] = fma(D63, mk, acc[3]);
  }
  { const T mk = Mb[32];
    acc[0] = fma(D46, mk, acc[0]);
  }
  { const T mk = Mb[33];
    acc[0] = fma(D47, mk, acc[0]);
  }
  { const T mk = Mb[34];
    acc[0] = fma(D48, mk, acc[0]);
  }
  { const T mk = Mb[35];
    acc[0] = fma(D49, mk, acc[0]);
  }
  { const T mk = Mb[36];
    acc[0] = fma(D50, mk, acc[0]);
  }
  { const T mk = Mb[37];
    acc[0] = fma(D52, mk, acc[0]);
  }
  { const T mk = Mb[38];
    acc[0] = fma(D53, mk, acc[0]);
  }
  { const T mk = Mb[39];
    acc[0] = fma(D55, mk, acc[0]);
  }
  { const T mk = Mb[40];
    acc[0] = fma(D56, mk, acc[0]);
  }
  { const T mk = Mb[41];
    acc[0] = fma(D58, mk, acc[0]);
  }
  { const T mk = Mb[42];
    acc[0] = fma(D59, mk, acc[0]);
  }
  { const T mk = Mb[43];
    acc[0] = fma(D61, mk, acc[0]);
  }
  { const T mk = Mb[44];
    acc[0] = fma(D62, mk, acc[0]);
  }
}
static __constant__ unsigned char m2l_w_m2_p6[375] = {
  4, 10, 11, 12, 19, 20, 21, 22, 23, 31, 32, 33, 34, 35, 37, 38, 46, 47, 48, 49, 50, 52, 53, 55, 56, 5, 11, 13, 14, 20, 22, 23, 25, 26, 32, 34, 35, 37, 38, 40, 41, 47, 49, 50, 52, 53, 55, 56, 58, 59, 6, 12, 14, 15, 21, 23, 24, 26, 27, 33, 35, 36, 38, 39, 41, 42, 48, 50, 51, 53, 54, 56, 57, 59, 60, 7, 13, 16, 17, 22, 25, 26, 28, 29, 34, 37, 38, 40, 41, 43, 44, 49, 52, 53, 55, 56, 58, 59, 61, 62, 8, 14, 17, 18, 23, 26, 27, 29, 30, 35, 38, 39, 41, 42, 44, 45, 50, 53, 54, 56, 57, 59, 60, 62, 63, 10, 19, 20, 21, 31, 32, 33, 34, 35, 46, 47, 48, 49, 50, 52, 53, 11, 20, 22, 23, 32, 34, 35, 37, 38, 47, 49, 50, 52, 53, 55, 56, 12, 21, 23, 24, 33, 35, 36, 38, 39, 48, 50, 51, 53, 54, 56, 57, 13, 22, 25, 26, 34, 37, 38, 40, 41, 49, 52, 53, 55, 56, 58, 59, 14, 23, 26, 27, 35, 38, 39, 41, 42, 50, 53, 54, 56, 57, 59, 60, 16, 25, 28, 29, 37, 40, 41, 43, 44, 52, 55, 56, 58, 59, 61, 62, 17, 26, 29, 30, 38, 41, 42, 44, 45, 53, 56, 57, 59, 60, 62, 63, 19, 31, 32, 33, 46, 47, 48, 49, 50, 20, 32, 34, 35, 47, 49, 50, 52, 53, 21, 33, 35, 36, 48, 50, 51, 53, 54, 22, 34, 37, 38, 49, 52, 53, 55, 56, 23, 35, 38, 39, 50, 53, 54, 56, 57, 25, 37, 40, 41, 52, 55, 56, 58, 59, 26, 38, 41, 42, 53, 56, 57, 59, 60, 28, 40, 43, 44, 55, 58, 59, 61, 62, 29, 41, 44, 45, 56, 59, 60, 62, 63, 31, 46, 47, 48, 32, 47, 49, 50, 33, 48, 50, 51, 34, 49, 52, 53, 35, 50, 53, 54, 37, 52, 55, 56, 38, 53, 56, 57, 40, 55, 58, 59, 41, 56, 59, 60, 43, 58, 61, 62, 44, 59, 62, 63, 46, 47, 48, 49, 50, 52, 53, 55, 56, 58, 59, 61, 62};
static __device__ const signed char m2l_fold_m2_p6[45][6][2] = {
  {{0, 1}, {5, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{3, 1}, {5, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{6, 1}, {11, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{7, 1}, {14, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{8, 1}, {15, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{9, 1}, {11, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{12, 1}, {14, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{13, 1}, {15, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{16, 1}, {21, -1}, {30, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{17, 1}, {24, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{18, 1}, {25, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{19, 1}, {21, -1}, {28, -1}, {30, 2}, {0, 0}, {0, 0}},
  {{20, 1}, {29, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{22, 1}, {24, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{23, 1}, {25, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{26, 1}, {28, -1}, {30, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{27, 1}, {29, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{31, 1}, {36, -1}, {45, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{32, 1}, {39, -1}, {50, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{33, 1}, {40, -1}, {51, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{34, 1}, {36, -1}, {43, -1}, {45, 2}, {0, 0}, {0, 0}},
  {{35, 1}, {44, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{37, 1}, {39, -1}, {48, -1}, {50, 2}, {0, 0}, {0, 0}},
  {{38, 1}, {40, -1}, {49, -1}, {51, 2}, {0, 0}, {0, 0}},
  {{41, 1}, {43, -1}, {45, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{42, 1}, {44, -1}, {0, 0}, {0, 0}, {0, 0}, {0, 0}},
  {{46, 1}, {48, -1}, {50, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{47, 1}, {49, -1}, {51, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{52, 1}, {57, -1}, {66, 1}, {79, -1}, {0, 0}, {0, 0}},
  {{53, 1}, {60, -1}, {71, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{54, 1}, {61, -1}, {72, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{55, 1}, {57, -1}, {64, -1}, {66, 2}, {77, 1}, {79, -3}},
  {{56, 1}, {65, -1}, {78, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{58, 1}, {60, -1}, {69, -1}, {71, 2}, {0, 0}, {0, 0}},
  {{59, 1}, {61, -1}, {70, -1}, {72, 2}, {0, 0}, {0, 0}},
  {{62, 1}, {64, -1}, {66, 1}, {75, -1}, {77, 2}, {79, -3}},
  {{63, 1}, {65, -1}, {76, -1}, {78, 2}, {0, 0}, {0, 0}},
  {{67, 1}, {69, -1}, {71, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{68, 1}, {70, -1}, {72, 1}, {0, 0}, {0, 0}, {0, 0}},
  {{73, 1}, {75, -1}, {77, 1}, {79, -1}, {0, 0}, {0, 0}},
  {{74, 1}, {76, -1}, {78, 1}, {0, 0}, {0, 0}, {0, 0}},
};
static __device__ const signed char m2l_unfold_m2_p6[35][3][2] = {
  {{0, 1}, {0, 0}, {0, 0}},
  {{1, 1}, {0, 0}, {0, 0}},
  {{2, 1}, {0, 0}, {0, 0}},
  {{3, 1}, {0, 0}, {0, 0}},
  {{4, 1}, {0, 0}, {0, 0}},
  {{5, 1}, {0, 0}, {0, 0}},
  {{6, 1}, {0, 0}, {0, 0}},
  {{7, 1}, {0, 0}, {0, 0}},
  {{8, 1}, {0, 0}, {0, 0}},
  {{7, -1}, {4, -1}, {0, 0}},
  {{9, 1}, {0, 0}, {0, 0}},
  {{10, 1}, {0, 0}, {0, 0}},
  {{11, 1}, {0, 0}, {0, 0}},
  {{12, 1}, {0, 0}, {0, 0}},
  {{13, 1}, {0, 0}, {0, 0}},
  {{12, -1}, {9, -1}, {0, 0}},
  {{14, 1}, {0, 0}, {0, 0}},
  {{15, 1}, {0, 0}, {0, 0}},
  {{14, -1}, {10, -1}, {0, 0}},
  {{15, -1}, {11, -1}, {0, 0}},
  {{16, 1}, {0, 0}, {0, 0}},
  {{17, 1}, {0, 0}, {0, 0}},
  {{18, 1}, {0, 0}, {0, 0}},
  {{19, 1}, {0, 0}, {0, 0}},
  {{20, 1}, {0, 0}, {0, 0}},
  {{19, -1}, {16, -1}, {0, 0}},
  {{21, 1}, {0, 0}, {0, 0}},
  {{22, 1}, {0, 0}, {0, 0}},
  {{21, -1}, {17, -1}, {0, 0}},
  {{22, -1}, {18, -1}, {0, 0}},
  {{23, 1}, {0, 0}, {0, 0}},
  {{24, 1}, {0, 0}, {0, 0}},
  {{23, -1}, {19, -1}, {0, 0}},
  {{24, -1}, {20, -1}, {0, 0}},
  {{23, 1}, {19, 2}, {16, 1}},
};

// P2M of a dipole (s0, s1, s2) at offset (x, y, z) = centre - site, order 5
template <typename T>
__device__ __forceinline__ void p2m_m1_p5(T x, T y, T z, T s0, T s1, T s2, T* __restrict__ acc) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  { const T v = s0;
    acc[0] = fma(T(1), v, acc[0]);
    acc[3] = fma(px1, v, acc[3]);
    acc[4] = fma(py1, v, acc[4]);
    acc[5] = fma(pz1, v, acc[5]);
    acc[9] = fma(px2, v, acc[9]);
    acc[10] = fma(m_1_1_0, v, acc[10]);
    acc[11] = fma(m_1_0_1, v, acc[11]);
    acc[12] = fma(py2, v, acc[12]);
    acc[13] = fma(m_0_1_1, v, acc[13]);
    acc[14] = fma(pz2, v, acc[14]);
    acc[19] = fma(px3, v, acc[19]);
    acc[20] = fma(m_2_1_0, v, acc[20]);
    acc[21] = fma(m_2_0_1, v, acc[21]);
    acc[22] = fma(m_1_2_0, v, acc[22]);
    acc[23] = fma(m_1_1_1, v, acc[23]);
    acc[24] = fma(m_1_0_2, v, acc[24]);
    acc[25] = fma(py3, v, acc[25]);
    acc[26] = fma(m_0_2_1, v, acc[26]);
    acc[27] = fma(m_0_1_2, v, acc[27]);
    acc[28] = fma(pz3, v, acc[28]);
    acc[34] = fma(px4, v, acc[34]);
    acc[35] = fma(m_3_1_0, v, acc[35]);
    acc[36] = fma(m_3_0_1, v, acc[36]);
    acc[37] = fma(m_2_2_0, v, acc[37]);
    acc[38] = fma(m_2_1_1, v, acc[38]);
    acc[39] = fma(m_2_0_2, v, acc[39]);
    acc[40] = fma(m_1_3_0, v, acc[40]);
    acc[41] = fma(m_1_2_1, v, acc[41]);
    acc[42] = fma(m_1_1_2, v, acc[42]);
    acc[43] = fma(m_1_0_3, v, acc[43]);
    acc[44] = fma(py4, v, acc[44]);
    acc[45] = fma(m_0_3_1, v, acc[45]);
    acc[46] = fma(m_0_2_2, v, acc[46]);
    acc[47] = fma(m_0_1_3, v, acc[47]);
    acc[48] = fma(pz4, v, acc[48]);
  }
  { const T v = s1;
    acc[1] = fma(T(1), v, acc[1]);
    acc[4] = fma(px1, v, acc[4]);
    acc[6] = fma(py1, v, acc[6]);
    acc[7] = fma(pz1, v, acc[7]);
    acc[10] = fma(px2, v, acc[10]);
    acc[12] = fma(m_1_1_0, v, acc[12]);
    acc[13] = fma(m_1_0_1, v, acc[13]);
    acc[15] = fma(py2, v, acc[15]);
    acc[16] = fma(m_0_1_1, v, acc[16]);
    acc[17] = fma(pz2, v, acc[17]);
    acc[20] = fma(px3, v, acc[20]);
    acc[22] = fma(m_2_1_0, v, acc[22]);
    acc[23] = fma(m_2_0_1, v, acc[23]);
    acc[25] = fma(m_1_2_0, v, acc[25]);
    acc[26] = fma(m_1_1_1, v, acc[26]);
    acc[27] = fma(m_1_0_2, v, acc[27]);
    acc[29] = fma(py3, v, acc[29]);
    acc[30] = fma(m_0_2_1, v, acc[30]);
    acc[31] = fma(m_0_1_2, v, acc[31]);
    acc[32] = fma(pz3, v, acc[32]);
    acc[35] = fma(px4, v, acc[35]);
    acc[37] = fma(m_3_1_0, v, acc[37]);
    acc[38] = fma(m_3_0_1, v, acc[38]);
    acc[40] = fma(m_2_2_0, v, acc[40]);
    acc[41] = fma(m_2_1_1, v, acc[41]);
    acc[42] = fma(m_2_0_2, v, acc[42]);
    acc[44] = fma(m_1_3_0, v, acc[44]);
    acc[45] = fma(m_1_2_1, v, acc[45]);
    acc[46] = fma(m_1_1_2, v, acc[46]);
    acc[47] = fma(m_1_0_3, v, acc[47]);
    acc[49] = fma(py4, v, acc[49]);
    acc[50] = fma(m_0_3_1, v, acc[50]);
    acc[51] = fma(m_0_2_2, v, acc[51]);
    acc[52] = fma(m_0_1_3, v, acc[52]);
    acc[53] = fma(pz4, v, acc[53]);
  }
  { const T v = s2;
    acc[2] = fma(T(1), v, acc[2]);
    acc[5] = fma(px1, v, acc[5]);
    acc[7] = fma(py1, v, acc[7]);
    acc[8] = fma(pz1, v, acc[8]);
    acc[11] = fma(px2, v, acc[11]);
    acc[13] = fma(m_1_1_0, v, acc[13]);
    acc[14] = fma(m_1_0_1, v, acc[14]);
    acc[16] = fma(py2, v, acc[16]);
    acc[17] = fma(m_0_1_1, v, acc[17]);
    acc[18] = fma(pz2, v, acc[18]);
    acc[21] = fma(px3, v, acc[21]);
    acc[23] = fma(m_2_1_0, v, acc[23]);
    acc[24] = fma(m_2_0_1, v, acc[24]);
    acc[26] = fma(m_1_2_0, v, acc[26]);
    acc[27] = fma(m_1_1_1, v, acc[27]);
    acc[28] = fma(m_1_0_2, v, acc[28]);
    acc[30] = fma(py3, v, acc[30]);
    acc[31] = fma(m_0_2_1, v, acc[31]);
    acc[32] = fma(m_0_1_2, v, acc[32]);
    acc[33] = fma(pz3, v, acc[33]);
    acc[36] = fma(px4, v, acc[36]);
    acc[38] = fma(m_3_1_0, v, acc[38]);
    acc[39] = fma(m_3_0_1, v, acc[39]);
    acc[41] = fma(m_2_2_0, v, acc[41]);
    acc[42] = fma(m_2_1_1, v, acc[42]);
    acc[43] = fma(m_2_0_2, v, acc[43]);
    acc[45] = fma(m_1_3_0, v, acc[45]);
    acc[46] = fma(m_1_2_1, v, acc[46]);
    acc[47] = fma(m_1_1_2, v, acc[47]);
    acc[48] = fma(m_1_0_3, v, acc[48]);
    acc[50] = fma(py4, v, acc[50]);
    acc[51] = fma(m_0_3_1, v, acc[51]);
    acc[52] = fma(m_0_2_2, v, acc[52]);
    acc[53] = fma(m_0_1_3, v, acc[53]);
    acc[54] = fma(pz4, v, acc[54]);
  }
}
// M2M: multipole Mc about a centre at (x, y, z) from this one, order 5
template <typename T>
__device__ __forceinline__ void m2m_m1_p5(T x, T y, T z, const T* __restrict__ Mc, T* __restrict__ acc) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  { const T v = Mc[0];
    acc[0] = fma(T(1), v, acc[0]);
    acc[3] = fma(px1, v, acc[3]);
    acc[4] = fma(py1, v, acc[4]);
    acc[5] = fma(pz1, v, acc[5]);
    acc[9] = fma(px2, v, acc[9]);
    acc[10] = fma(m_1_1_0, v, acc[10]);
    acc[11] = fma(m_1_0_1, v, acc[11]);
    acc[12] = fma(py2, v, acc[12]);
    acc[13] = fma(m_0_1_1, v, acc[13]);
    acc[14] = fma(pz2, v, acc[14]);
    acc[19] = fma(px3, v, acc[19]);
    acc[20] = fma(m_2_1_0, v, acc[20]);
    acc[21] = fma(m_2_0_1, v, acc[21]);
    acc[22] = fma(m_1_2_0, v, acc[22]);
    acc[23] = fma(m_1_1_1, v, acc[23]);
    acc[24] = fma(m_1_0_2, v, acc[24]);
    acc[25] = fma(py3, v, acc[25]);
    acc[26] = fma(m_0_2_1, v, acc[26]);
    acc[27] = fma(m_0_1_2, v, acc[27]);
    acc[28] = fma(pz3, v, acc[28]);
    acc[34] = fma(px4, v, acc[34]);
    acc[35] = fma(m_3_1_0, v, acc[35]);
    acc[36] = fma(m_3_0_1, v, acc[36]);
    acc[37] = fma(m_2_2_0, v, acc[37]);
    acc[38] = fma(m_2_1_1, v, acc[38]);
    acc[39] = fma(m_2_0_2, v, acc[39]);
    acc[40] = fma(m_1_3_0, v, acc[40]);
    acc[41] = fma(m_1_2_1, v, acc[41]);
    acc[42] = fma(m_1_1_2, v, acc[42]);
    acc[43] = fma(m_1_0_3, v, acc[43]);
    acc[44] = fma(py4, v, acc[44]);
    acc[45] = fma(m_0_3_1, v, acc[45]);
    acc[46] = fma(m_0_2_2, v, acc[46]);
    acc[47] = fma(m_0_1_3, v, acc[47]);
    acc[48] = fma(pz4, v, acc[48]);
  }
  { const T v = Mc[1];
    acc[1] = fma(T(1), v, acc[1]);
    acc[4] = fma(px1, v, acc[4]);
    acc[6] = fma(py1, v, acc[6]);
    acc[7] = fma(pz1, v, acc[7]);
    acc[10] = fma(px2, v, acc[10]);
    acc[12] = fma(m_1_1_0, v, acc[12]);
    acc[13] = fma(m_1_0_1, v, acc[13]);
    acc[15] = fma(py2, v, acc[15]);
    acc[16] = fma(m_0_1_1, v, acc[16]);
    acc[17] = fma(pz2, v, acc[17]);
    acc[20] = fma(px3, v, acc[20]);
    acc[22] = fma(m_2_1_0, v, acc[22]);
    acc[23] = fma(m_2_0_1, v, acc[23]);
    acc[25] = fma(m_1_2_0, v, acc[25]);
    acc[26] = fma(m_1_1_1, v, acc[26]);
    acc[27] = fma(m_1_0_2, v, acc[27]);
    acc[29] = fma(py3, v, acc[29]);
    acc[30] = fma(m_0_2_1, v, acc[30]);
    acc[31] = fma(m_0_1_2, v, acc[31]);
    acc[32] = fma(pz3, v, acc[32]);
    acc[35] = fma(px4, v, acc[35]);
    acc[37] = fma(m_3_1_0, v, acc[37]);
    acc[38] = fma(m_3_0_1, v, acc[38]);
    acc[40] = fma(m_2_2_0, v, acc[40]);
    acc[41] = fma(m_2_1_1, v, acc[41]);
    acc[42] = fma(m_2_0_2, v, acc[42]);
    acc[44] = fma(m_1_3_0, v, acc[44]);
    acc[45] = fma(m_1_2_1, v, acc[45]);
    acc[46] = fma(m_1_1_2, v, acc[46]);
    acc[47] = fma(m_1_0_3, v, acc[47]);
    acc[49] = fma(py4, v, acc[49]);
    acc[50] = fma(m_0_3_1, v, acc[50]);
    acc[51] = fma(m_0_2_2, v, acc[51]);
    acc[52] = fma(m_0_1_3, v, acc[52]);
    acc[53] = fma(pz4, v, acc[53]);
  }
  { const T v = Mc[2];
    acc[2] = fma(T(1), v, acc[2]);
    acc[5] = fma(px1, v, acc[5]);
    acc[7] = fma(py1, v, acc[7]);
    acc[8] = fma(pz1, v, acc[8]);
    acc[11] = fma(px2, v, acc[11]);
    acc[13] = fma(m_1_1_0, v, acc[13]);
    acc[14] = fma(m_1_0_1, v, acc[14]);
    acc[16] = fma(py2, v, acc[16]);
    acc[17] = fma(m_0_1_1, v, acc[17]);
    acc[18] = fma(pz2, v, acc[18]);
    acc[21] = fma(px3, v, acc[21]);
    acc[23] = fma(m_2_1_0, v, acc[23]);
    acc[24] = fma(m_2_0_1, v, acc[24]);
    acc[26] = fma(m_1_2_0, v, acc[26]);
    acc[27] = fma(m_1_1_1, v, acc[27]);
    acc[28] = fma(m_1_0_2, v, acc[28]);
    acc[30] = fma(py3, v, acc[30]);
    acc[31] = fma(m_0_2_1, v, acc[31]);
    acc[32] = fma(m_0_1_2, v, acc[32]);
    acc[33] = fma(pz3, v, acc[33]);
    acc[36] = fma(px4, v, acc[36]);
    acc[38] = fma(m_3_1_0, v, acc[38]);
    acc[39] = fma(m_3_0_1, v, acc[39]);
    acc[41] = fma(m_2_2_0, v, acc[41]);
    acc[42] = fma(m_2_1_1, v, acc[42]);
    acc[43] = fma(m_2_0_2, v, acc[43]);
    acc[45] = fma(m_1_3_0, v, acc[45]);
    acc[46] = fma(m_1_2_1, v, acc[46]);
    acc[47] = fma(m_1_1_2, v, acc[47]);
    acc[48] = fma(m_1_0_3, v, acc[48]);
    acc[50] = fma(py4, v, acc[50]);
    acc[51] = fma(m_0_3_1, v, acc[51]);
    acc[52] = fma(m_0_2_2, v, acc[52]);
    acc[53] = fma(m_0_1_3, v, acc[53]);
    acc[54] = fma(pz4, v, acc[54]);
  }
  { const T v = Mc[3];
    acc[3] = fma(T(1), v, acc[3]);
    acc[9] = fma(px1, v, acc[9]);
    acc[10] = fma(py1, v, acc[10]);
    acc[11] = fma(pz1, v, acc[11]);
    acc[19] = fma(px2, v, acc[19]);
    acc[20] = fma(m_1_1_0, v, acc[20]);
    acc[21] = fma(m_1_0_1, v, acc[21]);
    acc[22] = fma(py2, v, acc[22]);
    acc[23] = fma(m_0_1_1, v, acc[23]);
    acc[24] = fma(pz2, v, acc[24]);
    acc[34] = fma(px3, v, acc[34]);
    acc[35] = fma(m_2_1_0, v, acc[35]);
    acc[36] = fma(m_2_0_1, v, acc[36]);
    acc[37] = fma(m_1_2_0, v, acc[37]);
    acc[38] = fma(m_1_1_1, v, acc[38]);
    acc[39] = fma(m_1_0_2, v, acc[39]);
    acc[40] = fma(py3, v, acc[40]);
    acc[41] = fma(m_0_2_1, v, acc[41]);
    acc[42] = fma(m_0_1_2, v, acc[42]);
    acc[43] = fma(pz3, v, acc[43]);
  }
  { const T v = Mc[4];
    acc[4] = fma(T(1), v, acc[4]);
    acc[10] = fma(px1, v, acc[10]);
    acc[12] = fma(py1, v, acc[12]);
    acc[13] = fma(pz1, v, acc[13]);
    acc[20] = fma(px2, v, acc[20]);
    acc[22] = fma(m_1_1_0, v, acc[22]);
    acc[23] = fma(m_1_0_1, v, acc[23]);
    acc[25] = fma(py2, v, acc[25]);
    acc[26] = fma(m_0_1_1, v, acc[26]);
    acc[27] = fma(pz2, v, acc[27]);
    acc[35] = fma(px3, v, acc[35]);
    acc[37] = fma(m_2_1_0, v, acc[37]);
    acc[38] = fma(m_2_0_1, v, acc[38]);
    acc[40] = fma(m_1_2_0, v, acc[40]);
    acc[41] = fma(m_1_1_1, v, acc[41]);
    acc[42] = fma(m_1_0_2, v, acc[42]);
    acc[44] = fma(py3, v, acc[44]);
    acc[45] = fma(m_0_2_1, v, acc[45]);
    acc[46] = fma(m_0_1_2, v, acc[46]);
    acc[47] = fma(pz3, v, acc[47]);
  }
  { const T v = Mc[5];
    acc[5] = fma(T(1), v, acc[5]);
    acc[11] = fma(px1, v, acc[11]);
    acc[13] = fma(py1, v, acc[13]);
    acc[14] = fma(pz1, v, acc[14]);
    acc[21] = fma(px2, v, acc[21]);
    acc[23] = fma(m_1_1_0, v, acc[23]);
    acc[24] = fma(m_1_0_1, v, acc[24]);
    acc[26] = fma(py2, v, acc[26]);
    acc[27] = fma(m_0_1_1, v, acc[27]);
    acc[28] = fma(pz2, v, acc[28]);
    acc[36] = fma(px3, v, acc[36]);
    acc[38] = fma(m_2_1_0, v, acc[38]);
    acc[39] = fma(m_2_0_1, v, acc[39]);
    acc[41] = fma(m_1_2_0, v, acc[41]);
    acc[42] = fma(m_1_1_1, v, acc[42]);
    acc[43] = fma(m_1_0_2, v, acc[43]);
    acc[45] = fma(py3, v, acc[45]);
    acc[46] = fma(m_0_2_1, v, acc[46]);
    acc[47] = fma(m_0_1_2, v, acc[47]);
    acc[48] = fma(pz3, v, acc[48]);
  }
  { const T v = Mc[6];
    acc[6] = fma(T(1), v, acc[6]);
    acc[12] = fma(px1, v, acc[12]);
    acc[15] = fma(py1, v, acc[15]);
    acc[16] = fma(pz1, v, acc[16]);
    acc[22] = fma(px2, v, acc[22]);
    acc[25] = fma(m_1_1_0, v, acc[25]);
    acc[26] = fma(m_1_0_1, v, acc[26]);
    acc[29] = fma(py2, v, acc[29]);
    acc[30] = fma(m_0_1_1, v, acc[30]);
    acc[31] = fma(pz2, v, acc[31]);
    acc[37] = fma(px3, v, acc[37]);
    acc[40] = fma(m_2_1_0, v, acc[40]);
    acc[41] = fma(m_2_0_1, v, acc[41]);
    acc[44] = fma(m_1_2_0, v, acc[44]);
    acc[45] = fma(m_1_1_1, v, acc[45]);
    acc[46] = fma(m_1_0_2, v, acc[46]);
    acc[49] = fma(py3, v, acc[49]);
    acc[50] = fma(m_0_2_1, v, acc[50]);
    acc[51] = fma(m_0_1_2, v, acc[51]);
    acc[52] = fma(pz3, v, acc[52]);
  }
  { const T v = Mc[7];
    acc[7] = fma(T(1), v, acc[7]);
    acc[13] = fma(px1, v, acc[13]);
    acc[16] = fma(py1, v, acc[16]);
    acc[17] = fma(pz1, v, acc[17]);
    acc[23] = fma(px2, v, acc[23]);
    acc[26] = fma(m_1_1_0, v, acc[26]);
    acc[27] = fma(m_1_0_1, v, acc[27]);
    acc[30] = fma(py2, v, acc[30]);
    acc[31] = fma(m_0_1_1, v, acc[31]);
    acc[32] = fma(pz2, v, acc[32]);
    acc[38] = fma(px3, v, acc[38]);
    acc[41] = fma(m_2_1_0, v, acc[41]);
    acc[42] = fma(m_2_0_1, v, acc[42]);
    acc[45] = fma(m_1_2_0, v, acc[45]);
    acc[46] = fma(m_1_1_1, v, acc[46]);
    acc[47] = fma(m_1_0_2, v, acc[47]);
    acc[50] = fma(py3, v, acc[50]);
    acc[51] = fma(m_0_2_1, v, acc[51]);
    acc[52] = fma(m_0_1_2, v, acc[52]);
    acc[53] = fma(pz3, v, acc[53]);
  }
  { const T v = Mc[8];
    acc[8] = fma(T(1), v, acc[8]);
    acc[14] = fma(px1, v, acc[14]);
    acc[17] = fma(py1, v, acc[17]);
    acc[18] = fma(pz1, v, acc[18]);
    acc[24] = fma(px2, v, acc[24]);
    acc[27] = fma(m_1_1_0, v, acc[27]);
    acc[28] = fma(m_1_0_1, v, acc[28]);
    acc[31] = fma(py2, v, acc[31]);
    acc[32] = fma(m_0_1_1, v, acc[32]);
    acc[33] = fma(pz2, v, acc[33]);
    acc[39] = fma(px3, v, acc[39]);
    acc[42] = fma(m_2_1_0, v, acc[42]);
    acc[43] = fma(m_2_0_1, v, acc[43]);
    acc[46] = fma(m_1_2_0, v, acc[46]);
    acc[47] = fma(m_1_1_1, v, acc[47]);
    acc[48] = fma(m_1_0_2, v, acc[48]);
    acc[51] = fma(py3, v, acc[51]);
    acc[52] = fma(m_0_2_1, v, acc[52]);
    acc[53] = fma(m_0_1_2, v, acc[53]);
    acc[54] = fma(pz3, v, acc[54]);
  }
  { const T v = Mc[9];
    acc[9] = fma(T(1), v, acc[9]);
    acc[19] = fma(px1, v, acc[19]);
    acc[20] = fma(py1, v, acc[20]);
    acc[21] = fma(pz1, v, acc[21]);
    acc[34] = fma(px2, v, acc[34]);
    acc[35] = fma(m_1_1_0, v, acc[35]);
    acc[36] = fma(m_1_0_1, v, acc[36]);
    acc[37] = fma(py2, v, acc[37]);
    acc[38] = fma(m_0_1_1, v, acc[38]);
    acc[39] = fma(pz2, v, acc[39]);
  }
  { const T v = Mc[10];
    acc[10] = fma(T(1), v, acc[10]);
    acc[20] = fma(px1, v, acc[20]);
    acc[22] = fma(py1, v, acc[22]);
    acc[23] = fma(pz1, v, acc[23]);
    acc[35] = fma(px2, v, acc[35]);
    acc[37] = fma(m_1_1_0, v, acc[37]);
    acc[38] = fma(m_1_0_1, v, acc[38]);
    acc[40] = fma(py2, v, acc[40]);
    acc[41] = fma(m_0_1_1, v, acc[41]);
    acc[42] = fma(pz2, v, acc[42]);
  }
  { const T v = Mc[11];
    acc[11] = fma(T(1), v, acc[11]);
    acc[21] = fma(px1, v, acc[21]);
    acc[23] = fma(py1, v, acc[23]);
    acc[24] = fma(pz1, v, acc[24]);
    acc[36] = fma(px2, v, acc[36]);
    acc[38] = fma(m_1_1_0, v, acc[38]);
    acc[39] = fma(m_1_0_1, v, acc[39]);
    acc[41] = fma(py2, v, acc[41]);
    acc[42] = fma(m_0_1_1, v, acc[42]);
    acc[43] = fma(pz2, v, acc[43]);
  }
  { const T v = Mc[12];
    acc[12] = fma(T(1), v, acc[12]);
    acc[22] = fma(px1, v, acc[22]);
    acc[25] = fma(py1, v, acc[25]);
    acc[26] = fma(pz1, v, acc[26]);
    acc[37] = fma(px2, v, acc[37]);
    acc[40] = fma(m_1_1_0, v, acc[40]);
    acc[41] = fma(m_1_0_1, v, acc[41]);
    acc[44] = fma(py2, v, acc[44]);
    acc[45] = fma(m_0_1_1, v, acc[45]);
    acc[46] = fma(pz2, v, acc[46]);
  }
  { const T v = Mc[13];
    acc[13] = fma(T(1), v, acc[13]);
    acc[23] = fma(px1, v, acc[23]);
    acc[26] = fma(py1, v, acc[26]);
    acc[27] = fma(pz1, v, acc[27]);
    acc[38] = fma(px2, v, acc[38]);
    acc[41] = fma(m_1_1_0, v, acc[41]);
    acc[42] = fma(m_1_0_1, v, acc[42]);
    acc[45] = fma(py2, v, acc[45]);
    acc[46] = fma(m_0_1_1, v, acc[46]);
    acc[47] = fma(pz2, v, acc[47]);
  }
  { const T v = Mc[14];
    acc[14] = fma(T(1), v, acc[14]);
    acc[24] = fma(px1, v, acc[24]);
    acc[27] = fma(py1, v, acc[27]);
    acc[28] = fma(pz1, v, acc[28]);
    acc[39] = fma(px2, v, acc[39]);
    acc[42] = fma(m_1_1_0, v, acc[42]);
    acc[43] = fma(m_1_0_1, v, acc[43]);
    acc[46] = fma(py2, v, acc[46]);
    acc[47] = fma(m_0_1_1, v, acc[47]);
    acc[48] = fma(pz2, v, acc[48]);
  }
  { const T v = Mc[15];
    acc[15] = fma(T(1), v, acc[15]);
    acc[25] = fma(px1, v, acc[25]);
    acc[29] = fma(py1, v, acc[29]);
    acc[30] = fma(pz1, v, acc[30]);
    acc[40] = fma(px2, v, acc[40]);
    acc[44] = fma(m_1_1_0, v, acc[44]);
    acc[45] = fma(m_1_0_1, v, acc[45]);
    acc[49] = fma(py2, v, acc[49]);
    acc[50] = fma(m_0_1_1, v, acc[50]);
    acc[51] = fma(pz2, v, acc[51]);
  }
  { const T v = Mc[16];
    acc[16] = fma(T(1), v, acc[16]);
    acc[26] = fma(px1, v, acc[26]);
    acc[30] = fma(py1, v, acc[30]);
    acc[31] = fma(pz1, v, acc[31]);
    acc[41] = fma(px2, v, acc[41]);
    acc[45] = fma(m_1_1_0, v, acc[45]);
    acc[46] = fma(m_1_0_1, v, acc[46]);
    acc[50] = fma(py2, v, acc[50]);
    acc[51] = fma(m_0_1_1, v, acc[51]);
    acc[52] = fma(pz2, v, acc[52]);
  }
  { const T v = Mc[17];
    acc[17] = fma(T(1), v, acc[17]);
    acc[27] = fma(px1, v, acc[27]);
    acc[31] = fma(py1, v, acc[31]);
    acc[32] = fma(pz1, v, acc[32]);
    acc[42] = fma(px2, v, acc[42]);
    acc[46] = fma(m_1_1_0, v, acc[46]);
    acc[47] = fma(m_1_0_1, v, acc[47]);
    acc[51] = fma(py2, v, acc[51]);
    acc[52] = fma(m_0_1_1, v, acc[52]);
    acc[53] = fma(pz2, v, acc[53]);
  }
  { const T v = Mc[18];
    acc[18] = fma(T(1), v, acc[18]);
    acc[28] = fma(px1, v, acc[28]);
    acc[32] = fma(py1, v, acc[32]);
    acc[33] = fma(pz1, v, acc[33]);
    acc[43] = fma(px2, v, acc[43]);
    acc[47] = fma(m_1_1_0, v, acc[47]);
    acc[48] = fma(m_1_0_1, v, acc[48]);
    acc[52] = fma(py2, v, acc[52]);
    acc[53] = fma(m_0_1_1, v, acc[53]);
    acc[54] = fma(pz2, v, acc[54]);
  }
  { const T v = Mc[19];
    acc[19] = fma(T(1), v, acc[19]);
    acc[34] = fma(px1, v, acc[34]);
    acc[35] = fma(py1, v, acc[35]);
    acc[36] = fma(pz1, v, acc[36]);
  }
  { const T v = Mc[20];
    acc[20] = fma(T(1), v, acc[20]);
    acc[35] = fma(px1, v, acc[35]);
    acc[37] = fma(py1, v, acc[37]);
    acc[38] = fma(pz1, v, acc[38]);
  }
  { const T v = Mc[21];
    acc[21] = fma(T(1), v, acc[21]);
    acc[36] = fma(px1, v, acc[36]);
    acc[38] = fma(py1, v, acc[38]);
    acc[39] = fma(pz1, v, acc[39]);
  }
  { const T v = Mc[22];
    acc[22] = fma(T(1), v, acc[22]);
    acc[37] = fma(px1, v, acc[37]);
    acc[40] = fma(py1, v, acc[40]);
    acc[41] = fma(pz1, v, acc[41]);
  }
  { const T v = Mc[23];
    acc[23] = fma(T(1), v, acc[23]);
    acc[38] = fma(px1, v, acc[38]);
    acc[41] = fma(py1, v, acc[41]);
    acc[42] = fma(pz1, v, acc[42]);
  }
  { const T v = Mc[24];
    acc[24] = fma(T(1), v, acc[24]);
    acc[39] = fma(px1, v, acc[39]);
    acc[42] = fma(py1, v, acc[42]);
    acc[43] = fma(pz1, v, acc[43]);
  }
  { const T v = Mc[25];
    acc[25] = fma(T(1), v, acc[25]);
    acc[40] = fma(px1, v, acc[40]);
    acc[44] = fma(py1, v, acc[44]);
    acc[45] = fma(pz1, v, acc[45]);
  }
  { const T v = Mc[26];
    acc[26] = fma(T(1), v, acc[26]);
    acc[41] = fma(px1, v, acc[41]);
    acc[45] = fma(py1, v, acc[45]);
    acc[46] = fma(pz1, v, acc[46]);
  }
  { const T v = Mc[27];
    acc[27] = fma(T(1), v, acc[27]);
    acc[42] = fma(px1, v, acc[42]);
    acc[46] = fma(py1, v, acc[46]);
    acc[47] = fma(pz1, v, acc[47]);
  }
  { const T v = Mc[28];
    acc[28] = fma(T(1), v, acc[28]);
    acc[43] = fma(px1, v, acc[43]);
    acc[47] = fma(py1, v, acc[47]);
    acc[48] = fma(pz1, v, acc[48]);
  }
  { const T v = Mc[29];
    acc[29] = fma(T(1), v, acc[29]);
    acc[44] = fma(px1, v, acc[44]);
    acc[49] = fma(py1, v, acc[49]);
    acc[50] = fma(pz1, v, acc[50]);
  }
  { const T v = Mc[30];
    acc[30] = fma(T(1), v, acc[30]);
    acc[45] = fma(px1, v, acc[45]);
    acc[50] = fma(py1, v, acc[50]);
    acc[51] = fma(pz1, v, acc[51]);
  }
  { const T v = Mc[31];
    acc[31] = fma(T(1), v, acc[31]);
    acc[46] = fma(px1, v, acc[46]);
    acc[51] = fma(py1, v, acc[51]);
    acc[52] = fma(pz1, v, acc[52]);
  }
  { const T v = Mc[32];
    acc[32] = fma(T(1), v, acc[32]);
    acc[47] = fma(px1, v, acc[47]);
    acc[52] = fma(py1, v, acc[52]);
    acc[53] = fma(pz1, v, acc[53]);
  }
  { const T v = Mc[33];
    acc[33] = fma(T(1), v, acc[33]);
    acc[48] = fma(px1, v, acc[48]);
    acc[53] = fma(py1, v, acc[53]);
    acc[54] = fma(pz1, v, acc[54]);
  }
  { const T v = Mc[34];
    acc[34] = fma(T(1), v, acc[34]);
  }
  { const T v = Mc[35];
    acc[35] = fma(T(1), v, acc[35]);
  }
  { const T v = Mc[36];
    acc[36] = fma(T(1), v, acc[36]);
  }
  { const T v = Mc[37];
    acc[37] = fma(T(1), v, acc[37]);
  }
  { const T v = Mc[38];
    acc[38] = fma(T(1), v, acc[38]);
  }
  { const T v = Mc[39];
    acc[39] = fma(T(1), v, acc[39]);
  }
  { const T v = Mc[40];
    acc[40] = fma(T(1), v, acc[40]);
  }
  { const T v = Mc[41];
    acc[41] = fma(T(1), v, acc[41]);
  }
  { const T v = Mc[42];
    acc[42] = fma(T(1), v, acc[42]);
  }
  { const T v = Mc[43];
    acc[43] = fma(T(1), v, acc[43]);
  }
  { const T v = Mc[44];
    acc[44] = fma(T(1), v, acc[44]);
  }
  { const T v = Mc[45];
    acc[45] = fma(T(1), v, acc[45]);
  }
  { const T v = Mc[46];
    acc[46] = fma(T(1), v, acc[46]);
  }
  { const T v = Mc[47];
    acc[47] = fma(T(1), v, acc[47]);
  }
  { const T v = Mc[48];
    acc[48] = fma(T(1), v, acc[48]);
  }
  { const T v = Mc[49];
    acc[49] = fma(T(1), v, acc[49]);
  }
  { const T v = Mc[50];
    acc[50] = fma(T(1), v, acc[50]);
  }
  { const T v = Mc[51];
    acc[51] = fma(T(1), v, acc[51]);
  }
  { const T v = Mc[52];
    acc[52] = fma(T(1), v, acc[52]);
  }
  { const T v = Mc[53];
    acc[53] = fma(T(1), v, acc[53]);
  }
  { const T v = Mc[54];
    acc[54] = fma(T(1), v, acc[54]);
  }
}
// L2L: local expansion Lc about a centre at -(x, y, z) from this one, order 5
template <typename T>
__device__ __forceinline__ void l2l_m1_p5(T x, T y, T z, const T* __restrict__ Lc, T* __restrict__ acc) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  { const T v = Lc[0];
    acc[0] = fma(T(1), v, acc[0]);
  }
  { const T v = Lc[1];
    acc[0] = fma(px1, v, acc[0]);
    acc[1] = fma(T(1), v, acc[1]);
  }
  { const T v = Lc[2];
    acc[0] = fma(py1, v, acc[0]);
    acc[2] = fma(T(1), v, acc[2]);
  }
  { const T v = Lc[3];
    acc[0] = fma(pz1, v, acc[0]);
    acc[3] = fma(T(1), v, acc[3]);
  }
  { const T v = Lc[4];
    acc[0] = fma(px2, v, acc[0]);
    acc[1] = fma(px1, v, acc[1]);
    acc[4] = fma(T(1), v, acc[4]);
  }
  { const T v = Lc[5];
    acc[0] = fma(m_1_1_0, v, acc[0]);
    acc[1] = fma(py1, v, acc[1]);
    acc[2] = fma(px1, v, acc[2]);
    acc[5] = fma(T(1), v, acc[5]);
  }
  { const T v = Lc[6];
    acc[0] = fma(m_1_0_1, v, acc[0]);
    acc[1] = fma(pz1, v, acc[1]);
    acc[3] = fma(px1, v, acc[3]);
    acc[6] = fma(T(1), v, acc[6]);
  }
  { const T v = Lc[7];
    acc[0] = fma(py2, v, acc[0]);
    acc[2] = fma(py1, v, acc[2]);
    acc[7] = fma(T(1), v, acc[7]);
  }
  { const T v = Lc[8];
    acc[0] = fma(m_0_1_1, v, acc[0]);
    acc[2] = fma(pz1, v, acc[2]);
    acc[3] = fma(py1, v, acc[3]);
    acc[8] = fma(T(1), v, acc[8]);
  }
  { const T v = Lc[9];
    acc[0] = fma(pz2, v, acc[0]);
    acc[3] = fma(pz1, v, acc[3]);
    acc[9] = fma(T(1), v, acc[9]);
  }
  { const T v = Lc[10];
    acc[0] = fma(px3, v, acc[0]);
    acc[1] = fma(px2, v, acc[1]);
    acc[4] = fma(px1, v, acc[4]);
    acc[10] = fma(T(1), v, acc[10]);
  }
  { const T v = Lc[11];
    acc[0] = fma(m_2_1_0, v, acc[0]);
    acc[1] = fma(m_1_1_0, v, acc[1]);
    acc[2] = fma(px2, v, acc[2]);
    acc[4] = fma(py1, v, acc[4]);
    acc[5] = fma(px1, v, acc[5]);
    acc[11] = fma(T(1), v, acc[11]);
  }
  { const T v = Lc[12];
    acc[0] = fma(m_2_0_1, v, acc[0]);
    acc[1] = fma(m_1_0_1, v, acc[1]);
    acc[3] = fma(px2, v, acc[3]);
    acc[4] = fma(pz1, v, acc[4]);
    acc[6] = fma(px1, v, acc[6]);
    acc[12] = fma(T(1), v, acc[12]);
  }
  { const T v = Lc[13];
    acc[0] = fma(m_1_2_0, v, acc[0]);
    acc[1] = fma(py2, v, acc[1]);
    acc[2] = fma(m_1_1_0, v, acc[2]);
    acc[5] = fma(py1, v, acc[5]);
    acc[7] = fma(px1, v, acc[7]);
    acc[13] = fma(T(1), v, acc[13]);
  }
  { const T v = Lc[14];
    acc[0] = fma(m_1_1_1, v, acc[0]);
    acc[1] = fma(m_0_1_1, v, acc[1]);
    acc[2] = fma(m_1_0_1, v, acc[2]);
    acc[3] = fma(m_1_1_0, v, acc[3]);
    acc[5] = fma(pz1, v, acc[5]);
    acc[6] = fma(py1, v, acc[6]);
    acc[8] = fma(px1, v, acc[8]);
    acc[14] = fma(T(1), v, acc[14]);
  }
  { const T v = Lc[15];
    acc[0] = fma(m_1_0_2, v, acc[0]);
    acc[1] = fma(pz2, v, acc[1]);
    acc[3] = fma(m_1_0_1, v, acc[3]);
    acc[6] = fma(pz1, v, acc[6]);
    acc[9] = fma(px1, v, acc[9]);
    acc[15] = fma(T(1), v, acc[15]);
  }
  { const T v = Lc[16];
    acc[0] = fma(py3, v, acc[0]);
    acc[2] = fma(py2, v, acc[2]);
    acc[7] = fma(py1, v, acc[7]);
    acc[16] = fma(T(1), v, acc[16]);
  }
  { const T v = Lc[17];
    acc[0] = fma(m_0_2_1, v, acc[0]);
    acc[2] = fma(m_0_1_1, v, acc[2]);
    acc[3] = fma(py2, v, acc[3]);
    acc[7] = fma(pz1, v, acc[7]);
    acc[8] = fma(py1, v, acc[8]);
    acc[17] = fma(T(1), v, acc[17]);
  }
  { const T v = Lc[18];
    acc[0] = fma(m_0_1_2, v, acc[0]);
    acc[2] = fma(pz2, v, acc[2]);
    acc[3] = fma(m_0_1_1, v, acc[3]);
    acc[8] = fma(pz1, v, acc[8]);
    acc[9] = fma(py1, v, acc[9]);
    acc[18] = fma(T(1), v, acc[18]);
  }
  { const T v = Lc[19];
    acc[0] = fma(pz3, v, acc[0]);
    acc[3] = fma(pz2, v, acc[3]);
    acc[9] = fma(pz1, v, acc[9]);
    acc[19] = fma(T(1), v, acc[19]);
  }
  { const T v = Lc[20];
    acc[0] = fma(px4, v, acc[0]);
    acc[1] = fma(px3, v, acc[1]);
    acc[4] = fma(px2, v, acc[4]);
    acc[10] = fma(px1, v, acc[10]);
    acc[20] = fma(T(1), v, acc[20]);
  }
  { const T v = Lc[21];
    acc[0] = fma(m_3_1_0, v, acc[0]);
    acc[1] = fma(m_2_1_0, v, acc[1]);
    acc[2] = fma(px3, v, acc[2]);
    acc[4] = fma(m_1_1_0, v, acc[4]);
    acc[5] = fma(px2, v, acc[5]);
    acc[10] = fma(py1, v, acc[10]);
    acc[11] = fma(px1, v, acc[11]);
    acc[21] = fma(T(1), v, acc[21]);
  }
  { const T v = Lc[22];
    acc[0] = fma(m_3_0_1, v, acc[0]);
    acc[1] = fma(m_2_0_1, v, acc[1]);
    acc[3] = fma(px3, v, acc[3]);
    acc[4] = fma(m_1_0_1, v, acc[4]);
    acc[6] = fma(px2, v, acc[6]);
    acc[10] = fma(pz1, v, acc[10]);
    acc[12] = fma(px1, v, acc[12]);
    acc[22] = fma(T(1), v, acc[22]);
  }
  { const T v = Lc[23];
    acc[0] = fma(m_2_2_0, v, acc[0]);
    acc[1] = fma(m_1_2_0, v, acc[1]);
    acc[2] = fma(m_2_1_0, v, acc[2]);
    acc[4] = fma(py2, v, acc[4]);
    acc[5] = fma(m_1_1_0, v, acc[5]);
    acc[7] = fma(px2, v, acc[7]);
    acc[11] = fma(py1, v, acc[11]);
    acc[13] = fma(px1, v, acc[13]);
    acc[23] = fma(T(1), v, acc[23]);
  }
  { const T v = Lc[24];
    acc[0] = fma(m_2_1_1, v, acc[0]);
    acc[1] = fma(m_1_1_1, v, acc[1]);
    acc[2] = fma(m_2_0_1, v, acc[2]);
    acc[3] = fma(m_2_1_0, v, acc[3]);
    acc[4] = fma(m_0_1_1, v, acc[4]);
    acc[5] = fma(m_1_0_1, v, acc[5]);
    acc[6] = fma(m_1_1_0, v, acc[6]);
    acc[8] = fma(px2, v, acc[8]);
    acc[11] = fma(pz1, v, acc[11]);
    acc[12] = fma(py1, v, acc[12]);
    acc[14] = fma(px1, v, acc[14]);
    acc[24] = fma(T(1), v, acc[24]);
  }
  { const T v = Lc[25];
    acc[0] = fma(m_2_0_2, v, acc[0]);
    acc[1] = fma(m_1_0_2, v, acc[1]);
    acc[3] = fma(m_2_0_1, v, acc[3]);
    acc[4] = fma(pz2, v, acc[4]);
    acc[6] = fma(m_1_0_1, v, acc[6]);
    acc[9] = fma(px2, v, acc[9]);
    acc[12] = fma(pz1, v, acc[12]);
    acc[15] = fma(px1, v, acc[15]);
    acc[25] = fma(T(1), v, acc[25]);
  }
  { const T v = Lc[26];
    acc[0] = fma(m_1_3_0, v, acc[0]);
    acc[1] = fma(py3, v, acc[1]);
    acc[2] = fma(m_1_2_0, v, acc[2]);
    acc[5] = fma(py2, v, acc[5]);
    acc[7] = fma(m_1_1_0, v, acc[7]);
    acc[13] = fma(py1, v, acc[13]);
    acc[16] = fma(px1, v, acc[16]);
    acc[26] = fma(T(1), v, acc[26]);
  }
  { const T v = Lc[27];
    acc[0] = fma(m_1_2_1, v, acc[0]);
    acc[1] = fma(m_0_2_1, v, acc[1]);
    acc[2] = fma(m_1_1_1, v, acc[2]);
    acc[3] = fma(m_1_2_0, v, acc[3]);
    acc[5] = fma(m_0_1_1, v, acc[5]);
    acc[6] = fma(py2, v, acc[6]);
    acc[7] = fma(m_1_0_1, v, acc[7]);
    acc[8] = fma(m_1_1_0, v, acc[8]);
    acc[13] = fma(pz1, v, acc[13]);
    acc[14] = fma(py1, v, acc[14]);
    acc[17] = fma(px1, v, acc[17]);
    acc[27] = fma(T(1), v, acc[27]);
  }
  { const T v = Lc[28];
    acc[0] = fma(m_1_1_2, v, acc[0]);
    acc[1] = fma(m_0_1_2, v, acc[1]);
    acc[2] = fma(m_1_0_2, v, acc[2]);
    acc[3] = fma(m_1_1_1, v, acc[3]);
    acc[5] = fma(pz2, v, acc[5]);
    acc[6] = fma(m_0_1_1, v, acc[6]);
    acc[8] = fma(m_1_0_1, v, acc[8]);
    acc[9] = fma(m_1_1_0, v, acc[9]);
    acc[14] = fma(pz1, v, acc[14]);
    acc[15] = fma(py1, v, acc[15]);
    acc[18] = fma(px1, v, acc[18]);
    acc[28] = fma(T(1), v, acc[28]);
  }
  { const T v = Lc[29];
    acc[0] = fma(m_1_0_3, v, acc[0]);
    acc[1] = fma(pz3, v, acc[1]);
    acc[3] = fma(m_1_0_2, v, acc[3]);
    acc[6] = fma(pz2, v, acc[6]);
    acc[9] = fma(m_1_0_1, v, acc[9]);
    acc[15] = fma(pz1, v, acc[15]);
    acc[19] = fma(px1, v, acc[19]);
    acc[29] = fma(T(1), v, acc[29]);
  }
  { const T v = Lc[30];
    acc[0] = fma(py4, v, acc[0]);
    acc[2] = fma(py3, v, acc[2]);
    acc[7] = fma(py2, v, acc[7]);
    acc[16] = fma(py1, v, acc[16]);
    acc[30] = fma(T(1), v, acc[30]);
  }
  { const T v = Lc[31];
    acc[0] = fma(m_0_3_1, v, acc[0]);
    acc[2] = fma(m_0_2_1, v, acc[2]);
    acc[3] = fma(py3, v, acc[3]);
    acc[7] = fma(m_0_1_1, v, acc[7]);
    acc[8] = fma(py2, v, acc[8]);
    acc[16] = fma(pz1, v, acc[16]);
    acc[17] = fma(py1, v, acc[17]);
    acc[31] = fma(T(1), v, acc[31]);
  }
  { const T v = Lc[32];
    acc[0] = fma(m_0_2_2, v, acc[0]);
    acc[2] = fma(m_0_1_2, v, acc[2]);
    acc[3] = fma(m_0_2_1, v, acc[3]);
    acc[7] = fma(pz2, v, acc[7]);
    acc[8] = fma(m_0_1_1, v, acc[8]);
    acc[9] = fma(py2, v, acc[9]);
    acc[17] = fma(pz1, v, acc[17]);
    acc[18] = fma(py1, v, acc[18]);
    acc[32] = fma(T(1), v, acc[32]);
  }
  { const T v = Lc[33];
    acc[0] = fma(m_0_1_3, v, acc[0]);
    acc[2] = fma(pz3, v, acc[2]);
    acc[3] = fma(m_0_1_2, v, acc[3]);
    acc[8] = fma(pz2, v, acc[8]);
    acc[9] = fma(m_0_1_1, v, acc[9]);
    acc[18] = fma(pz1, v, acc[18]);
    acc[19] = fma(py1, v, acc[19]);
    acc[33] = fma(T(1), v, acc[33]);
  }
  { const T v = Lc[34];
    acc[0] = fma(pz4, v, acc[0]);
    acc[3] = fma(pz3, v, acc[3]);
    acc[9] = fma(pz2, v, acc[9]);
    acc[19] = fma(pz1, v, acc[19]);
    acc[34] = fma(T(1), v, acc[34]);
  }
}
// L2P: field -grad of the local expansion Lc at offset (x, y, z) = site - centre, order 5
template <typename T>
__device__ __forceinline__ void l2p_m1_p5(T x, T y, T z, const T* __restrict__ Lc, T& f0, T& f1, T& f2) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  { const T v = -Lc[1];
    f0 = fma(T(1), v, f0);
  }
  { const T v = -Lc[2];
    f1 = fma(T(1), v, f1);
  }
  { const T v = -Lc[3];
    f2 = fma(T(1), v, f2);
  }
  { const T v = -Lc[4];
    f0 = fma(px1, v, f0);
  }
  { const T v = -Lc[5];
    f0 = fma(py1, v, f0);
    f1 = fma(px1, v, f1);
  }
  { const T v = -Lc[6];
    f0 = fma(pz1, v, f0);
    f2 = fma(px1, v, f2);
  }
  { const T v = -Lc[7];
    f1 = fma(py1, v, f1);
  }
  { const T v = -Lc[8];
    f1 = fma(pz1, v, f1);
    f2 = fma(py1, v, f2);
  }
  { const T v = -Lc[9];
    f2 = fma(pz1, v, f2);
  }
  { const T v = -Lc[10];
    f0 = fma(px2, v, f0);
  }
  { const T v = -Lc[11];
    f0 = fma(m_1_1_0, v, f0);
    f1 = fma(px2, v, f1);
  }
  { const T v = -Lc[12];
    f0 = fma(m_1_0_1, v, f0);
    f2 = fma(px2, v, f2);
  }
  { const T v = -Lc[13];
    f0 = fma(py2, v, f0);
    f1 = fma(m_1_1_0, v, f1);
  }
  { const T v = -Lc[14];
    f0 = fma(m_0_1_1, v, f0);
    f1 = fma(m_1_0_1, v, f1);
    f2 = fma(m_1_1_0, v, f2);
  }
  { const T v = -Lc[15];
    f0 = fma(pz2, v, f0);
    f2 = fma(m_1_0_1, v, f2);
  }
  { const T v = -Lc[16];
    f1 = fma(py2, v, f1);
  }
  { const T v = -Lc[17];
    f1 = fma(m_0_1_1, v, f1);
    f2 = fma(py2, v, f2);
  }
  { const T v = -Lc[18];
    f1 = fma(pz2, v, f1);
    f2 = fma(m_0_1_1, v, f2);
  }
  { const T v = -Lc[19];
    f2 = fma(pz2, v, f2);
  }
  { const T v = -Lc[20];
    f0 = fma(px3, v, f0);
  }
  { const T v = -Lc[21];
    f0 = fma(m_2_1_0, v, f0);
    f1 = fma(px3, v, f1);
  }
  { const T v = -Lc[22];
    f0 = fma(m_2_0_1, v, f0);
    f2 = fma(px3, v, f2);
  }
  { const T v = -Lc[23];
    f0 = fma(m_1_2_0, v, f0);
    f1 = fma(m_2_1_0, v, f1);
  }
  { const T v = -Lc[24];
    f0 = fma(m_1_1_1, v, f0);
    f1 = fma(m_2_0_1, v, f1);
    f2 = fma(m_2_1_0, v, f2);
  }
  { const T v = -Lc[25];
    f0 = fma(m_1_0_2, v, f0);
    f2 = fma(m_2_0_1, v, f2);
  }
  { const T v = -Lc[26];
    f0 = fma(py3, v, f0);
    f1 = fma(m_1_2_0, v, f1);
  }
  { const T v = -Lc[27];
    f0 = fma(m_0_2_1, v, f0);
    f1 = fma(m_1_1_1, v, f1);
    f2 = fma(m_1_2_0, v, f2);
  }
  { const T v = -Lc[28];
    f0 = fma(m_0_1_2, v, f0);
    f1 = fma(m_1_0_2, v, f1);
    f2 = fma(m_1_1_1, v, f2);
  }
  { const T v = -Lc[29];
    f0 = fma(pz3, v, f0);
    f2 = fma(m_1_0_2, v, f2);
  }
  { const T v = -Lc[30];
    f1 = fma(py3, v, f1);
  }
  { const T v = -Lc[31];
    f1 = fma(m_0_2_1, v, f1);
    f2 = fma(py3, v, f2);
  }
  { const T v = -Lc[32];
    f1 = fma(m_0_1_2, v, f1);
    f2 = fma(m_0_2_1, v, f2);
  }
  { const T v = -Lc[33];
    f1 = fma(pz3, v, f1);
    f2 = fma(m_0_1_2, v, f2);
  }
  { const T v = -Lc[34];
    f2 = fma(pz3, v, f2);
  }
}

// P2M of a dipole (s0, s1, s2) at offset (x, y, z) = centre - site, order 6
template <typename T>
__device__ __forceinline__ void p2m_m1_p6(T x, T y, T z, T s0, T s1, T s2, T* __restrict__ acc) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T px5 = px4 * x * cinv<T>(5);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T py5 = py4 * y * cinv<T>(5);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T pz5 = pz4 * z * cinv<T>(5);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  const T m_4_1_0 = px4 * py1;
  const T m_4_0_1 = px4 * pz1;
  const T m_3_2_0 = px3 * py2;
  const T m_3_1_1 = px3 * py1 * pz1;
  const T m_3_0_2 = px3 * pz2;
  const T m_2_3_0 = px2 * py3;
  const T m_2_2_1 = px2 * py2 * pz1;
  const T m_2_1_2 = px2 * py1 * pz2;
  const T m_2_0_3 = px2 * pz3;
  const T m_1_4_0 = px1 * py4;
  const T m_1_3_1 = px1 * py3 * pz1;
  const T m_1_2_2 = px1 * py2 * pz2;
  const T m_1_1_3 = px1 * py1 * pz3;
  const T m_1_0_4 = px1 * pz4;
  const T m_0_4_1 = py4 * pz1;
  const T m_0_3_2 = py3 * pz2;
  const T m_0_2_3 = py2 * pz3;
  const T m_0_1_4 = py1 * pz4;
  { const T v = s0;
    acc[0] = fma(T(1), v, acc[0]);
    acc[3] = fma(px1, v, acc[3]);
    acc[4] = fma(py1, v, acc[4]);
    acc[5] = fma(pz1, v, acc[5]);
    acc[9] = fma(px2, v, acc[9]);
    acc[10] = fma(m_1_1_0, v, acc[10]);
    acc[11] = fma(m_1_0_1, v, acc[11]);
    acc[12] = fma(py2, v, acc[12]);
    acc[13] = fma(m_0_1_1, v, acc[13]);
    acc[14] = fma(pz2, v, acc[14]);
    acc[19] = fma(px3, v, acc[19]);
    acc[20] = fma(m_2_1_0, v, acc[20]);
    acc[21] = fma(m_2_0_1, v, acc[21]);
    acc[22] = fma(m_1_2_0, v, acc[22]);
    acc[23] = fma(m_1_1_1, v, acc[23]);
    acc[24] = fma(m_1_0_2, v, acc[24]);
    acc[25] = fma(py3, v, acc[25]);
    acc[26] = fma(m_0_2_1, v, acc[26]);
    acc[27] = fma(m_0_1_2, v, acc[27]);
    acc[28] = fma(pz3, v, acc[28]);
    acc[34] = fma(px4, v, acc[34]);
    acc[35] = fma(m_3_1_0, v, acc[35]);
    acc[36] = fma(m_3_0_1, v, acc[36]);
    acc[37] = fma(m_2_2_0, v, acc[37]);
    acc[38] = fma(m_2_1_1, v, acc[38]);
    acc[39] = fma(m_2_0_2, v, acc[39]);
    acc[40] = fma(m_1_3_0, v, acc[40]);
    acc[41] = fma(m_1_2_1, v, acc[41]);
    acc[42] = fma(m_1_1_2, v, acc[42]);
    acc[43] = fma(m_1_0_3, v, acc[43]);
    acc[44] = fma(py4, v, acc[44]);
    acc[45] = fma(m_0_3_1, v, acc[45]);
    acc[46] = fma(m_0_2_2, v, acc[46]);
    acc[47] = fma(m_0_1_3, v, acc[47]);
    acc[48] = fma(pz4, v, acc[48]);
    acc[55] = fma(px5, v, acc[55]);
    acc[56] = fma(m_4_1_0, v, acc[56]);
    acc[57] = fma(m_4_0_1, v, acc[57]);
    acc[58] = fma(m_3_2_0, v, acc[58]);
    acc[59] = fma(m_3_1_1, v, acc[59]);
    acc[60] = fma(m_3_0_2, v, acc[60]);
    acc[61] = fma(m_2_3_0, v, acc[61]);
    acc[62] = fma(m_2_2_1, v, acc[62]);
    acc[63] = fma(m_2_1_2, v, acc[63]);
    acc[64] = fma(m_2_0_3, v, acc[64]);
    acc[65] = fma(m_1_4_0, v, acc[65]);
    acc[66] = fma(m_1_3_1, v, acc[66]);
    acc[67] = fma(m_1_2_2, v, acc[67]);
    acc[68] = fma(m_1_1_3, v, acc[68]);
    acc[69] = fma(m_1_0_4, v, acc[69]);
    acc[70] = fma(py5, v, acc[70]);
    acc[71] = fma(m_0_4_1, v, acc[71]);
    acc[72] = fma(m_0_3_2, v, acc[72]);
    acc[73] = fma(m_0_2_3, v, acc[73]);
    acc[74] = fma(m_0_1_4, v, acc[74]);
    acc[75] = fma(pz5, v, acc[75]);
  }
  { const T v = s1;
    acc[1] = fma(T(1), v, acc[1]);
    acc[4] = fma(px1, v, acc[4]);
    acc[6] = fma(py1, v, acc[6]);
    acc[7] = fma(pz1, v, acc[7]);
    acc[10] = fma(px2, v, acc[10]);
    acc[12] = fma(m_1_1_0, v, acc[12]);
    acc[13] = fma(m_1_0_1, v, acc[13]);
    acc[15] = fma(py2, v, acc[15]);
    acc[16] = fma(m_0_1_1, v, acc[16]);
    acc[17] = fma(pz2, v, acc[17]);
    acc[20] = fma(px3, v, acc[20]);
    acc[22] = fma(m_2_1_0, v, acc[22]);
    acc[23] = fma(m_2_0_1, v, acc[23]);
    acc[25] = fma(m_1_2_0, v, acc[25]);
    acc[26] = fma(m_1_1_1, v, acc[26]);
    acc[27] = fma(m_1_0_2, v, acc[27]);
    acc[29] = fma(py3, v, acc[29]);
    acc[30] = fma(m_0_2_1, v, acc[30]);
    acc[31] = fma(m_0_1_2, v, acc[31]);
    acc[32] = fma(pz3, v, acc[32]);
    acc[35] = fma(px4, v, acc[35]);
    acc[37] = fma(m_3_1_0, v, acc[37]);
    acc[38] = fma(m_3_0_1, v, acc[38]);
    acc[40] = fma(m_2_2_0, v, acc[40]);
    acc[41] = fma(m_2_1_1, v, acc[41]);
    acc[42] = fma(m_2_0_2, v, acc[42]);
    acc[44] = fma(m_1_3_0, v, acc[44]);
    acc[45] = fma(m_1_2_1, v, acc[45]);
    acc[46] = fma(m_1_1_2, v, acc[46]);
    acc[47] = fma(m_1_0_3, v, acc[47]);
    acc[49] = fma(py4, v, acc[49]);
    acc[50] = fma(m_0_3_1, v, acc[50]);
    acc[51] = fma(m_0_2_2, v, acc[51]);
    acc[52] = fma(m_0_1_3, v, acc[52]);
    acc[53] = fma(pz4, v, acc[53]);
    acc[56] = fma(px5, v, acc[56]);
    acc[58] = fma(m_4_1_0, v, acc[58]);
    acc[59] = fma(m_4_0_1, v, acc[59]);
    acc[61] = fma(m_3_2_0, v, acc[61]);
    acc[62] = fma(m_3_1_1, v, acc[62]);
    acc[63] = fma(m_3_0_2, v, acc[63]);
    acc[65] = fma(m_2_3_0, v, acc[65]);
    acc[66] = fma(m_2_2_1, v, acc[66]);
    acc[67] = fma(m_2_1_2, v, acc[67]);
    acc[68] = fma(m_2_0_3, v, acc[68]);
    acc[70] = fma(m_1_4_0, v, acc[70]);
    acc[71] = fma(m_1_3_1, v, acc[71]);
    acc[72] = fma(m_1_2_2, v, acc[72]);
    acc[73] = fma(m_1_1_3, v, acc[73]);
    acc[74] = fma(m_1_0_4, v, acc[74]);
    acc[76] = fma(py5, v, acc[76]);
    acc[77] = fma(m_0_4_1, v, acc[77]);
    acc[78] = fma(m_0_3_2, v, acc[78]);
    acc[79] = fma(m_0_2_3, v, acc[79]);
    acc[80] = fma(m_0_1_4, v, acc[80]);
    acc[81] = fma(pz5, v, acc[81]);
  }
  { const T v = s2;
    acc[2] = fma(T(1), v, acc[2]);
    acc[5] = fma(px1, v, acc[5]);
    acc[7] = fma(py1, v, acc[7]);
    acc[8] = fma(pz1, v, acc[8]);
    acc[11] = fma(px2, v, acc[11]);
    acc[13] = fma(m_1_1_0, v, acc[13]);
    acc[14] = fma(m_1_0_1, v, acc[14]);
    acc[16] = fma(py2, v, acc[16]);
    acc[17] = fma(m_0_1_1, v, acc[17]);
    acc[18] = fma(pz2, v, acc[18]);
    acc[21] = fma(px3, v, acc[21]);
    acc[23] = fma(m_2_1_0, v, acc[23]);
    acc[24] = fma(m_2_0_1, v, acc[24]);
    acc[26] = fma(m_1_2_0, v, acc[26]);
    acc[27] = fma(m_1_1_1, v, acc[27]);
    acc[28] = fma(m_1_0_2, v, acc[28]);
    acc[30] = fma(py3, v, acc[30]);
    acc[31] = fma(m_0_2_1, v, acc[31]);
    acc[32] = fma(m_0_1_2, v, acc[32]);
    acc[33] = fma(pz3, v, acc[33]);
    acc[36] = fma(px4, v, acc[36]);
    acc[38] = fma(m_3_1_0, v, acc[38]);
    acc[39] = fma(m_3_0_1, v, acc[39]);
    acc[41] = fma(m_2_2_0, v, acc[41]);
    acc[42] = fma(m_2_1_1, v, acc[42]);
    acc[43] = fma(m_2_0_2, v, acc[43]);
    acc[45] = fma(m_1_3_0, v, acc[45]);
    acc[46] = fma(m_1_2_1, v, acc[46]);
    acc[47] = fma(m_1_1_2, v, acc[47]);
    acc[48] = fma(m_1_0_3, v, acc[48]);
    acc[50] = fma(py4, v, acc[50]);
    acc[51] = fma(m_0_3_1, v, acc[51]);
    acc[52] = fma(m_0_2_2, v, acc[52]);
    acc[53] = fma(m_0_1_3, v, acc[53]);
    acc[54] = fma(pz4, v, acc[54]);
    acc[57] = fma(px5, v, acc[57]);
    acc[59] = fma(m_4_1_0, v, acc[59]);
    acc[60] = fma(m_4_0_1, v, acc[60]);
    acc[62] = fma(m_3_2_0, v, acc[62]);
    acc[63] = fma(m_3_1_1, v, acc[63]);
    acc[64] = fma(m_3_0_2, v, acc[64]);
    acc[66] = fma(m_2_3_0, v, acc[66]);
    acc[67] = fma(m_2_2_1, v, acc[67]);
    acc[68] = fma(m_2_1_2, v, acc[68]);
    acc[69] = fma(m_2_0_3, v, acc[69]);
    acc[71] = fma(m_1_4_0, v, acc[71]);
    acc[72] = fma(m_1_3_1, v, acc[72]);
    acc[73] = fma(m_1_2_2, v, acc[73]);
    acc[74] = fma(m_1_1_3, v, acc[74]);
    acc[75] = fma(m_1_0_4, v, acc[75]);
    acc[77] = fma(py5, v, acc[77]);
    acc[78] = fma(m_0_4_1, v, acc[78]);
    acc[79] = fma(m_0_3_2, v, acc[79]);
    acc[80] = fma(m_0_2_3, v, acc[80]);
    acc[81] = fma(m_0_1_4, v, acc[81]);
    acc[82] = fma(pz5, v, acc[82]);
  }
}
// M2M: multipole Mc about a centre at (x, y, z) from this one, order 6
template <typename T>
__device__ __forceinline__ void m2m_m1_p6(T x, T y, T z, const T* __restrict__ Mc, T* __restrict__ acc) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T px5 = px4 * x * cinv<T>(5);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T py5 = py4 * y * cinv<T>(5);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T pz5 = pz4 * z * cinv<T>(5);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  const T m_4_1_0 = px4 * py1;
  const T m_4_0_1 = px4 * pz1;
  const T m_3_2_0 = px3 * py2;
  const T m_3_1_1 = px3 * py1 * pz1;
  const T m_3_0_2 = px3 * pz2;
  const T m_2_3_0 = px2 * py3;
  const T m_2_2_1 = px2 * py2 * pz1;
  const T m_2_1_2 = px2 * py1 * pz2;
  const T m_2_0_3 = px2 * pz3;
  const T m_1_4_0 = px1 * py4;
  const T m_1_3_1 = px1 * py3 * pz1;
  const T m_1_2_2 = px1 * py2 * pz2;
  const T m_1_1_3 = px1 * py1 * pz3;
  const T m_1_0_4 = px1 * pz4;
  const T m_0_4_1 = py4 * pz1;
  const T m_0_3_2 = py3 * pz2;
  const T m_0_2_3 = py2 * pz3;
  const T m_0_1_4 = py1 * pz4;
  { const T v = Mc[0];
    acc[0] = fma(T(1), v, acc[0]);
    acc[3] = fma(px1, v, acc[3]);
    acc[4] = fma(py1, v, acc[4]);
    acc[5] = fma(pz1, v, acc[5]);
    acc[9] = fma(px2, v, acc[9]);
    acc[10] = fma(m_1_1_0, v, acc[10]);
    acc[11] = fma(m_1_0_1, v, acc[11]);
    acc[12] = fma(py2, v, acc[12]);
    acc[13] = fma(m_0_1_1, v, acc[13]);
    acc[14] = fma(pz2, v, acc[14]);
    acc[19] = fma(px3, v, acc[19]);
    acc[20] = fma(m_2_1_0, v, acc[20]);
    acc[21] = fma(m_2_0_1, v, acc[21]);
    acc[22] = fma(m_1_2_0, v, acc[22]);
    acc[23] = fma(m_1_1_1, v, acc[23]);
    acc[24] = fma(m_1_0_2, v, acc[24]);
    acc[25] = fma(py3, v, acc[25]);
    acc[26] = fma(m_0_2_1, v, acc[26]);
    acc[27] = fma(m_0_1_2, v, acc[27]);
    acc[28] = fma(pz3, v, acc[28]);
    acc[34] = fma(px4, v, acc[34]);
    acc[35] = fma(m_3_1_0, v, acc[35]);
    acc[36] = fma(m_3_0_1, v, acc[36]);
    acc[37] = fma(m_2_2_0, v, acc[37]);
    acc[38] = fma(m_2_1_1, v, acc[38]);
    acc[39] = fma(m_2_0_2, v, acc[39]);
    acc[40] = fma(m_1_3_0, v, acc[40]);
    acc[41] = fma(m_1_2_1, v, acc[41]);
    acc[42] = fma(m_1_1_2, v, acc[42]);
    acc[43] = fma(m_1_0_3, v, acc[43]);
    acc[44] = fma(py4, v, acc[44]);
    acc[45] = fma(m_0_3_1, v, acc[45]);
    acc[46] = fma(m_0_2_2, v, acc[46]);
    acc[47] = fma(m_0_1_3, v, acc[47]);
    acc[48] = fma(pz4, v, acc[48]);
    acc[55] = fma(px5, v, acc[55]);
    acc[56] = fma(m_4_1_0, v, acc[56]);
    acc[57] = fma(m_4_0_1, v, acc[57]);
    acc[58] = fma(m_3_2_0, v, acc[58]);
    acc[59] = fma(m_3_1_1, v, acc[59]);
    acc[60] = fma(m_3_0_2, v, acc[60]);
    acc[61] = fma(m_2_3_0, v, acc[61]);
    acc[62] = fma(m_2_2_1, v, acc[62]);
    acc[63] = fma(m_2_1_2, v, acc[63]);
    acc[64] = fma(m_2_0_3, v, acc[64]);
    acc[65] = fma(m_1_4_0, v, acc[65]);
    acc[66] = fma(m_1_3_1, v, acc[66]);
    acc[67] = fma(m_1_2_2, v, acc[67]);
    acc[68] = fma(m_1_1_3, v, acc[68]);
    acc[69] = fma(m_1_0_4, v, acc[69]);
    acc[70] = fma(py5, v, acc[70]);
    acc[71] = fma(m_0_4_1, v, acc[71]);
    acc[72] = fma(m_0_3_2, v, acc[72]);
    acc[73] = fma(m_0_2_3, v, acc[73]);
    acc[74] = fma(m_0_1_4, v, acc[74]);
    acc[75] = fma(pz5, v, acc[75]);
  }
  { const T v = Mc[1];
    acc[1] = fma(T(1), v, acc[1]);
    acc[4] = fma(px1, v, acc[4]);
    acc[6] = fma(py1, v, acc[6]);
    acc[7] = fma(pz1, v, acc[7]);
    acc[10] = fma(px2, v, acc[10]);
    acc[12] = fma(m_1_1_0, v, acc[12]);
    acc[13] = fma(m_1_0_1, v, acc[13]);
    acc[15] = fma(py2, v, acc[15]);
    acc[16] = fma(m_0_1_1, v, acc[16]);
    acc[17] = fma(pz2, v, acc[17]);
    acc[20] = fma(px3, v, acc[20]);
    acc[22] = fma(m_2_1_0, v, acc[22]);
    acc[23] = fma(m_2_0_1, v, acc[23]);
    acc[25] = fma(m_1_2_0, v, acc[25]);
    acc[26] = fma(m_1_1_1, v, acc[26]);
    acc[27] = fma(m_1_0_2, v, acc[27]);
    acc[29] = fma(py3, v, acc[29]);
    acc[30] = fma(m_0_2_1, v, acc[30]);
    acc[31] = fma(m_0_1_2, v, acc[31]);
    acc[32] = fma(pz3, v, acc[32]);
    acc[35] = fma(px4, v, acc[35]);
    acc[37] = fma(m_3_1_0, v, acc[37]);
    acc[38] = fma(m_3_0_1, v, acc[38]);
    acc[40] = fma(m_2_2_0, v, acc[40]);
    acc[41] = fma(m_2_1_1, v, acc[41]);
    acc[42] = fma(m_2_0_2, v, acc[42]);
    acc[44] = fma(m_1_3_0, v, acc[44]);
    acc[45] = fma(m_1_2_1, v, acc[45]);
    acc[46] = fma(m_1_1_2, v, acc[46]);
    acc[47] = fma(m_1_0_3, v, acc[47]);
    acc[49] = fma(py4, v, acc[49]);
    acc[50] = fma(m_0_3_1, v, acc[50]);
    acc[51] = fma(m_0_2_2, v, acc[51]);
    acc[52] = fma(m_0_1_3, v, acc[52]);
    acc[53] = fma(pz4, v, acc[53]);
    acc[56] = fma(px5, v, acc[56]);
    acc[58] = fma(m_4_1_0, v, acc[58]);
    acc[59] = fma(m_4_0_1, v, acc[59]);
    acc[61] = fma(m_3_2_0, v, acc[61]);
    acc[62] = fma(m_3_1_1, v, acc[62]);
    acc[63] = fma(m_3_0_2, v, acc[63]);
    acc[65] = fma(m_2_3_0, v, acc[65]);
    acc[66] = fma(m_2_2_1, v, acc[66]);
    acc[67] = fma(m_2_1_2, v, acc[67]);
    acc[68] = fma(m_2_0_3, v, acc[68]);
    acc[70] = fma(m_1_4_0, v, acc[70]);
    acc[71] = fma(m_1_3_1, v, acc[71]);
    acc[72] = fma(m_1_2_2, v, acc[72]);
    acc[73] = fma(m_1_1_3, v, acc[73]);
    acc[74] = fma(m_1_0_4, v, acc[74]);
    acc[76] = fma(py5, v, acc[76]);
    acc[77] = fma(m_0_4_1, v, acc[77]);
    acc[78] = fma(m_0_3_2, v, acc[78]);
    acc[79] = fma(m_0_2_3, v, acc[79]);
    acc[80] = fma(m_0_1_4, v, acc[80]);
    acc[81] = fma(pz5, v, acc[81]);
  }
  { const T v = Mc[2];
    acc[2] = fma(T(1), v, acc[2]);
    acc[5] = fma(px1, v, acc[5]);
    acc[7] = fma(py1, v, acc[7]);
    acc[8] = fma(pz1, v, acc[8]);
    acc[11] = fma(px2, v, acc[11]);
    acc[13] = fma(m_1_1_0, v, acc[13]);
    acc[14] = fma(m_1_0_1, v, acc[14]);
    acc[16] = fma(py2, v, acc[16]);
    acc[17] = fma(m_0_1_1, v, acc[17]);
    acc[18] = fma(pz2, v, acc[18]);
    acc[21] = fma(px3, v, acc[21]);
    acc[23] = fma(m_2_1_0, v, acc[23]);
    acc[24] = fma(m_2_0_1, v, acc[24]);
    acc[26] = fma(m_1_2_0, v, acc[26]);
    acc[27] = fma(m_1_1_1, v, acc[27]);
    acc[28] = fma(m_1_0_2, v, acc[28]);
    acc[30] = fma(py3, v, acc[30]);
    acc[31] = fma(m_0_2_1, v, acc[31]);
    acc[32] = fma(m_0_1_2, v, acc[32]);
    acc[33] = fma(pz3, v, acc[33]);
    acc[36] = fma(px4, v, acc[36]);
    acc[38] = fma(m_3_1_0, v, acc[38]);
    acc[39] = fma(m_3_0_1, v, acc[39]);
    acc[41] = fma(m_2_2_0, v, acc[41]);
    acc[42] = fma(m_2_1_1, v, acc[42]);
    acc[43] = fma(m_2_0_2, v, acc[43]);
    acc[45] = fma(m_1_3_0, v, acc[45]);
    acc[46] = fma(m_1_2_1, v, acc[46]);
    acc[47] = fma(m_1_1_2, v, acc[47]);
    acc[48] = fma(m_1_0_3, v, acc[48]);
    acc[50] = fma(py4, v, acc[50]);
    acc[51] = fma(m_0_3_1, v, acc[51]);
    acc[52] = fma(m_0_2_2, v, acc[52]);
    acc[53] = fma(m_0_1_3, v, acc[53]);
    acc[54] = fma(pz4, v, acc[54]);
    acc[57] = fma(px5, v, acc[57]);
    acc[59] = fma(m_4_1_0, v, acc[59]);
    acc[60] = fma(m_4_0_1, v, acc[60]);
    acc[62] = fma(m_3_2_0, v, acc[62]);
    acc[63] = fma(m_3_1_1, v, acc[63]);
    acc[64] = fma(m_3_0_2, v, acc[64]);
    acc[66] = fma(m_2_3_0, v, acc[66]);
    acc[67] = fma(m_2_2_1, v, acc[67]);
    acc[68] = fma(m_2_1_2, v, acc[68]);
    acc[69] = fma(m_2_0_3, v, acc[69]);
    acc[71] = fma(m_1_4_0, v, acc[71]);
    acc[72] = fma(m_1_3_1, v, acc[72]);
    acc[73] = fma(m_1_2_2, v, acc[73]);
    acc[74] = fma(m_1_1_3, v, acc[74]);
    acc[75] = fma(m_1_0_4, v, acc[75]);
    acc[77] = fma(py5, v, acc[77]);
    acc[78] = fma(m_0_4_1, v, acc[78]);
    acc[79] = fma(m_0_3_2, v, acc[79]);
    acc[80] = fma(m_0_2_3, v, acc[80]);
    acc[81] = fma(m_0_1_4, v, acc[81]);
    acc[82] = fma(pz5, v, acc[82]);
  }
  { const T v = Mc[3];
    acc[3] = fma(T(1), v, acc[3]);
    acc[9] = fma(px1, v, acc[9]);
    acc[10] = fma(py1, v, acc[10]);
    acc[11] = fma(pz1, v, acc[11]);
    acc[19] = fma(px2, v, acc[19]);
    acc[20] = fma(m_1_1_0, v, acc[20]);
    acc[21] = fma(m_1_0_1, v, acc[21]);
    acc[22] = fma(py2, v, acc[22]);
    acc[23] = fma(m_0_1_1, v, acc[23]);
    acc[24] = fma(pz2, v, acc[24]);
    acc[34] = fma(px3, v, acc[34]);
    acc[35] = fma(m_2_1_0, v, acc[35]);
    acc[36] = fma(m_2_0_1, v, acc[36]);
    acc[37] = fma(m_1_2_0, v, acc[37]);
    acc[38] = fma(m_1_1_1, v, acc[38]);
    acc[39] = fma(m_1_0_2, v, acc[39]);
    acc[40] = fma(py3, v, acc[40]);
    acc[41] = fma(m_0_2_1, v, acc[41]);
    acc[42] = fma(m_0_1_2, v, acc[42]);
    acc[43] = fma(pz3, v, acc[43]);
    acc[55] = fma(px4, v, acc[55]);
    acc[56] = fma(m_3_1_0, v, acc[56]);
    acc[57] = fma(m_3_0_1, v, acc[57]);
    acc[58] = fma(m_2_2_0, v, acc[58]);
    acc[59] = fma(m_2_1_1, v, acc[59]);
    acc[60] = fma(m_2_0_2, v, acc[60]);
    acc[61] = fma(m_1_3_0, v, acc[61]);
    acc[62] = fma(m_1_2_1, v, acc[62]);
    acc[63] = fma(m_1_1_2, v, acc[63]);
    acc[64] = fma(m_1_0_3, v, acc[64]);
    acc[65] = fma(py4, v, acc[65]);
    acc[66] = fma(m_0_3_1, v, acc[66]);
    acc[67] = fma(m_0_2_2, v, acc[67]);
    acc[68] = fma(m_0_1_3, v, acc[68]);
    acc[69] = fma(pz4, v, acc[69]);
  }
  { const T v = Mc[4];
    acc[4] = fma(T(1), v, acc[4]);
    acc[10] = fma(px1, v, acc[10]);
    acc[12] = fma(py1, v, acc[12]);
    acc[13] = fma(pz1, v, acc[13]);
    acc[20] = fma(px2, v, acc[20]);
    acc[22] = fma(m_1_1_0, v, acc[22]);
    acc[23] = fma(m_1_0_1, v, acc[23]);
    acc[25] = fma(py2, v, acc[25]);
    acc[26] = fma(m_0_1_1, v, acc[26]);
    acc[27] = fma(pz2, v, acc[27]);
    acc[35] = fma(px3, v, acc[35]);
    acc[37] = fma(m_2_1_0, v, acc[37]);
    acc[38] = fma(m_2_0_1, v, acc[38]);
    acc[40] = fma(m_1_2_0, v, acc[40]);
    acc[41] = fma(m_1_1_1, v, acc[41]);
    acc[42] = fma(m_1_0_2, v, acc[42]);
    acc[44] = fma(py3, v, acc[44]);
    acc[45] = fma(m_0_2_1, v, acc[45]);
    acc[46] = fma(m_0_1_2, v, acc[46]);
    acc[47] = fma(pz3, v, acc[47]);
    acc[56] = fma(px4, v, acc[56]);
    acc[58] = fma(m_3_1_0, v, acc[58]);
    acc[59] = fma(m_3_0_1, v, acc[59]);
    acc[61] = fma(m_2_2_0, v, acc[61]);
    acc[62] = fma(m_2_1_1, v, acc[62]);
    acc[63] = fma(m_2_0_2, v, acc[63]);
    acc[65] = fma(m_1_3_0, v, acc[65]);
    acc[66] = fma(m_1_2_1, v, acc[66]);
    acc[67] = fma(m_1_1_2, v, acc[67]);
    acc[68] = fma(m_1_0_3, v, acc[68]);
    acc[70] = fma(py4, v, acc[70]);
    acc[71] = fma(m_0_3_1, v, acc[71]);
    acc[72] = fma(m_0_2_2, v, acc[72]);
    acc[73] = fma(m_0_1_3, v, acc[73]);
    acc[74] = fma(pz4, v, acc[74]);
  }
  { const T v = Mc[5];
    acc[5] = fma(T(1), v, acc[5]);
    acc[11] = fma(px1, v, acc[11]);
    acc[13] = fma(py1, v, acc[13]);
    acc[14] = fma(pz1, v, acc[14]);
    acc[21] = fma(px2, v, acc[21]);
    acc[23] = fma(m_1_1_0, v, acc[23]);
    acc[24] = fma(m_1_0_1, v, acc[24]);
    acc[26] = fma(py2, v, acc[26]);
    acc[27] = fma(m_0_1_1, v, acc[27]);
    acc[28] = fma(pz2, v, acc[28]);
    acc[36] = fma(px3, v, acc[36]);
    acc[38] = fma(m_2_1_0, v, acc[38]);
    acc[39] = fma(m_2_0_1, v, acc[39]);
    acc[41] = fma(m_1_2_0, v, acc[41]);
    acc[42] = fma(m_1_1_1, v, acc[42]);
    acc[43] = fma(m_1_0_2, v, acc[43]);
    acc[45] = fma(py3, v, acc[45]);
    acc[46] = fma(m_0_2_1, v, acc[46]);
    acc[47] = fma(m_0_1_2, v, acc[47]);
    acc[48] = fma(pz3, v, acc[48]);
    acc[57] = fma(px4, v, acc[57]);
    acc[59] = fma(m_3_1_0, v, acc[59]);
    acc[60] = fma(m_3_0_1, v, acc[60]);
    acc[62] = fma(m_2_2_0, v, acc[62]);
    acc[63] = fma(m_2_1_1, v, acc[63]);
    acc[64] = fma(m_2_0_2, v, acc[64]);
    acc[66] = fma(m_1_3_0, v, acc[66]);
    acc[67] = fma(m_1_2_1, v, acc[67]);
    acc[68] = fma(m_1_1_2, v, acc[68]);
    acc[69] = fma(m_1_0_3, v, acc[69]);
    acc[71] = fma(py4, v, acc[71]);
    acc[72] = fma(m_0_3_1, v, acc[72]);
    acc[73] = fma(m_0_2_2, v, acc[73]);
    acc[74] = fma(m_0_1_3, v, acc[74]);
    acc[75] = fma(pz4, v, acc[75]);
  }
  { const T v = Mc[6];
    acc[6] = fma(T(1), v, acc[6]);
    acc[12] = fma(px1, v, acc[12]);
    acc[15] = fma(py1, v, acc[15]);
    acc[16] = fma(pz1, v, acc[16]);
    acc[22] = fma(px2, v, acc[22]);
    acc[25] = fma(m_1_1_0, v, acc[25]);
    acc[26] = fma(m_1_0_1, v, acc[26]);
    acc[29] = fma(py2, v, acc[29]);
    acc[30] = fma(m_0_1_1, v, acc[30]);
    acc[31] = fma(pz2, v, acc[31]);
    acc[37] = fma(px3, v, acc[37]);
    acc[40] = fma(m_2_1_0, v, acc[40]);
    acc[41] = fma(m_2_0_1, v, acc[41]);
    acc[44] = fma(m_1_2_0, v, acc[44]);
    acc[45] = fma(m_1_1_1, v, acc[45]);
    acc[46] = fma(m_1_0_2, v, acc[46]);
    acc[49] = fma(py3, v, acc[49]);
    acc[50] = fma(m_0_2_1, v, acc[50]);
    acc[51] = fma(m_0_1_2, v, acc[51]);
    acc[52] = fma(pz3, v, acc[52]);
    acc[58] = fma(px4, v, acc[58]);
    acc[61] = fma(m_3_1_0, v, acc[61]);
    acc[62] = fma(m_3_0_1, v, acc[62]);
    acc[65] = fma(m_2_2_0, v, acc[65]);
    acc[66] = fma(m_2_1_1, v, acc[66]);
    acc[67] = fma(m_2_0_2, v, acc[67]);
    acc[70] = fma(m_1_3_0, v, acc[70]);
    acc[71] = fma(m_1_2_1, v, acc[71]);
    acc[72] = fma(m_1_1_2, v, acc[72]);
    acc[73] = fma(m_1_0_3, v, acc[73]);
    acc[76] = fma(py4, v, acc[76]);
    acc[77] = fma(m_0_3_1, v, acc[77]);
    acc[78] = fma(m_0_2_2, v, acc[78]);
    acc[79] = fma(m_0_1_3, v, acc[79]);
    acc[80] = fma(pz4, v, acc[80]);
  }
  { const T v = Mc[7];
    acc[7] = fma(T(1), v, acc[7]);
    acc[13] = fma(px1, v, acc[13]);
    acc[16] = fma(py1, v, acc[16]);
    acc[17] = fma(pz1, v, acc[17]);
    acc[23] = fma(px2, v, acc[23]);
    acc[26] = fma(m_1_1_0, v, acc[26]);
    acc[27] = fma(m_1_0_1, v, acc[27]);
    acc[30] = fma(py2, v, acc[30]);
    acc[31] = fma(m_0_1_1, v, acc[31]);
    acc[32] = fma(pz2, v, acc[32]);
    acc[38] = fma(px3, v, acc[38]);
    acc[41] = fma(m_2_1_0, v, acc[41]);
    acc[42] = fma(m_2_0_1, v, acc[42]);
    acc[45] = fma(m_1_2_0, v, acc[45]);
    acc[46] = fma(m_1_1_1, v, acc[46]);
    acc[47] = fma(m_1_0_2, v, acc[47]);
    acc[50] = fma(py3, v, acc[50]);
    acc[51] = fma(m_0_2_1, v, acc[51]);
    acc[52] = fma(m_0_1_2, v, acc[52]);
    acc[53] = fma(pz3, v, acc[53]);
    acc[59] = fma(px4, v, acc[59]);
    acc[62] = fma(m_3_1_0, v, acc[62]);
    acc[63] = fma(m_3_0_1, v, acc[63]);
    acc[66] = fma(m_2_2_0, v, acc[66]);
    acc[67] = fma(m_2_1_1, v, acc[67]);
    acc[68] = fma(m_2_0_2, v, acc[68]);
    acc[71] = fma(m_1_3_0, v, acc[71]);
    acc[72] = fma(m_1_2_1, v, acc[72]);
    acc[73] = fma(m_1_1_2, v, acc[73]);
    acc[74] = fma(m_1_0_3, v, acc[74]);
    acc[77] = fma(py4, v, acc[77]);
    acc[78] = fma(m_0_3_1, v, acc[78]);
    acc[79] = fma(m_0_2_2, v, acc[79]);
    acc[80] = fma(m_0_1_3, v, acc[80]);
    acc[81] = fma(pz4, v, acc[81]);
  }
  { const T v = Mc[8];
    acc[8] = fma(T(1), v, acc[8]);
    acc[14] = fma(px1, v, acc[14]);
    acc[17] = fma(py1, v, acc[17]);
    acc[18] = fma(pz1, v, acc[18]);
    acc[24] = fma(px2, v, acc[24]);
    acc[27] = fma(m_1_1_0, v, acc[27]);
    acc[28] = fma(m_1_0_1, v, acc[28]);
    acc[31] = fma(py2, v, acc[31]);
    acc[32] = fma(m_0_1_1, v, acc[32]);
    acc[33] = fma(pz2, v, acc[33]);
    acc[39] = fma(px3, v, acc[39]);
    acc[42] = fma(m_2_1_0, v, acc[42]);
    acc[43] = fma(m_2_0_1, v, acc[43]);
    acc[46] = fma(m_1_2_0, v, acc[46]);
    acc[47] = fma(m_1_1_1, v, acc[47]);
    acc[48] = fma(m_1_0_2, v, acc[48]);
    acc[51] = fma(py3, v, acc[51]);
    acc[52] = fma(m_0_2_1, v, acc[52]);
    acc[53] = fma(m_0_1_2, v, acc[53]);
    acc[54] = fma(pz3, v, acc[54]);
    acc[60] = fma(px4, v, acc[60]);
    acc[63] = fma(m_3_1_0, v, acc[63]);
    acc[64] = fma(m_3_0_1, v, acc[64]);
    acc[67] = fma(m_2_2_0, v, acc[67]);
    acc[68] = fma(m_2_1_1, v, acc[68]);
    acc[69] = fma(m_2_0_2, v, acc[69]);
    acc[72] = fma(m_1_3_0, v, acc[72]);
    acc[73] = fma(m_1_2_1, v, acc[73]);
    acc[74] = fma(m_1_1_2, v, acc[74]);
    acc[75] = fma(m_1_0_3, v, acc[75]);
    acc[78] = fma(py4, v, acc[78]);
    acc[79] = fma(m_0_3_1, v, acc[79]);
    acc[80] = fma(m_0_2_2, v, acc[80]);
    acc[81] = fma(m_0_1_3, v, acc[81]);
    acc[82] = fma(pz4, v, acc[82]);
  }
  { const T v = Mc[9];
    acc[9] = fma(T(1), v, acc[9]);
    acc[19] = fma(px1, v, acc[19]);
    acc[20] = fma(py1, v, acc[20]);
    acc[21] = fma(pz1, v, acc[21]);
    acc[34] = fma(px2, v, acc[34]);
    acc[35] = fma(m_1_1_0, v, acc[35]);
    acc[36] = fma(m_1_0_1, v, acc[36]);
    acc[37] = fma(py2, v, acc[37]);
    acc[38] = fma(m_0_1_1, v, acc[38]);
    acc[39] = fma(pz2, v, acc[39]);
    acc[55] = fma(px3, v, acc[55]);
    acc[56] = fma(m_2_1_0, v, acc[56]);
    acc[57] = fma(m_2_0_1, v, acc[57]);
    acc[58] = fma(m_1_2_0, v, acc[58]);
    acc[59] = fma(m_1_1_1, v, acc[59]);
    acc[60] = fma(m_1_0_2, v, acc[60]);
    acc[61] = fma(py3, v, acc[61]);
    acc[62] = fma(m_0_2_1, v, acc[62]);
    acc[63] = fma(m_0_1_2, v, acc[63]);
    acc[64] = fma(pz3, v, acc[64]);
  }
  { const T v = Mc[10];
    acc[10] = fma(T(1), v, acc[10]);
    acc[20] = fma(px1, v, acc[20]);
    acc[22] = fma(py1, v, acc[22]);
    acc[23] = fma(pz1, v, acc[23]);
    acc[35] = fma(px2, v, acc[35]);
    acc[37] = fma(m_1_1_0, v, acc[37]);
    acc[38] = fma(m_1_0_1, v, acc[38]);
    acc[40] = fma(py2, v, acc[40]);
    acc[41] = fma(m_0_1_1, v, acc[41]);
    acc[42] = fma(pz2, v, acc[42]);
    acc[56] = fma(px3, v, acc[56]);
    acc[58] = fma(m_2_1_0, v, acc[58]);
    acc[59] = fma(m_2_0_1, v, acc[59]);
    acc[61] = fma(m_1_2_0, v, acc[61]);
    acc[62] = fma(m_1_1_1, v, acc[62]);
    acc[63] = fma(m_1_0_2, v, acc[63]);
    acc[65] = fma(py3, v, acc[65]);
    acc[66] = fma(m_0_2_1, v, acc[66]);
    acc[67] = fma(m_0_1_2, v, acc[67]);
    acc[68] = fma(pz3, v, acc[68]);
  }
  { const T v = Mc[11];
    acc[11] = fma(T(1), v, acc[11]);
    acc[21] = fma(px1, v, acc[21]);
    acc[23] = fma(py1, v, acc[23]);
    acc[24] = fma(pz1, v, acc[24]);
    acc[36] = fma(px2, v, acc[36]);
    acc[38] = fma(m_1_1_0, v, acc[38]);
    acc[39] = fma(m_1_0_1, v, acc[39]);
    acc[41] = fma(py2, v, acc[41]);
    acc[42] = fma(m_0_1_1, v, acc[42]);
    acc[43] = fma(pz2, v, acc[43]);
    acc[57] = fma(px3, v, acc[57]);
    acc[59] = fma(m_2_1_0, v, acc[59]);
    acc[60] = fma(m_2_0_1, v, acc[60]);
    acc[62] = fma(m_1_2_0, v, acc[62]);
    acc[63] = fma(m_1_1_1, v, acc[63]);
    acc[64] = fma(m_1_0_2, v, acc[64]);
    acc[66] = fma(py3, v, acc[66]);
    acc[67] = fma(m_0_2_1, v, acc[67]);
    acc[68] = fma(m_0_1_2, v, acc[68]);
    acc[69] = fma(pz3, v, acc[69]);
  }
  { const T v = Mc[12];
    acc[12] = fma(T(1), v, acc[12]);
    acc[22] = fma(px1, v, acc[22]);
    acc[25] = fma(py1, v, acc[25]);
    acc[26] = fma(pz1, v, acc[26]);
    acc[37] = fma(px2, v, acc[37]);
    acc[40] = fma(m_1_1_0, v, acc[40]);
    acc[41] = fma(m_1_0_1, v, acc[41]);
    acc[44] = fma(py2, v, acc[44]);
    acc[45] = fma(m_0_1_1, v, acc[45]);
    acc[46] = fma(pz2, v, acc[46]);
    acc[58] = fma(px3, v, acc[58]);
    acc[61] = fma(m_2_1_0, v, acc[61]);
    acc[62] = fma(m_2_0_1, v, acc[62]);
    acc[65] = fma(m_1_2_0, v, acc[65]);
    acc[66] = fma(m_1_1_1, v, acc[66]);
    acc[67] = fma(m_1_0_2, v, acc[67]);
    acc[70] = fma(py3, v, acc[70]);
    acc[71] = fma(m_0_2_1, v, acc[71]);
    acc[72] = fma(m_0_1_2, v, acc[72]);
    acc[73] = fma(pz3, v, acc[73]);
  }
  { const T v = Mc[13];
    acc[13] = fma(T(1), v, acc[13]);
    acc[23] = fma(px1, v, acc[23]);
    acc[26] = fma(py1, v, acc[26]);
    acc[27] = fma(pz1, v, acc[27]);
    acc[38] = fma(px2, v, acc[38]);
    acc[41] = fma(m_1_1_0, v, acc[41]);
    acc[42] = fma(m_1_0_1, v, acc[42]);
    acc[45] = fma(py2, v, acc[45]);
    acc[46] = fma(m_0_1_1, v, acc[46]);
    acc[47] = fma(pz2, v, acc[47]);
    acc[59] = fma(px3, v, acc[59]);
    acc[62] = fma(m_2_1_0, v, acc[62]);
    acc[63] = fma(m_2_0_1, v, acc[63]);
    acc[66] = fma(m_1_2_0, v, acc[66]);
    acc[67] = fma(m_1_1_1, v, acc[67]);
    acc[68] = fma(m_1_0_2, v, acc[68]);
    acc[71] = fma(py3, v, acc[71]);
    acc[72] = fma(m_0_2_1, v, acc[72]);
    acc[73] = fma(m_0_1_2, v, acc[73]);
    acc[74] = fma(pz3, v, acc[74]);
  }
  { const T v = Mc[14];
    acc[14] = fma(T(1), v, acc[14]);
    acc[24] = fma(px1, v, acc[24]);
    acc[27] = fma(py1, v, acc[27]);
    acc[28] = fma(pz1, v, acc[28]);
    acc[39] = fma(px2, v, acc[39]);
    acc[42] = fma(m_1_1_0, v, acc[42]);
    acc[43] = fma(m_1_0_1, v, acc[43]);
    acc[46] = fma(py2, v, acc[46]);
    acc[47] = fma(m_0_1_1, v, acc[47]);
    acc[48] = fma(pz2, v, acc[48]);
    acc[60] = fma(px3, v, acc[60]);
    acc[63] = fma(m_2_1_0, v, acc[63]);
    acc[64] = fma(m_2_0_1, v, acc[64]);
    acc[67] = fma(m_1_2_0, v, acc[67]);
    acc[68] = fma(m_1_1_1, v, acc[68]);
    acc[69] = fma(m_1_0_2, v, acc[69]);
    acc[72] = fma(py3, v, acc[72]);
    acc[73] = fma(m_0_2_1, v, acc[73]);
    acc[74] = fma(m_0_1_2, v, acc[74]);
    acc[75] = fma(pz3, v, acc[75]);
  }
  { const T v = Mc[15];
    acc[15] = fma(T(1), v, acc[15]);
    acc[25] = fma(px1, v, acc[25]);
    acc[29] = fma(py1, v, acc[29]);
    acc[30] = fma(pz1, v, acc[30]);
    acc[40] = fma(px2, v, acc[40]);
    acc[44] = fma(m_1_1_0, v, acc[44]);
    acc[45] = fma(m_1_0_1, v, acc[45]);
    acc[49] = fma(py2, v, acc[49]);
    acc[50] = fma(m_0_1_1, v, acc[50]);
    acc[51] = fma(pz2, v, acc[51]);
    acc[61] = fma(px3, v, acc[61]);
    acc[65] = fma(m_2_1_0, v, acc[65]);
    acc[66] = fma(m_2_0_1, v, acc[66]);
    acc[70] = fma(m_1_2_0, v, acc[70]);
    acc[71] = fma(m_1_1_1, v, acc[71]);
    acc[72] = fma(m_1_0_2, v, acc[72]);
    acc[76] = fma(py3, v, acc[76]);
    acc[77] = fma(m_0_2_1, v, acc[77]);
    acc[78] = fma(m_0_1_2, v, acc[78]);
    acc[79] = fma(pz3, v, acc[79]);
  }
  { const T v = Mc[16];
    acc[16] = fma(T(1), v, acc[16]);
    acc[26] = fma(px1, v, acc[26]);
    acc[30] = fma(py1, v, acc[30]);
    acc[31] = fma(pz1, v, acc[31]);
    acc[41] = fma(px2, v, acc[41]);
    acc[45] = fma(m_1_1_0, v, acc[45]);
    acc[46] = fma(m_1_0_1, v, acc[46]);
    acc[50] = fma(py2, v, acc[50]);
    acc[51] = fma(m_0_1_1, v, acc[51]);
    acc[52] = fma(pz2, v, acc[52]);
    acc[62] = fma(px3, v, acc[62]);
    acc[66] = fma(m_2_1_0, v, acc[66]);
    acc[67] = fma(m_2_0_1, v, acc[67]);
    acc[71] = fma(m_1_2_0, v, acc[71]);
    acc[72] = fma(m_1_1_1, v, acc[72]);
    acc[73] = fma(m_1_0_2, v, acc[73]);
    acc[77] = fma(py3, v, acc[77]);
    acc[78] = fma(m_0_2_1, v, acc[78]);
    acc[79] = fma(m_0_1_2, v, acc[79]);
    acc[80] = fma(pz3, v, acc[80]);
  }
  { const T v = Mc[17];
    acc[17] = fma(T(1), v, acc[17]);
    acc[27] = fma(px1, v, acc[27]);
    acc[31] = fma(py1, v, acc[31]);
    acc[32] = fma(pz1, v, acc[32]);
    acc[42] = fma(px2, v, acc[42]);
    acc[46] = fma(m_1_1_0, v, acc[46]);
    acc[47] = fma(m_1_0_1, v, acc[47]);
    acc[51] = fma(py2, v, acc[51]);
    acc[52] = fma(m_0_1_1, v, acc[52]);
    acc[53] = fma(pz2, v, acc[53]);
    acc[63] = fma(px3, v, acc[63]);
    acc[67] = fma(m_2_1_0, v, acc[67]);
    acc[68] = fma(m_2_0_1, v, acc[68]);
    acc[72] = fma(m_1_2_0, v, acc[72]);
    acc[73] = fma(m_1_1_1, v, acc[73]);
    acc[74] = fma(m_1_0_2, v, acc[74]);
    acc[78] = fma(py3, v, acc[78]);
    acc[79] = fma(m_0_2_1, v, acc[79]);
    acc[80] = fma(m_0_1_2, v, acc[80]);
    acc[81] = fma(pz3, v, acc[81]);
  }
  { const T v = Mc[18];
    acc[18] = fma(T(1), v, acc[18]);
    acc[28] = fma(px1, v, acc[28]);
    acc[32] = fma(py1, v, acc[32]);
    acc[33] = fma(pz1, v, acc[33]);
    acc[43] = fma(px2, v, acc[43]);
    acc[47] = fma(m_1_1_0, v, acc[47]);
    acc[48] = fma(m_1_0_1, v, acc[48]);
    acc[52] = fma(py2, v, acc[52]);
    acc[53] = fma(m_0_1_1, v, acc[53]);
    acc[54] = fma(pz2, v, acc[54]);
    acc[64] = fma(px3, v, acc[64]);
    acc[68] = fma(m_2_1_0, v, acc[68]);
    acc[69] = fma(m_2_0_1, v, acc[69]);
    acc[73] = fma(m_1_2_0, v, acc[73]);
    acc[74] = fma(m_1_1_1, v, acc[74]);
    acc[75] = fma(m_1_0_2, v, acc[75]);
    acc[79] = fma(py3, v, acc[79]);
    acc[80] = fma(m_0_2_1, v, acc[80]);
    acc[81] = fma(m_0_1_2, v, acc[81]);
    acc[82] = fma(pz3, v, acc[82]);
  }
  { const T v = Mc[19];
    acc[19] = fma(T(1), v, acc[19]);
    acc[34] = fma(px1, v, acc[34]);
    acc[35] = fma(py1, v, acc[35]);
    acc[36] = fma(pz1, v, acc[36]);
    acc[55] = fma(px2, v, acc[55]);
    acc[56] = fma(m_1_1_0, v, acc[56]);
    acc[57] = fma(m_1_0_1, v, acc[57]);
    acc[58] = fma(py2, v, acc[58]);
    acc[59] = fma(m_0_1_1, v, acc[59]);
    acc[60] = fma(pz2, v, acc[60]);
  }
  { const T v = Mc[20];
    acc[20] = fma(T(1), v, acc[20]);
    acc[35] = fma(px1, v, acc[35]);
    acc[37] = fma(py1, v, acc[37]);
    acc[38] = fma(pz1, v, acc[38]);
    acc[56] = fma(px2, v, acc[56]);
    acc[58] = fma(m_1_1_0, v, acc[58]);
    acc[59] = fma(m_1_0_1, v, acc[59]);
    acc[61] = fma(py2, v, acc[61]);
    acc[62] = fma(m_0_1_1, v, acc[62]);
    acc[63] = fma(pz2, v, acc[63]);
  }
  { const T v = Mc[21];
    acc[21] = fma(T(1), v, acc[21]);
    acc[36] = fma(px1, v, acc[36]);
    acc[38] = fma(py1, v, acc[38]);
    acc[39] = fma(pz1, v, acc[39]);
    acc[57] = fma(px2, v, acc[57]);
    acc[59] = fma(m_1_1_0, v, acc[59]);
    acc[60] = fma(m_1_0_1, v, acc[60]);
    acc[62] = fma(py2, v, acc[62]);
    acc[63] = fma(m_0_1_1, v, acc[63]);
    acc[64] = fma(pz2, v, acc[64]);
  }
  { const T v = Mc[22];
    acc[22] = fma(T(1), v, acc[22]);
    acc[37] = fma(px1, v, acc[37]);
    acc[40] = fma(py1, v, acc[40]);
    acc[41] = fma(pz1, v, acc[41]);
    acc[58] = fma(px2, v, acc[58]);
    acc[61] = fma(m_1_1_0, v, acc[61]);
    acc[62] = fma(m_1_0_1, v, acc[62]);
    acc[65] = fma(py2, v, acc[65]);
    acc[66] = fma(m_0_1_1, v, acc[66]);
    acc[67] = fma(pz2, v, acc[67]);
  }
  { const T v = Mc[23];
    acc[23] = fma(T(1), v, acc[23]);
    acc[38] = fma(px1, v, acc[38]);
    acc[41] = fma(py1, v, acc[41]);
    acc[42] = fma(pz1, v, acc[42]);
    acc[59] = fma(px2, v, acc[59]);
    acc[62] = fma(m_1_1_0, v, acc[62]);
    acc[63] = fma(m_1_0_1, v, acc[63]);
    acc[66] = fma(py2, v, acc[66]);
    acc[67] = fma(m_0_1_1, v, acc[67]);
    acc[68] = fma(pz2, v, acc[68]);
  }
  { const T v = Mc[24];
    acc[24] = fma(T(1), v, acc[24]);
    acc[39] = fma(px1, v, acc[39]);
    acc[42] = fma(py1, v, acc[42]);
    acc[43] = fma(pz1, v, acc[43]);
    acc[60] = fma(px2, v, acc[60]);
    acc[63] = fma(m_1_1_0, v, acc[63]);
    acc[64] = fma(m_1_0_1, v, acc[64]);
    acc[67] = fma(py2, v, acc[67]);
    acc[68] = fma(m_0_1_1, v, acc[68]);
    acc[69] = fma(pz2, v, acc[69]);
  }
  { const T v = Mc[25];
    acc[25] = fma(T(1), v, acc[25]);
    acc[40] = fma(px1, v, acc[40]);
    acc[44] = fma(py1, v, acc[44]);
    acc[45] = fma(pz1, v, acc[45]);
    acc[61] = fma(px2, v, acc[61]);
    acc[65] = fma(m_1_1_0, v, acc[65]);
    acc[66] = fma(m_1_0_1, v, acc[66]);
    acc[70] = fma(py2, v, acc[70]);
    acc[71] = fma(m_0_1_1, v, acc[71]);
    acc[72] = fma(pz2, v, acc[72]);
  }
  { const T v = Mc[26];
    acc[26] = fma(T(1), v, acc[26]);
    acc[41] = fma(px1, v, acc[41]);
    acc[45] = fma(py1, v, acc[45]);
    acc[46] = fma(pz1, v, acc[46]);
    acc[62] = fma(px2, v, acc[62]);
    acc[66] = fma(m_1_1_0, v, acc[66]);
    acc[67] = fma(m_1_0_1, v, acc[67]);
    acc[71] = fma(py2, v, acc[71]);
    acc[72] = fma(m_0_1_1, v, acc[72]);
    acc[73] = fma(pz2, v, acc[73]);
  }
  { const T v = Mc[27];
    acc[27] = fma(T(1), v, acc[27]);
    acc[42] = fma(px1, v, acc[42]);
    acc[46] = fma(py1, v, acc[46]);
    acc[47] = fma(pz1, v, acc[47]);
    acc[63] = fma(px2, v, acc[63]);
    acc[67] = fma(m_1_1_0, v, acc[67]);
    acc[68] = fma(m_1_0_1, v, acc[68]);
    acc[72] = fma(py2, v, acc[72]);
    acc[73] = fma(m_0_1_1, v, acc[73]);
    acc[74] = fma(pz2, v, acc[74]);
  }
  { const T v = Mc[28];
    acc[28] = fma(T(1), v, acc[28]);
    acc[43] = fma(px1, v, acc[43]);
    acc[47] = fma(py1, v, acc[47]);
    acc[48] = fma(pz1, v, acc[48]);
    acc[64] = fma(px2, v, acc[64]);
    acc[68] = fma(m_1_1_0, v, acc[68]);
    acc[69] = fma(m_1_0_1, v, acc[69]);
    acc[73] = fma(py2, v, acc[73]);
    acc[74] = fma(m_0_1_1, v, acc[74]);
    acc[75] = fma(pz2, v, acc[75]);
  }
  { const T v = Mc[29];
    acc[29] = fma(T(1), v, acc[29]);
    acc[44] = fma(px1, v, acc[44]);
    acc[49] = fma(py1, v, acc[49]);
    acc[50] = fma(pz1, v, acc[50]);
    acc[65] = fma(px2, v, acc[65]);
    acc[70] = fma(m_1_1_0, v, acc[70]);
    acc[71] = fma(m_1_0_1, v, acc[71]);
    acc[76] = fma(py2, v, acc[76]);
    acc[77] = fma(m_0_1_1, v, acc[77]);
    acc[78] = fma(pz2, v, acc[78]);
  }
  { const T v = Mc[30];
    acc[30] = fma(T(1), v, acc[30]);
    acc[45] = fma(px1, v, acc[45]);
    acc[50] = fma(py1, v, acc[50]);
    acc[51] = fma(pz1, v, acc[51]);
    acc[66] = fma(px2, v, acc[66]);
    acc[71] = fma(m_1_1_0, v, acc[71]);
    acc[72] = fma(m_1_0_1, v, acc[72]);
    acc[77] = fma(py2, v, acc[77]);
    acc[78] = fma(m_0_1_1, v, acc[78]);
    acc[79] = fma(pz2, v, acc[79]);
  }
  { const T v = Mc[31];
    acc[31] = fma(T(1), v, acc[31]);
    acc[46] = fma(px1, v, acc[46]);
    acc[51] = fma(py1, v, acc[51]);
    acc[52] = fma(pz1, v, acc[52]);
    acc[67] = fma(px2, v, acc[67]);
    acc[72] = fma(m_1_1_0, v, acc[72]);
    acc[73] = fma(m_1_0_1, v, acc[73]);
    acc[78] = fma(py2, v, acc[78]);
    acc[79] = fma(m_0_1_1, v, acc[79]);
    acc[80] = fma(pz2, v, acc[80]);
  }
  { const T v = Mc[32];
    acc[32] = fma(T(1), v, acc[32]);
    acc[47] = fma(px1, v, acc[47]);
    acc[52] = fma(py1, v, acc[52]);
    acc[53] = fma(pz1, v, acc[53]);
    acc[68] = fma(px2, v, acc[68]);
    acc[73] = fma(m_1_1_0, v, acc[73]);
    acc[74] = fma(m_1_0_1, v, acc[74]);
    acc[79] = fma(py2, v, acc[79]);
    acc[80] = fma(m_0_1_1, v, acc[80]);
    acc[81] = fma(pz2, v, acc[81]);
  }
  { const T v = Mc[33];
    acc[33] = fma(T(1), v, acc[33]);
    acc[48] = fma(px1, v, acc[48]);
    acc[53] = fma(py1, v, acc[53]);
    acc[54] = fma(pz1, v, acc[54]);
    acc[69] = fma(px2, v, acc[69]);
    acc[74] = fma(m_1_1_0, v, acc[74]);
    acc[75] = fma(m_1_0_1, v, acc[75]);
    acc[80] = fma(py2, v, acc[80]);
    acc[81] = fma(m_0_1_1, v, acc[81]);
    acc[82] = fma(pz2, v, acc[82]);
  }
  { const T v = Mc[34];
    acc[34] = fma(T(1), v, acc[34]);
    acc[55] = fma(px1, v, acc[55]);
    acc[56] = fma(py1, v, acc[56]);
    acc[57] = fma(pz1, v, acc[57]);
  }
  { const T v = Mc[35];
    acc[35] = fma(T(1), v, acc[35]);
    acc[56] = fma(px1, v, acc[56]);
    acc[58] = fma(py1, v, acc[58]);
    acc[59] = fma(pz1, v, acc[59]);
  }
  { const T v = Mc[36];
    acc[36] = fma(T(1), v, acc[36]);
    acc[57] = fma(px1, v, acc[57]);
    acc[59] = fma(py1, v, acc[59]);
    acc[60] = fma(pz1, v, acc[60]);
  }
  { const T v = Mc[37];
    acc[37] = fma(T(1), v, acc[37]);
    acc[58] = fma(px1, v, acc[58]);
    acc[61] = fma(py1, v, acc[61]);
    acc[62] = fma(pz1, v, acc[62]);
  }
  { const T v = Mc[38];
    acc[38] = fma(T(1), v, acc[38]);
    acc[59] = fma(px1, v, acc[59]);
    acc[62] = fma(py1, v, acc[62]);
    acc[63] = fma(pz1, v, acc[63]);
  }
  { const T v = Mc[39];
    acc[39] = fma(T(1), v, acc[39]);
    acc[60] = fma(px1, v, acc[60]);
    acc[63] = fma(py1, v, acc[63]);
    acc[64] = fma(pz1, v, acc[64]);
  }
  { const T v = Mc[40];
    acc[40] = fma(T(1), v, acc[40]);
    acc[61] = fma(px1, v, acc[61]);
    acc[65] = fma(py1, v, acc[65]);
    acc[66] = fma(pz1, v, acc[66]);
  }
  { const T v = Mc[41];
    acc[41] = fma(T(1), v, acc[41]);
    acc[62] = fma(px1, v, acc[62]);
    acc[66] = fma(py1, v, acc[66]);
    acc[67] = fma(pz1, v, acc[67]);
  }
  { const T v = Mc[42];
    acc[42] = fma(T(1), v, acc[42]);
    acc[63] = fma(px1, v, acc[63]);
    acc[67] = fma(py1, v, acc[67]);
    acc[68] = fma(pz1, v, acc[68]);
  }
  { const T v = Mc[43];
    acc[43] = fma(T(1), v, acc[43]);
    acc[64] = fma(px1, v, acc[64]);
    acc[68] = fma(py1, v, acc[68]);
    acc[69] = fma(pz1, v, acc[69]);
  }
  { const T v = Mc[44];
    acc[44] = fma(T(1), v, acc[44]);
    acc[65] = fma(px1, v, acc[65]);
    acc[70] = fma(py1, v, acc[70]);
    acc[71] = fma(pz1, v, acc[71]);
  }
  { const T v = Mc[45];
    acc[45] = fma(T(1), v, acc[45]);
    acc[66] = fma(px1, v, acc[66]);
    acc[71] = fma(py1, v, acc[71]);
    acc[72] = fma(pz1, v, acc[72]);
  }
  { const T v = Mc[46];
    acc[46] = fma(T(1), v, acc[46]);
    acc[67] = fma(px1, v, acc[67]);
    acc[72] = fma(py1, v, acc[72]);
    acc[73] = fma(pz1, v, acc[73]);
  }
  { const T v = Mc[47];
    acc[47] = fma(T(1), v, acc[47]);
    acc[68] = fma(px1, v, acc[68]);
    acc[73] = fma(py1, v, acc[73]);
    acc[74] = fma(pz1, v, acc[74]);
  }
  { const T v = Mc[48];
    acc[48] = fma(T(1), v, acc[48]);
    acc[69] = fma(px1, v, acc[69]);
    acc[74] = fma(py1, v, acc[74]);
    acc[75] = fma(pz1, v, acc[75]);
  }
  { const T v = Mc[49];
    acc[49] = fma(T(1), v, acc[49]);
    acc[70] = fma(px1, v, acc[70]);
    acc[76] = fma(py1, v, acc[76]);
    acc[77] = fma(pz1, v, acc[77]);
  }
  { const T v = Mc[50];
    acc[50] = fma(T(1), v, acc[50]);
    acc[71] = fma(px1, v, acc[71]);
    acc[77] = fma(py1, v, acc[77]);
    acc[78] = fma(pz1, v, acc[78]);
  }
  { const T v = Mc[51];
    acc[51] = fma(T(1), v, acc[51]);
    acc[72] = fma(px1, v, acc[72]);
    acc[78] = fma(py1, v, acc[78]);
    acc[79] = fma(pz1, v, acc[79]);
  }
  { const T v = Mc[52];
    acc[52] = fma(T(1), v, acc[52]);
    acc[73] = fma(px1, v, acc[73]);
    acc[79] = fma(py1, v, acc[79]);
    acc[80] = fma(pz1, v, acc[80]);
  }
  { const T v = Mc[53];
    acc[53] = fma(T(1), v, acc[53]);
    acc[74] = fma(px1, v, acc[74]);
    acc[80] = fma(py1, v, acc[80]);
    acc[81] = fma(pz1, v, acc[81]);
  }
  { const T v = Mc[54];
    acc[54] = fma(T(1), v, acc[54]);
    acc[75] = fma(px1, v, acc[75]);
    acc[81] = fma(py1, v, acc[81]);
    acc[82] = fma(pz1, v, acc[82]);
  }
  { const T v = Mc[55];
    acc[55] = fma(T(1), v, acc[55]);
  }
  { const T v = Mc[56];
    acc[56] = fma(T(1), v, acc[56]);
  }
  { const T v = Mc[57];
    acc[57] = fma(T(1), v, acc[57]);
  }
  { const T v = Mc[58];
    acc[58] = fma(T(1), v, acc[58]);
  }
  { const T v = Mc[59];
    acc[59] = fma(T(1), v, acc[59]);
  }
  { const T v = Mc[60];
    acc[60] = fma(T(1), v, acc[60]);
  }
  { const T v = Mc[61];
    acc[61] = fma(T(1), v, acc[61]);
  }
  { const T v = Mc[62];
    acc[62] = fma(T(1), v, acc[62]);
  }
  { const T v = Mc[63];
    acc[63] = fma(T(1), v, acc[63]);
  }
  { const T v = Mc[64];
    acc[64] = fma(T(1), v, acc[64]);
  }
  { const T v = Mc[65];
    acc[65] = fma(T(1), v, acc[65]);
  }
  { const T v = Mc[66];
    acc[66] = fma(T(1), v, acc[66]);
  }
  { const T v = Mc[67];
    acc[67] = fma(T(1), v, acc[67]);
  }
  { const T v = Mc[68];
    acc[68] = fma(T(1), v, acc[68]);
  }
  { const T v = Mc[69];
    acc[69] = fma(T(1), v, acc[69]);
  }
  { const T v = Mc[70];
    acc[70] = fma(T(1), v, acc[70]);
  }
  { const T v = Mc[71];
    acc[71] = fma(T(1), v, acc[71]);
  }
  { const T v = Mc[72];
    acc[72] = fma(T(1), v, acc[72]);
  }
  { const T v = Mc[73];
    acc[73] = fma(T(1), v, acc[73]);
  }
  { const T v = Mc[74];
    acc[74] = fma(T(1), v, acc[74]);
  }
  { const T v = Mc[75];
    acc[75] = fma(T(1), v, acc[75]);
  }
  { const T v = Mc[76];
    acc[76] = fma(T(1), v, acc[76]);
  }
  { const T v = Mc[77];
    acc[77] = fma(T(1), v, acc[77]);
  }
  { const T v = Mc[78];
    acc[78] = fma(T(1), v, acc[78]);
  }
  { const T v = Mc[79];
    acc[79] = fma(T(1), v, acc[79]);
  }
  { const T v = Mc[80];
    acc[80] = fma(T(1), v, acc[80]);
  }
  { const T v = Mc[81];
    acc[81] = fma(T(1), v, acc[81]);
  }
  { const T v = Mc[82];
    acc[82] = fma(T(1), v, acc[82]);
  }
}
// L2L: local expansion Lc about a centre at -(x, y, z) from this one, order 6
template <typename T>
__device__ __forceinline__ void l2l_m1_p6(T x, T y, T z, const T* __restrict__ Lc, T* __restrict__ acc) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T px5 = px4 * x * cinv<T>(5);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T py5 = py4 * y * cinv<T>(5);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T pz5 = pz4 * z * cinv<T>(5);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  const T m_4_1_0 = px4 * py1;
  const T m_4_0_1 = px4 * pz1;
  const T m_3_2_0 = px3 * py2;
  const T m_3_1_1 = px3 * py1 * pz1;
  const T m_3_0_2 = px3 * pz2;
  const T m_2_3_0 = px2 * py3;
  const T m_2_2_1 = px2 * py2 * pz1;
  const T m_2_1_2 = px2 * py1 * pz2;
  const T m_2_0_3 = px2 * pz3;
  const T m_1_4_0 = px1 * py4;
  const T m_1_3_1 = px1 * py3 * pz1;
  const T m_1_2_2 = px1 * py2 * pz2;
  const T m_1_1_3 = px1 * py1 * pz3;
  const T m_1_0_4 = px1 * pz4;
  const T m_0_4_1 = py4 * pz1;
  const T m_0_3_2 = py3 * pz2;
  const T m_0_2_3 = py2 * pz3;
  const T m_0_1_4 = py1 * pz4;
  { const T v = Lc[0];
    acc[0] = fma(T(1), v, acc[0]);
  }
  { const T v = Lc[1];
    acc[0] = fma(px1, v, acc[0]);
    acc[1] = fma(T(1), v, acc[1]);
  }
  { const T v = Lc[2];
    acc[0] = fma(py1, v, acc[0]);
    acc[2] = fma(T(1), v, acc[2]);
  }
  { const T v = Lc[3];
    acc[0] = fma(pz1, v, acc[0]);
    acc[3] = fma(T(1), v, acc[3]);
  }
  { const T v = Lc[4];
    acc[0] = fma(px2, v, acc[0]);
    acc[1] = fma(px1, v, acc[1]);
    acc[4] = fma(T(1), v, acc[4]);
  }
  { const T v = Lc[5];
    acc[0] = fma(m_1_1_0, v, acc[0]);
    acc[1] = fma(py1, v, acc[1]);
    acc[2] = fma(px1, v, acc[2]);
    acc[5] = fma(T(1), v, acc[5]);
  }
  { const T v = Lc[6];
    acc[0] = fma(m_1_0_1, v, acc[0]);
    acc[1] = fma(pz1, v, acc[1]);
    acc[3] = fma(px1, v, acc[3]);
    acc[6] = fma(T(1), v, acc[6]);
  }
  { const T v = Lc[7];
    acc[0] = fma(py2, v, acc[0]);
    acc[2] = fma(py1, v, acc[2]);
    acc[7] = fma(T(1), v, acc[7]);
  }
  { const T v = Lc[8];
    acc[0] = fma(m_0_1_1, v, acc[0]);
    acc[2] = fma(pz1, v, acc[2]);
    acc[3] = fma(py1, v, acc[3]);
    acc[8] = fma(T(1), v, acc[8]);
  }
  { const T v = Lc[9];
    acc[0] = fma(pz2, v, acc[0]);
    acc[3] = fma(pz1, v, acc[3]);
    acc[9] = fma(T(1), v, acc[9]);
  }
  { const T v = Lc[10];
    acc[0] = fma(px3, v, acc[0]);
    acc[1] = fma(px2, v, acc[1]);
    acc[4] = fma(px1, v, acc[4]);
    acc[10] = fma(T(1), v, acc[10]);
  }
  { const T v = Lc[11];
    acc[0] = fma(m_2_1_0, v, acc[0]);
    acc[1] = fma(m_1_1_0, v, acc[1]);
    acc[2] = fma(px2, v, acc[2]);
    acc[4] = fma(py1, v, acc[4]);
    acc[5] = fma(px1, v, acc[5]);
    acc[11] = fma(T(1), v, acc[11]);
  }
  { const T v = Lc[12];
    acc[0] = fma(m_2_0_1, v, acc[0]);
    acc[1] = fma(m_1_0_1, v, acc[1]);
    acc[3] = fma(px2, v, acc[3]);
    acc[4] = fma(pz1, v, acc[4]);
    acc[6] = fma(px1, v, acc[6]);
    acc[12] = fma(T(1), v, acc[12]);
  }
  { const T v = Lc[13];
    acc[0] = fma(m_1_2_0, v, acc[0]);
    acc[1] = fma(py2, v, acc[1]);
    acc[2] = fma(m_1_1_0, v, acc[2]);
    acc[5] = fma(py1, v, acc[5]);
    acc[7] = fma(px1, v, acc[7]);
    acc[13] = fma(T(1), v, acc[13]);
  }
  { const T v = Lc[14];
    acc[0] = fma(m_1_1_1, v, acc[0]);
    acc[1] = fma(m_0_1_1, v, acc[1]);
    acc[2] = fma(m_1_0_1, v, acc[2]);
    acc[3] = fma(m_1_1_0, v, acc[3]);
    acc[5] = fma(pz1, v, acc[5]);
    acc[6] = fma(py1, v, acc[6]);
    acc[8] = fma(px1, v, acc[8]);
    acc[14] = fma(T(1), v, acc[14]);
  }
  { const T v = Lc[15];
    acc[0] = fma(m_1_0_2, v, acc[0]);
    acc[1] = fma(pz2, v, acc[1]);
    acc[3] = fma(m_1_0_1, v, acc[3]);
    acc[6] = fma(pz1, v, acc[6]);
    acc[9] = fma(px1, v, acc[9]);
    acc[15] = fma(T(1), v, acc[15]);
  }
  { const T v = Lc[16];
    acc[0] = fma(py3, v, acc[0]);
    acc[2] = fma(py2, v, acc[2]);
    acc[7] = fma(py1, v, acc[7]);
    acc[16] = fma(T(1), v, acc[16]);
  }
  { const T v = Lc[17];
    acc[0] = fma(m_0_2_1, v, acc[0]);
    acc[2] = fma(m_0_1_1, v, acc[2]);
    acc[3] = fma(py2, v, acc[3]);
    acc[7] = fma(pz1, v, acc[7]);
    acc[8] = fma(py1, v, acc[8]);
    acc[17] = fma(T(1), v, acc[17]);
  }
  { const T v = Lc[18];
    acc[0] = fma(m_0_1_2, v, acc[0]);
    acc[2] = fma(pz2, v, acc[2]);
    acc[3] = fma(m_0_1_1, v, acc[3]);
    acc[8] = fma(pz1, v, acc[8]);
    acc[9] = fma(py1, v, acc[9]);
    acc[18] = fma(T(1), v, acc[18]);
  }
  { const T v = Lc[19];
    acc[0] = fma(pz3, v, acc[0]);
    acc[3] = fma(pz2, v, acc[3]);
    acc[9] = fma(pz1, v, acc[9]);
    acc[19] = fma(T(1), v, acc[19]);
  }
  { const T v = Lc[20];
    acc[0] = fma(px4, v, acc[0]);
    acc[1] = fma(px3, v, acc[1]);
    acc[4] = fma(px2, v, acc[4]);
    acc[10] = fma(px1, v, acc[10]);
    acc[20] = fma(T(1), v, acc[20]);
  }
  { const T v = Lc[21];
    acc[0] = fma(m_3_1_0, v, acc[0]);
    acc[1] = fma(m_2_1_0, v, acc[1]);
    acc[2] = fma(px3, v, acc[2]);
    acc[4] = fma(m_1_1_0, v, acc[4]);
    acc[5] = fma(px2, v, acc[5]);
    acc[10] = fma(py1, v, acc[10]);
    acc[11] = fma(px1, v, acc[11]);
    acc[21] = fma(T(1), v, acc[21]);
  }
  { const T v = Lc[22];
    acc[0] = fma(m_3_0_1, v, acc[0]);
    acc[1] = fma(m_2_0_1, v, acc[1]);
    acc[3] = fma(px3, v, acc[3]);
    acc[4] = fma(m_1_0_1, v, acc[4]);
    acc[6] = fma(px2, v, acc[6]);
    acc[10] = fma(pz1, v, acc[10]);
    acc[12] = fma(px1, v, acc[12]);
    acc[22] = fma(T(1), v, acc[22]);
  }
  { const T v = Lc[23];
    acc[0] = fma(m_2_2_0, v, acc[0]);
    acc[1] = fma(m_1_2_0, v, acc[1]);
    acc[2] = fma(m_2_1_0, v, acc[2]);
    acc[4] = fma(py2, v, acc[4]);
    acc[5] = fma(m_1_1_0, v, acc[5]);
    acc[7] = fma(px2, v, acc[7]);
    acc[11] = fma(py1, v, acc[11]);
    acc[13] = fma(px1, v, acc[13]);
    acc[23] = fma(T(1), v, acc[23]);
  }
  { const T v = Lc[24];
    acc[0] = fma(m_2_1_1, v, acc[0]);
    acc[1] = fma(m_1_1_1, v, acc[1]);
    acc[2] = fma(m_2_0_1, v, acc[2]);
    acc[3] = fma(m_2_1_0, v, acc[3]);
    acc[4] = fma(m_0_1_1, v, acc[4]);
    acc[5] = fma(m_1_0_1, v, acc[5]);
    acc[6] = fma(m_1_1_0, v, acc[6]);
    acc[8] = fma(px2, v, acc[8]);
    acc[11] = fma(pz1, v, acc[11]);
    acc[12] = fma(py1, v, acc[12]);
    acc[14] = fma(px1, v, acc[14]);
    acc[24] = fma(T(1), v, acc[24]);
  }
  { const T v = Lc[25];
    acc[0] = fma(m_2_0_2, v, acc[0]);
    acc[1] = fma(m_1_0_2, v, acc[1]);
    acc[3] = fma(m_2_0_1, v, acc[3]);
    acc[4] = fma(pz2, v, acc[4]);
    acc[6] = fma(m_1_0_1, v, acc[6]);
    acc[9] = fma(px2, v, acc[9]);
    acc[12] = fma(pz1, v, acc[12]);
    acc[15] = fma(px1, v, acc[15]);
    acc[25] = fma(T(1), v, acc[25]);
  }
  { const T v = Lc[26];
    acc[0] = fma(m_1_3_0, v, acc[0]);
    acc[1] = fma(py3, v, acc[1]);
    acc[2] = fma(m_1_2_0, v, acc[2]);
    acc[5] = fma(py2, v, acc[5]);
    acc[7] = fma(m_1_1_0, v, acc[7]);
    acc[13] = fma(py1, v, acc[13]);
    acc[16] = fma(px1, v, acc[16]);
    acc[26] = fma(T(1), v, acc[26]);
  }
  { const T v = Lc[27];
    acc[0] = fma(m_1_2_1, v, acc[0]);
    acc[1] = fma(m_0_2_1, v, acc[1]);
    acc[2] = fma(m_1_1_1, v, acc[2]);
    acc[3] = fma(m_1_2_0, v, acc[3]);
    acc[5] = fma(m_0_1_1, v, acc[5]);
    acc[6] = fma(py2, v, acc[6]);
    acc[7] = fma(m_1_0_1, v, acc[7]);
    acc[8] = fma(m_1_1_0, v, acc[8]);
    acc[13] = fma(pz1, v, acc[13]);
    acc[14] = fma(py1, v, acc[14]);
    acc[17] = fma(px1, v, acc[17]);
    acc[27] = fma(T(1), v, acc[27]);
  }
  { const T v = Lc[28];
    acc[0] = fma(m_1_1_2, v, acc[0]);
    acc[1] = fma(m_0_1_2, v, acc[1]);
    acc[2] = fma(m_1_0_2, v, acc[2]);
    acc[3] = fma(m_1_1_1, v, acc[3]);
    acc[5] = fma(pz2, v, acc[5]);
    acc[6] = fma(m_0_1_1, v, acc[6]);
    acc[8] = fma(m_1_0_1, v, acc[8]);
    acc[9] = fma(m_1_1_0, v, acc[9]);
    acc[14] = fma(pz1, v, acc[14]);
    acc[15] = fma(py1, v, acc[15]);
    acc[18] = fma(px1, v, acc[18]);
    acc[28] = fma(T(1), v, acc[28]);
  }
  { const T v = Lc[29];
    acc[0] = fma(m_1_0_3, v, acc[0]);
    acc[1] = fma(pz3, v, acc[1]);
    acc[3] = fma(m_1_0_2, v, acc[3]);
    acc[6] = fma(pz2, v, acc[6]);
    acc[9] = fma(m_1_0_1, v, acc[9]);
    acc[15] = fma(pz1, v, acc[15]);
    acc[19] = fma(px1, v, acc[19]);
    acc[29] = fma(T(1), v, acc[29]);
  }
  { const T v = Lc[30];
    acc[0] = fma(py4, v, acc[0]);
    acc[2] = fma(py3, v, acc[2]);
    acc[7] = fma(py2, v, acc[7]);
    acc[16] = fma(py1, v, acc[16]);
    acc[30] = fma(T(1), v, acc[30]);
  }
  { const T v = Lc[31];
    acc[0] = fma(m_0_3_1, v, acc[0]);
    acc[2] = fma(m_0_2_1, v, acc[2]);
    acc[3] = fma(py3, v, acc[3]);
    acc[7] = fma(m_0_1_1, v, acc[7]);
    acc[8] = fma(py2, v, acc[8]);
    acc[16] = fma(pz1, v, acc[16]);
    acc[17] = fma(py1, v, acc[17]);
    acc[31] = fma(T(1), v, acc[31]);
  }
  { const T v = Lc[32];
    acc[0] = fma(m_0_2_2, v, acc[0]);
    acc[2] = fma(m_0_1_2, v, acc[2]);
    acc[3] = fma(m_0_2_1, v, acc[3]);
    acc[7] = fma(pz2, v, acc[7]);
    acc[8] = fma(m_0_1_1, v, acc[8]);
    acc[9] = fma(py2, v, acc[9]);
    acc[17] = fma(pz1, v, acc[17]);
    acc[18] = fma(py1, v, acc[18]);
    acc[32] = fma(T(1), v, acc[32]);
  }
  { const T v = Lc[33];
    acc[0] = fma(m_0_1_3, v, acc[0]);
    acc[2] = fma(pz3, v, acc[2]);
    acc[3] = fma(m_0_1_2, v, acc[3]);
    acc[8] = fma(pz2, v, acc[8]);
    acc[9] = fma(m_0_1_1, v, acc[9]);
    acc[18] = fma(pz1, v, acc[18]);
    acc[19] = fma(py1, v, acc[19]);
    acc[33] = fma(T(1), v, acc[33]);
  }
  { const T v = Lc[34];
    acc[0] = fma(pz4, v, acc[0]);
    acc[3] = fma(pz3, v, acc[3]);
    acc[9] = fma(pz2, v, acc[9]);
    acc[19] = fma(pz1, v, acc[19]);
    acc[34] = fma(T(1), v, acc[34]);
  }
  { const T v = Lc[35];
    acc[0] = fma(px5, v, acc[0]);
    acc[1] = fma(px4, v, acc[1]);
    acc[4] = fma(px3, v, acc[4]);
    acc[10] = fma(px2, v, acc[10]);
    acc[20] = fma(px1, v, acc[20]);
    acc[35] = fma(T(1), v, acc[35]);
  }
  { const T v = Lc[36];
    acc[0] = fma(m_4_1_0, v, acc[0]);
    acc[1] = fma(m_3_1_0, v, acc[1]);
    acc[2] = fma(px4, v, acc[2]);
    acc[4] = fma(m_2_1_0, v, acc[4]);
    acc[5] = fma(px3, v, acc[5]);
    acc[10] = fma(m_1_1_0, v, acc[10]);
    acc[11] = fma(px2, v, acc[11]);
    acc[20] = fma(py1, v, acc[20]);
    acc[21] = fma(px1, v, acc[21]);
    acc[36] = fma(T(1), v, acc[36]);
  }
  { const T v = Lc[37];
    acc[0] = fma(m_4_0_1, v, acc[0]);
    acc[1] = fma(m_3_0_1, v, acc[1]);
    acc[3] = fma(px4, v, acc[3]);
    acc[4] = fma(m_2_0_1, v, acc[4]);
    acc[6] = fma(px3, v, acc[6]);
    acc[10] = fma(m_1_0_1, v, acc[10]);
    acc[12] = fma(px2, v, acc[12]);
    acc[20] = fma(pz1, v, acc[20]);
    acc[22] = fma(px1, v, acc[22]);
    acc[37] = fma(T(1), v, acc[37]);
  }
  { const T v = Lc[38];
    acc[0] = fma(m_3_2_0, v, acc[0]);
    acc[1] = fma(m_2_2_0, v, acc[1]);
    acc[2] = fma(m_3_1_0, v, acc[2]);
    acc[4] = fma(m_1_2_0, v, acc[4]);
    acc[5] = fma(m_2_1_0, v, acc[5]);
    acc[7] = fma(px3, v, acc[7]);
    acc[10] = fma(py2, v, acc[10]);
    acc[11] = fma(m_1_1_0, v, acc[11]);
    acc[13] = fma(px2, v, acc[13]);
    acc[21] = fma(py1, v, acc[21]);
    acc[23] = fma(px1, v, acc[23]);
    acc[38] = fma(T(1), v, acc[38]);
  }
  { const T v = Lc[39];
    acc[0] = fma(m_3_1_1, v, acc[0]);
    acc[1] = fma(m_2_1_1, v, acc[1]);
    acc[2] = fma(m_3_0_1, v, acc[2]);
    acc[3] = fma(m_3_1_0, v, acc[3]);
    acc[4] = fma(m_1_1_1, v, acc[4]);
    acc[5] = fma(m_2_0_1, v, acc[5]);
    acc[6] = fma(m_2_1_0, v, acc[6]);
    acc[8] = fma(px3, v, acc[8]);
    acc[10] = fma(m_0_1_1, v, acc[10]);
    acc[11] = fma(m_1_0_1, v, acc[11]);
    acc[12] = fma(m_1_1_0, v, acc[12]);
    acc[14] = fma(px2, v, acc[14]);
    acc[21] = fma(pz1, v, acc[21]);
    acc[22] = fma(py1, v, acc[22]);
    acc[24] = fma(px1, v, acc[24]);
    acc[39] = fma(T(1), v, acc[39]);
  }
  { const T v = Lc[40];
    acc[0] = fma(m_3_0_2, v, acc[0]);
    acc[1] = fma(m_2_0_2, v, acc[1]);
    acc[3] = fma(m_3_0_1, v, acc[3]);
    acc[4] = fma(m_1_0_2, v, acc[4]);
    acc[6] = fma(m_2_0_1, v, acc[6]);
    acc[9] = fma(px3, v, acc[9]);
    acc[10] = fma(pz2, v, acc[10]);
    acc[12] = fma(m_1_0_1, v, acc[12]);
    acc[15] = fma(px2, v, acc[15]);
    acc[22] = fma(pz1, v, acc[22]);
    acc[25] = fma(px1, v, acc[25]);
    acc[40] = fma(T(1), v, acc[40]);
  }
  { const T v = Lc[41];
    acc[0] = fma(m_2_3_0, v, acc[0]);
    acc[1] = fma(m_1_3_0, v, acc[1]);
    acc[2] = fma(m_2_2_0, v, acc[2]);
    acc[4] = fma(py3, v, acc[4]);
    acc[5] = fma(m_1_2_0, v, acc[5]);
    acc[7] = fma(m_2_1_0, v, acc[7]);
    acc[11] = fma(py2, v, acc[11]);
    acc[13] = fma(m_1_1_0, v, acc[13]);
    acc[16] = fma(px2, v, acc[16]);
    acc[23] = fma(py1, v, acc[23]);
    acc[26] = fma(px1, v, acc[26]);
    acc[41] = fma(T(1), v, acc[41]);
  }
  { const T v = Lc[42];
    acc[0] = fma(m_2_2_1, v, acc[0]);
    acc[1] = fma(m_1_2_1, v, acc[1]);
    acc[2] = fma(m_2_1_1, v, acc[2]);
    acc[3] = fma(m_2_2_0, v, acc[3]);
    acc[4] = fma(m_0_2_1, v, acc[4]);
    acc[5] = fma(m_1_1_1, v, acc[5]);
    acc[6] = fma(m_1_2_0, v, acc[6]);
    acc[7] = fma(m_2_0_1, v, acc[7]);
    acc[8] = fma(m_2_1_0, v, acc[8]);
    acc[11] = fma(m_0_1_1, v, acc[11]);
    acc[12] = fma(py2, v, acc[12]);
    acc[13] = fma(m_1_0_1, v, acc[13]);
    acc[14] = fma(m_1_1_0, v, acc[14]);
    acc[17] = fma(px2, v, acc[17]);
    acc[23] = fma(pz1, v, acc[23]);
    acc[24] = fma(py1, v, acc[24]);
    acc[27] = fma(px1, v, acc[27]);
    acc[42] = fma(T(1), v, acc[42]);
  }
  { const T v = Lc[43];
    acc[0] = fma(m_2_1_2, v, acc[0]);
    acc[1] = fma(m_1_1_2, v, acc[1]);
    acc[2] = fma(m_2_0_2, v, acc[2]);
    acc[3] = fma(m_2_1_1, v, acc[3]);
    acc[4] = fma(m_0_1_2, v, acc[4]);
    acc[5] = fma(m_1_0_2, v, acc[5]);
    acc[6] = fma(m_1_1_1, v, acc[6]);
    acc[8] = fma(m_2_0_1, v, acc[8]);
    acc[9] = fma(m_2_1_0, v, acc[9]);
    acc[11] = fma(pz2, v, acc[11]);
    acc[12] = fma(m_0_1_1, v, acc[12]);
    acc[14] = fma(m_1_0_1, v, acc[14]);
    acc[15] = fma(m_1_1_0, v, acc[15]);
    acc[18] = fma(px2, v, acc[18]);
    acc[24] = fma(pz1, v, acc[24]);
    acc[25] = fma(py1, v, acc[25]);
    acc[28] = fma(px1, v, acc[28]);
    acc[43] = fma(T(1), v, acc[43]);
  }
  { const T v = Lc[44];
    acc[0] = fma(m_2_0_3, v, acc[0]);
    acc[1] = fma(m_1_0_3, v, acc[1]);
    acc[3] = fma(m_2_0_2, v, acc[3]);
    acc[4] = fma(pz3, v, acc[4]);
    acc[6] = fma(m_1_0_2, v, acc[6]);
    acc[9] = fma(m_2_0_1, v, acc[9]);
    acc[12] = fma(pz2, v, acc[12]);
    acc[15] = fma(m_1_0_1, v, acc[15]);
    acc[19] = fma(px2, v, acc[19]);
    acc[25] = fma(pz1, v, acc[25]);
    acc[29] = fma(px1, v, acc[29]);
    acc[44] = fma(T(1), v, acc[44]);
  }
  { const T v = Lc[45];
    acc[0] = fma(m_1_4_0, v, acc[0]);
    acc[1] = fma(py4, v, acc[1]);
    acc[2] = fma(m_1_3_0, v, acc[2]);
    acc[5] = fma(py3, v, acc[5]);
    acc[7] = fma(m_1_2_0, v, acc[7]);
    acc[13] = fma(py2, v, acc[13]);
    acc[16] = fma(m_1_1_0, v, acc[16]);
    acc[26] = fma(py1, v, acc[26]);
    acc[30] = fma(px1, v, acc[30]);
    acc[45] = fma(T(1), v, acc[45]);
  }
  { const T v = Lc[46];
    acc[0] = fma(m_1_3_1, v, acc[0]);
    acc[1] = fma(m_0_3_1, v, acc[1]);
    acc[2] = fma(m_1_2_1, v, acc[2]);
    acc[3] = fma(m_1_3_0, v, acc[3]);
    acc[5] = fma(m_0_2_1, v, acc[5]);
    acc[6] = fma(py3, v, acc[6]);
    acc[7] = fma(m_1_1_1, v, acc[7]);
    acc[8] = fma(m_1_2_0, v, acc[8]);
    acc[13] = fma(m_0_1_1, v, acc[13]);
    acc[14] = fma(py2, v, acc[14]);
    acc[16] = fma(m_1_0_1, v, acc[16]);
    acc[17] = fma(m_1_1_0, v, acc[17]);
    acc[26] = fma(pz1, v, acc[26]);
    acc[27] = fma(py1, v, acc[27]);
    acc[31] = fma(px1, v, acc[31]);
    acc[46] = fma(T(1), v, acc[46]);
  }
  { const T v = Lc[47];
    acc[0] = fma(m_1_2_2, v, acc[0]);
    acc[1] = fma(m_0_2_2, v, acc[1]);
    acc[2] = fma(m_1_1_2, v, acc[2]);
    acc[3] = fma(m_1_2_1, v, acc[3]);
    acc[5] = fma(m_0_1_2, v, acc[5]);
    acc[6] = fma(m_0_2_1, v, acc[6]);
    acc[7] = fma(m_1_0_2, v, acc[7]);
    acc[8] = fma(m_1_1_1, v, acc[8]);
    acc[9] = fma(m_1_2_0, v, acc[9]);
    acc[13] = fma(pz2, v, acc[13]);
    acc[14] = fma(m_0_1_1, v, acc[14]);
    acc[15] = fma(py2, v, acc[15]);
    acc[17] = fma(m_1_0_1, v, acc[17]);
    acc[18] = fma(m_1_1_0, v, acc[18]);
    acc[27] = fma(pz1, v, acc[27]);
    acc[28] = fma(py1, v, acc[28]);
    acc[32] = fma(px1, v, acc[32]);
    acc[47] = fma(T(1), v, acc[47]);
  }
  { const T v = Lc[48];
    acc[0] = fma(m_1_1_3, v, acc[0]);
    acc[1] = fma(m_0_1_3, v, acc[1]);
    acc[2] = fma(m_1_0_3, v, acc[2]);
    acc[3] = fma(m_1_1_2, v, acc[3]);
    acc[5] = fma(pz3, v, acc[5]);
    acc[6] = fma(m_0_1_2, v, acc[6]);
    acc[8] = fma(m_1_0_2, v, acc[8]);
    acc[9] = fma(m_1_1_1, v, acc[9]);
    acc[14] = fma(pz2, v, acc[14]);
    acc[15] = fma(m_0_1_1, v, acc[15]);
    acc[18] = fma(m_1_0_1, v, acc[18]);
    acc[19] = fma(m_1_1_0, v, acc[19]);
    acc[28] = fma(pz1, v, acc[28]);
    acc[29] = fma(py1, v, acc[29]);
    acc[33] = fma(px1, v, acc[33]);
    acc[48] = fma(T(1), v, acc[48]);
  }
  { const T v = Lc[49];
    acc[0] = fma(m_1_0_4, v, acc[0]);
    acc[1] = fma(pz4, v, acc[1]);
    acc[3] = fma(m_1_0_3, v, acc[3]);
    acc[6] = fma(pz3, v, acc[6]);
    acc[9] = fma(m_1_0_2, v, acc[9]);
    acc[15] = fma(pz2, v, acc[15]);
    acc[19] = fma(m_1_0_1, v, acc[19]);
    acc[29] = fma(pz1, v, acc[29]);
    acc[34] = fma(px1, v, acc[34]);
    acc[49] = fma(T(1), v, acc[49]);
  }
  { const T v = Lc[50];
    acc[0] = fma(py5, v, acc[0]);
    acc[2] = fma(py4, v, acc[2]);
    acc[7] = fma(py3, v, acc[7]);
    acc[16] = fma(py2, v, acc[16]);
    acc[30] = fma(py1, v, acc[30]);
    acc[50] = fma(T(1), v, acc[50]);
  }
  { const T v = Lc[51];
    acc[0] = fma(m_0_4_1, v, acc[0]);
    acc[2] = fma(m_0_3_1, v, acc[2]);
    acc[3] = fma(py4, v, acc[3]);
    acc[7] = fma(m_0_2_1, v, acc[7]);
    acc[8] = fma(py3, v, acc[8]);
    acc[16] = fma(m_0_1_1, v, acc[16]);
    acc[17] = fma(py2, v, acc[17]);
    acc[30] = fma(pz1, v, acc[30]);
    acc[31] = fma(py1, v, acc[31]);
    acc[51] = fma(T(1), v, acc[51]);
  }
  { const T v = Lc[52];
    acc[0] = fma(m_0_3_2, v, acc[0]);
    acc[2] = fma(m_0_2_2, v, acc[2]);
    acc[3] = fma(m_0_3_1, v, acc[3]);
    acc[7] = fma(m_0_1_2, v, acc[7]);
    acc[8] = fma(m_0_2_1, v, acc[8]);
    acc[9] = fma(py3, v, acc[9]);
    acc[16] = fma(pz2, v, acc[16]);
    acc[17] = fma(m_0_1_1, v, acc[17]);
    acc[18] = fma(py2, v, acc[18]);
    acc[31] = fma(pz1, v, acc[31]);
    acc[32] = fma(py1, v, acc[32]);
    acc[52] = fma(T(1), v, acc[52]);
  }
  { const T v = Lc[53];
    acc[0] = fma(m_0_2_3, v, acc[0]);
    acc[2] = fma(m_0_1_3, v, acc[2]);
    acc[3] = fma(m_0_2_2, v, acc[3]);
    acc[7] = fma(pz3, v, acc[7]);
    acc[8] = fma(m_0_1_2, v, acc[8]);
    acc[9] = fma(m_0_2_1, v, acc[9]);
    acc[17] = fma(pz2, v, acc[17]);
    acc[18] = fma(m_0_1_1, v, acc[18]);
    acc[19] = fma(py2, v, acc[19]);
    acc[32] = fma(pz1, v, acc[32]);
    acc[33] = fma(py1, v, acc[33]);
    acc[53] = fma(T(1), v, acc[53]);
  }
  { const T v = Lc[54];
    acc[0] = fma(m_0_1_4, v, acc[0]);
    acc[2] = fma(pz4, v, acc[2]);
    acc[3] = fma(m_0_1_3, v, acc[3]);
    acc[8] = fma(pz3, v, acc[8]);
    acc[9] = fma(m_0_1_2, v, acc[9]);
    acc[18] = fma(pz2, v, acc[18]);
    acc[19] = fma(m_0_1_1, v, acc[19]);
    acc[33] = fma(pz1, v, acc[33]);
    acc[34] = fma(py1, v, acc[34]);
    acc[54] = fma(T(1), v, acc[54]);
  }
  { const T v = Lc[55];
    acc[0] = fma(pz5, v, acc[0]);
    acc[3] = fma(pz4, v, acc[3]);
    acc[9] = fma(pz3, v, acc[9]);
    acc[19] = fma(pz2, v, acc[19]);
    acc[34] = fma(pz1, v, acc[34]);
    acc[55] = fma(T(1), v, acc[55]);
  }
}
// L2P: field -grad of the local expansion Lc at offset (x, y, z) = site - centre, order 6
template <typename T>
__device__ __forceinline__ void l2p_m1_p6(T x, T y, T z, const T* __restrict__ Lc, T& f0, T& f1, T& f2) {
  const T px1 = x;
  const T px2 = px1 * x * cinv<T>(2);
  const T px3 = px2 * x * cinv<T>(3);
  const T px4 = px3 * x * cinv<T>(4);
  const T py1 = y;
  const T py2 = py1 * y * cinv<T>(2);
  const T py3 = py2 * y * cinv<T>(3);
  const T py4 = py3 * y * cinv<T>(4);
  const T pz1 = z;
  const T pz2 = pz1 * z * cinv<T>(2);
  const T pz3 = pz2 * z * cinv<T>(3);
  const T pz4 = pz3 * z * cinv<T>(4);
  const T m_1_1_0 = px1 * py1;
  const T m_1_0_1 = px1 * pz1;
  const T m_0_1_1 = py1 * pz1;
  const T m_2_1_0 = px2 * py1;
  const T m_2_0_1 = px2 * pz1;
  const T m_1_2_0 = px1 * py2;
  const T m_1_1_1 = px1 * py1 * pz1;
  const T m_1_0_2 = px1 * pz2;
  const T m_0_2_1 = py2 * pz1;
  const T m_0_1_2 = py1 * pz2;
  const T m_3_1_0 = px3 * py1;
  const T m_3_0_1 = px3 * pz1;
  const T m_2_2_0 = px2 * py2;
  const T m_2_1_1 = px2 * py1 * pz1;
  const T m_2_0_2 = px2 * pz2;
  const T m_1_3_0 = px1 * py3;
  const T m_1_2_1 = px1 * py2 * pz1;
  const T m_1_1_2 = px1 * py1 * pz2;
  const T m_1_0_3 = px1 * pz3;
  const T m_0_3_1 = py3 * pz1;
  const T m_0_2_2 = py2 * pz2;
  const T m_0_1_3 = py1 * pz3;
  { const T v = -Lc[1];
    f0 = fma(T(1), v, f0);
  }
  { const T v = -Lc[2];
    f1 = fma(T(1), v, f1);
  }
  { const T v = -Lc[3];
    f2 = fma(T(1), v, f2);
  }
  { const T v = -Lc[4];
    f0 = fma(px1, v, f0);
  }
  { const T v = -Lc[5];
    f0 = fma(py1, v, f0);
    f1 = fma(px1, v, f1);
  }
  { const T v = -Lc[6];
    f0 = fma(pz1, v, f0);
    f2 = fma(px1, v, f2);
  }
  { const T v = -Lc[7];
    f1 = fma(py1, v, f1);
  }
  { const T v = -Lc[8];
    f1 = fma(pz1, v, f1);
    f2 = fma(py1, v, f2);
  }
  { const T v = -Lc[9];
    f2 = fma(pz1, v, f2);
  }
  { const T v = -Lc[10];
    f0 = fma(px2, v, f0);
  }
  { const T v = -Lc[11];
    f0 = fma(m_1_1_0, v, f0);
    f1 = fma(px2, v, f1);
  }
  { const T v = -Lc[12];
    f0 = fma(m_1_0_1, v, f0);
    f2 = fma(px2, v, f2);
  }
  { const T v = -Lc[13];
    f0 = fma(py2, v, f0);
    f1 = fma(m_1_1_0, v, f1);
  }
  { const T v = -Lc[14];
    f0 = fma(m_0_1_1, v, f0);
    f1 = fma(m_1_0_1, v, f1);
    f2 = fma(m_1_1_0, v, f2);
  }
  { const T v = -Lc[15];
    f0 = fma(pz2, v, f0);
    f2 = fma(m_1_0_1, v, f2);
  }
  { const T v = -Lc[16];
    f1 = fma(py2, v, f1);
  }
  { const T v = -Lc[17];
    f1 = fma(m_0_1_1, v, f1);
    f2 = fma(py2, v, f2);
  }
  { const T v = -Lc[18];
    f1 = fma(pz2, v, f1);
    f2 = fma(m_0_1_1, v, f2);
  }
  { const T v = -Lc[19];
    f2 = fma(pz2, v, f2);
  }
  { const T v = -Lc[20];
    f0 = fma(px3, v, f0);
  }
  { const T v = -Lc[21];
    f0 = fma(m_2_1_0, v, f0);
    f1 = fma(px3, v, f1);
  }
  { const T v = -Lc[22];
    f0 = fma(m_2_0_1, v, f0);
    f2 = fma(px3, v, f2);
  }
  { const T v = -Lc[23];
    f0 = fma(m_1_2_0, v, f0);
    f1 = fma(m_2_1_0, v, f1);
  }
  { const T v = -Lc[24];
    f0 = fma(m_1_1_1, v, f0);
    f1 = fma(m_2_0_1, v, f1);
    f2 = fma(m_2_1_0, v, f2);
  }
  { const T v = -Lc[25];
    f0 = fma(m_1_0_2, v, f0);
    f2 = fma(m_2_0_1, v, f2);
  }
  { const T v = -Lc[26];
    f0 = fma(py3, v, f0);
    f1 = fma(m_1_2_0, v, f1);
  }
  { const T v = -Lc[27];
    f0 = fma(m_0_2_1, v, f0);
    f1 = fma(m_1_1_1, v, f1);
    f2 = fma(m_1_2_0, v, f2);
  }
  { const T v = -Lc[28];
    f0 = fma(m_0_1_2, v, f0);
    f1 = fma(m_1_0_2, v, f1);
    f2 = fma(m_1_1_1, v, f2);
  }
  { const T v = -Lc[29];
    f0 = fma(pz3, v, f0);
    f2 = fma(m_1_0_2, v, f2);
  }
  { const T v = -Lc[30];
    f1 = fma(py3, v, f1);
  }
  { const T v = -Lc[31];
    f1 = fma(m_0_2_1, v, f1);
    f2 = fma(py3, v, f2);
  }
  { const T v = -Lc[32];
    f1 = fma(m_0_1_2, v, f1);
    f2 = fma(m_0_2_1, v, f2);
  }
  { const T v = -Lc[33];
    f1 = fma(pz3, v, f1);
    f2 = fma(m_0_1_2, v, f2);
  }
  { const T v = -Lc[34];
    f2 = fma(pz3, v, f2);
  }
  { const T v = -Lc[35];
    f0 = fma(px4, v, f0);
  }
  { const T v = -Lc[36];
    f0 = fma(m_3_1_0, v, f0);
    f1 = fma(px4, v, f1);
  }
  { const T v = -Lc[37];
    f0 = fma(m_3_0_1, v, f0);
    f2 = fma(px4, v, f2);
  }
  { const T v = -Lc[38];
    f0 = fma(m_2_2_0, v, f0);
    f1 = fma(m_3_1_0, v, f1);
  }
  { const T v = -Lc[39];
    f0 = fma(m_2_1_1, v, f0);
    f1 = fma(m_3_0_1, v, f1);
    f2 = fma(m_3_1_0, v, f2);
  }
  { const T v = -Lc[40];
    f0 = fma(m_2_0_2, v, f0);
    f2 = fma(m_3_0_1, v, f2);
  }
  { const T v = -Lc[41];
    f0 = fma(m_1_3_0, v, f0);
    f1 = fma(m_2_2_0, v, f1);
  }
  { const T v = -Lc[42];
    f0 = fma(m_1_2_1, v, f0);
    f1 = fma(m_2_1_1, v, f1);
    f2 = fma(m_2_2_0, v, f2);
  }
  { const T v = -Lc[43];
    f0 = fma(m_1_1_2, v, f0);
    f1 = fma(m_2_0_2, v, f1);
    f2 = fma(m_2_1_1, v, f2);
  }
  { const T v = -Lc[44];
    f0 = fma(m_1_0_3, v, f0);
    f2 = fma(m_2_0_2, v, f2);
  }
  { const T v = -Lc[45];
    f0 = fma(py4, v, f0);
    f1 = fma(m_1_3_0, v, f1);
  }
  { const T v = -Lc[46];
    f0 = fma(m_0_3_1, v, f0);
    f1 = fma(m_1_2_1, v, f1);
    f2 = fma(m_1_3_0, v, f2);
  }
  { const T v = -Lc[47];
    f0 = fma(m_0_2_2, v, f0);
    f1 = fma(m_1_1_2, v, f1);
    f2 = fma(m_1_2_1, v, f2);
  }
  { const T v = -Lc[48];
    f0 = fma(m_0_1_3, v, f0);
    f1 = fma(m_1_0_3, v, f1);
    f2 = fma(m_1_1_2, v, f2);
  }
  { const T v = -Lc[49];
    f0 = fma(pz4, v, f0);
    f2 = fma(m_1_0_3, v, f2);
  }
  { const T v = -Lc[50];
    f1 = fma(py4, v, f1);
  }
  { const T v = -Lc[51];
    f1 = fma(m_0_3_1, v, f1);
    f2 = fma(py4, v, f2);
  }
  { const T v = -Lc[52];
    f1 = fma(m_0_2_2, v, f1);
    f2 = fma(m_0_3_1, v, f2);
  }
  { const T v = -Lc[53];
    f1 = fma(m_0_1_3, v, f1);
    f2 = fma(m_0_2_2, v, f2);
  }
  { const T v = -Lc[54];
    f1 = fma(pz4, v, f1);
    f2 = fma(m_0_1_3, v, f2);
  }
  { const T v = -Lc[55];
    f2 = fma(pz4, v, f2);
  }
}

#define CPPE_M2L_REDUCED(X) \
  X(1, 5, m1_p5, 46, 25, 35, 4, 3, 35) \
  X(1, 6, m1_p6, 64, 36, 48, 6, 3, 56) \
  X(0, 5, m0_p5, 46, 36, 36, 4, 3, 56) \
  X(0, 6, m0_p6, 64, 49, 49, 6, 4, 84) \
  X(2, 5, m2_p5, 46, 16, 32, 4, 2, 20) \
  X(2, 6, m2_p6, 64, 25, 45, 6, 3, 35)

#define CPPE_SHIFTS_GENERATED(X) \
  X(1, 5, 35, 55) \
  X(1, 6, 56, 83)
