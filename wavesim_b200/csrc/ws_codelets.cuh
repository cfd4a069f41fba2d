// Generated by gen_codelets.py - do not edit by hand.
// Small in-register DFTs: Dft<R, INV>::run(v) transforms v[0..R) in place,
// natural order, sign -1 (forward) or +1 (inverse, unnormalised).
#pragma once
#include <cuda_runtime.h>

namespace ws {

template <int R, bool INV> struct Dft;
template <bool INV> struct Dft<1, INV> { static __host__ __device__ __forceinline__ void run(float2 (&)[1]) {} };

template <> struct Dft<2, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[2]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = t1 + t3; const float t6 = t2 + t4;
    const float t7 = t1 - t3; const float t8 = t2 - t4;
    v[0] = make_float2(t5, t6);
    v[1] = make_float2(t7, t8);
  }
};

template <> struct Dft<2, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[2]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = t1 + t3; const float t6 = t2 + t4;
    const float t7 = t1 - t3; const float t8 = t2 - t4;
    v[0] = make_float2(t5, t6);
    v[1] = make_float2(t7, t8);
  }
};

template <> struct Dft<3, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[3]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = t3 + t5; const float t8 = t4 + t6;
    const float t9 = t3 - t5; const float t10 = t4 - t6;
    const float t11 = t1 + t7; const float t12 = t2 + t8;
    const float t13 = fmaf(t7, -0.49999999999999978f, t1); const float t14 = fmaf(t8, -0.49999999999999978f, t2);
    const float t15 = t9 * 0.86602540378443871f; const float t16 = t10 * 0.86602540378443871f;
    const float t17 = t13 + t16; const float t18 = t14 - t15;
    const float t19 = t13 - t16; const float t20 = t14 + t15;
    v[0] = make_float2(t11, t12);
    v[1] = make_float2(t17, t18);
    v[2] = make_float2(t19, t20);
  }
};

template <> struct Dft<3, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[3]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = t3 + t5; const float t8 = t4 + t6;
    const float t9 = t3 - t5; const float t10 = t4 - t6;
    const float t11 = t1 + t7; const float t12 = t2 + t8;
    const float t13 = fmaf(t7, -0.49999999999999978f, t1); const float t14 = fmaf(t8, -0.49999999999999978f, t2);
    const float t15 = t9 * 0.86602540378443871f; const float t16 = t10 * 0.86602540378443871f;
    const float t17 = t13 - t16; const float t18 = t14 + t15;
    const float t19 = t13 + t16; const float t20 = t14 - t15;
    v[0] = make_float2(t11, t12);
    v[1] = make_float2(t17, t18);
    v[2] = make_float2(t19, t20);
  }
};

template <> struct Dft<4, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[4]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = t1 + t5; const float t10 = t2 + t6;
    const float t11 = t1 - t5; const float t12 = t2 - t6;
    const float t13 = t3 + t7; const float t14 = t4 + t8;
    const float t15 = t3 - t7; const float t16 = t4 - t8;
    const float t17 = t16; const float t18 = -t15;
    const float t19 = t9 + t13; const float t20 = t10 + t14;
    const float t21 = t11 + t17; const float t22 = t12 + t18;
    const float t23 = t9 - t13; const float t24 = t10 - t14;
    const float t25 = t11 - t17; const float t26 = t12 - t18;
    v[0] = make_float2(t19, t20);
    v[1] = make_float2(t21, t22);
    v[2] = make_float2(t23, t24);
    v[3] = make_float2(t25, t26);
  }
};

template <> struct Dft<4, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[4]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = t1 + t5; const float t10 = t2 + t6;
    const float t11 = t1 - t5; const float t12 = t2 - t6;
    const float t13 = t3 + t7; const float t14 = t4 + t8;
    const float t15 = t3 - t7; const float t16 = t4 - t8;
    const float t17 = -t16; const float t18 = t15;
    const float t19 = t9 + t13; const float t20 = t10 + t14;
    const float t21 = t11 + t17; const float t22 = t12 + t18;
    const float t23 = t9 - t13; const float t24 = t10 - t14;
    const float t25 = t11 - t17; const float t26 = t12 - t18;
    v[0] = make_float2(t19, t20);
    v[1] = make_float2(t21, t22);
    v[2] = make_float2(t23, t24);
    v[3] = make_float2(t25, t26);
  }
};

template <> struct Dft<5, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[5]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = t3 + t9; const float t12 = t4 + t10;
    const float t13 = t5 + t7; const float t14 = t6 + t8;
    const float t15 = t3 - t9; const float t16 = t4 - t10;
    const float t17 = t5 - t7; const float t18 = t6 - t8;
    const float t19 = t1 + t11 + t13; const float t20 = t2 + t12 + t14;
    const float t21 = fmaf(t13, -0.80901699437494734f, fmaf(t11, 0.30901699437494745f, t1)); const float t22 = fmaf(t14, -0.80901699437494734f, fmaf(t12, 0.30901699437494745f, t2));
    const float t23 = fmaf(t17, 0.58778525229247325f, t15 * 0.95105651629515353f); const float t24 = fmaf(t18, 0.58778525229247325f, t16 * 0.95105651629515353f);
    const float t25 = t21 + t24; const float t26 = t22 - t23;
    const float t27 = t21 - t24; const float t28 = t22 + t23;
    const float t29 = fmaf(t13, 0.30901699437494723f, fmaf(t11, -0.80901699437494734f, t1)); const float t30 = fmaf(t14, 0.30901699437494723f, fmaf(t12, -0.80901699437494734f, t2));
    const float t31 = fmaf(t17, -0.95105651629515364f, t15 * 0.58778525229247325f); const float t32 = fmaf(t18, -0.95105651629515364f, t16 * 0.58778525229247325f);
    const float t33 = t29 + t32; const float t34 = t30 - t31;
    const float t35 = t29 - t32; const float t36 = t30 + t31;
    v[0] = make_float2(t19, t20);
    v[1] = make_float2(t25, t26);
    v[2] = make_float2(t33, t34);
    v[3] = make_float2(t35, t36);
    v[4] = make_float2(t27, t28);
  }
};

template <> struct Dft<5, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[5]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = t3 + t9; const float t12 = t4 + t10;
    const float t13 = t5 + t7; const float t14 = t6 + t8;
    const float t15 = t3 - t9; const float t16 = t4 - t10;
    const float t17 = t5 - t7; const float t18 = t6 - t8;
    const float t19 = t1 + t11 + t13; const float t20 = t2 + t12 + t14;
    const float t21 = fmaf(t13, -0.80901699437494734f, fmaf(t11, 0.30901699437494745f, t1)); const float t22 = fmaf(t14, -0.80901699437494734f, fmaf(t12, 0.30901699437494745f, t2));
    const float t23 = fmaf(t17, 0.58778525229247325f, t15 * 0.95105651629515353f); const float t24 = fmaf(t18, 0.58778525229247325f, t16 * 0.95105651629515353f);
    const float t25 = t21 - t24; const float t26 = t22 + t23;
    const float t27 = t21 + t24; const float t28 = t22 - t23;
    const float t29 = fmaf(t13, 0.30901699437494723f, fmaf(t11, -0.80901699437494734f, t1)); const float t30 = fmaf(t14, 0.30901699437494723f, fmaf(t12, -0.80901699437494734f, t2));
    const float t31 = fmaf(t17, -0.95105651629515364f, t15 * 0.58778525229247325f); const float t32 = fmaf(t18, -0.95105651629515364f, t16 * 0.58778525229247325f);
    const float t33 = t29 - t32; const float t34 = t30 + t31;
    const float t35 = t29 + t32; const float t36 = t30 - t31;
    v[0] = make_float2(t19, t20);
    v[1] = make_float2(t25, t26);
    v[2] = make_float2(t33, t34);
    v[3] = make_float2(t35, t36);
    v[4] = make_float2(t27, t28);
  }
};

template <> struct Dft<6, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[6]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = t1 + t7; const float t14 = t2 + t8;
    const float t15 = t1 - t7; const float t16 = t2 - t8;
    const float t17 = t3 + t9; const float t18 = t4 + t10;
    const float t19 = t3 - t9; const float t20 = t4 - t10;
    const float t21 = fmaf(t19, 0.50000000000000011f, -t20 * -0.8660254037844386f); const float t22 = fmaf(t19, -0.8660254037844386f, t20 * 0.50000000000000011f);
    const float t23 = t5 + t11; const float t24 = t6 + t12;
    const float t25 = t5 - t11; const float t26 = t6 - t12;
    const float t27 = fmaf(t25, -0.49999999999999978f, -t26 * -0.86602540378443871f); const float t28 = fmaf(t25, -0.86602540378443871f, t26 * -0.49999999999999978f);
    const float t29 = t17 + t23; const float t30 = t18 + t24;
    const float t31 = t17 - t23; const float t32 = t18 - t24;
    const float t33 = t13 + t29; const float t34 = t14 + t30;
    const float t35 = fmaf(t29, -0.49999999999999978f, t13); const float t36 = fmaf(t30, -0.49999999999999978f, t14);
    const float t37 = t31 * 0.86602540378443871f; const float t38 = t32 * 0.86602540378443871f;
    const float t39 = t35 + t38; const float t40 = t36 - t37;
    const float t41 = t35 - t38; const float t42 = t36 + t37;
    const float t43 = t21 + t27; const float t44 = t22 + t28;
    const float t45 = t21 - t27; const float t46 = t22 - t28;
    const float t47 = t15 + t43; const float t48 = t16 + t44;
    const float t49 = fmaf(t43, -0.49999999999999978f, t15); const float t50 = fmaf(t44, -0.49999999999999978f, t16);
    const float t51 = t45 * 0.86602540378443871f; const float t52 = t46 * 0.86602540378443871f;
    const float t53 = t49 + t52; const float t54 = t50 - t51;
    const float t55 = t49 - t52; const float t56 = t50 + t51;
    v[0] = make_float2(t33, t34);
    v[1] = make_float2(t47, t48);
    v[2] = make_float2(t39, t40);
    v[3] = make_float2(t53, t54);
    v[4] = make_float2(t41, t42);
    v[5] = make_float2(t55, t56);
  }
};

template <> struct Dft<6, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[6]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = t1 + t7; const float t14 = t2 + t8;
    const float t15 = t1 - t7; const float t16 = t2 - t8;
    const float t17 = t3 + t9; const float t18 = t4 + t10;
    const float t19 = t3 - t9; const float t20 = t4 - t10;
    const float t21 = fmaf(t19, 0.50000000000000011f, -t20 * 0.8660254037844386f); const float t22 = fmaf(t19, 0.8660254037844386f, t20 * 0.50000000000000011f);
    const float t23 = t5 + t11; const float t24 = t6 + t12;
    const float t25 = t5 - t11; const float t26 = t6 - t12;
    const float t27 = fmaf(t25, -0.49999999999999978f, -t26 * 0.86602540378443871f); const float t28 = fmaf(t25, 0.86602540378443871f, t26 * -0.49999999999999978f);
    const float t29 = t17 + t23; const float t30 = t18 + t24;
    const float t31 = t17 - t23; const float t32 = t18 - t24;
    const float t33 = t13 + t29; const float t34 = t14 + t30;
    const float t35 = fmaf(t29, -0.49999999999999978f, t13); const float t36 = fmaf(t30, -0.49999999999999978f, t14);
    const float t37 = t31 * 0.86602540378443871f; const float t38 = t32 * 0.86602540378443871f;
    const float t39 = t35 - t38; const float t40 = t36 + t37;
    const float t41 = t35 + t38; const float t42 = t36 - t37;
    const float t43 = t21 + t27; const float t44 = t22 + t28;
    const float t45 = t21 - t27; const float t46 = t22 - t28;
    const float t47 = t15 + t43; const float t48 = t16 + t44;
    const float t49 = fmaf(t43, -0.49999999999999978f, t15); const float t50 = fmaf(t44, -0.49999999999999978f, t16);
    const float t51 = t45 * 0.86602540378443871f; const float t52 = t46 * 0.86602540378443871f;
    const float t53 = t49 - t52; const float t54 = t50 + t51;
    const float t55 = t49 + t52; const float t56 = t50 - t51;
    v[0] = make_float2(t33, t34);
    v[1] = make_float2(t47, t48);
    v[2] = make_float2(t39, t40);
    v[3] = make_float2(t53, t54);
    v[4] = make_float2(t41, t42);
    v[5] = make_float2(t55, t56);
  }
};

template <> struct Dft<7, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[7]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = t3 + t13; const float t16 = t4 + t14;
    const float t17 = t5 + t11; const float t18 = t6 + t12;
    const float t19 = t7 + t9; const float t20 = t8 + t10;
    const float t21 = t3 - t13; const float t22 = t4 - t14;
    const float t23 = t5 - t11; const float t24 = t6 - t12;
    const float t25 = t7 - t9; const float t26 = t8 - t10;
    const float t27 = t1 + t15 + t17 + t19; const float t28 = t2 + t16 + t18 + t20;
    const float t29 = fmaf(t19, -0.90096886790241903f, fmaf(t17, -0.22252093395631434f, fmaf(t15, 0.62348980185873359f, t1))); const float t30 = fmaf(t20, -0.90096886790241903f, fmaf(t18, -0.22252093395631434f, fmaf(t16, 0.62348980185873359f, t2)));
    const float t31 = fmaf(t25, 0.43388373911755823f, fmaf(t23, 0.97492791218182362f, t21 * 0.7818314824680298f)); const float t32 = fmaf(t26, 0.43388373911755823f, fmaf(t24, 0.97492791218182362f, t22 * 0.7818314824680298f));
    const float t33 = t29 + t32; const float t34 = t30 - t31;
    const float t35 = t29 - t32; const float t36 = t30 + t31;
    const float t37 = fmaf(t19, 0.62348980185873337f, fmaf(t17, -0.90096886790241915f, fmaf(t15, -0.22252093395631434f, t1))); const float t38 = fmaf(t20, 0.62348980185873337f, fmaf(t18, -0.90096886790241915f, fmaf(t16, -0.22252093395631434f, t2)));
    const float t39 = fmaf(t25, -0.78183148246802991f, fmaf(t23, -0.43388373911755801f, t21 * 0.97492791218182362f)); const float t40 = fmaf(t26, -0.78183148246802991f, fmaf(t24, -0.43388373911755801f, t22 * 0.97492791218182362f));
    const float t41 = t37 + t40; const float t42 = t38 - t39;
    const float t43 = t37 - t40; const float t44 = t38 + t39;
    const float t45 = fmaf(t19, -0.22252093395631409f, fmaf(t17, 0.62348980185873337f, fmaf(t15, -0.90096886790241903f, t1))); const float t46 = fmaf(t20, -0.22252093395631409f, fmaf(t18, 0.62348980185873337f, fmaf(t16, -0.90096886790241903f, t2)));
    const float t47 = fmaf(t25, 0.97492791218182373f, fmaf(t23, -0.78183148246802991f, t21 * 0.43388373911755823f)); const float t48 = fmaf(t26, 0.97492791218182373f, fmaf(t24, -0.78183148246802991f, t22 * 0.43388373911755823f));
    const float t49 = t45 + t48; const float t50 = t46 - t47;
    const float t51 = t45 - t48; const float t52 = t46 + t47;
    v[0] = make_float2(t27, t28);
    v[1] = make_float2(t33, t34);
    v[2] = make_float2(t41, t42);
    v[3] = make_float2(t49, t50);
    v[4] = make_float2(t51, t52);
    v[5] = make_float2(t43, t44);
    v[6] = make_float2(t35, t36);
  }
};

template <> struct Dft<7, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[7]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = t3 + t13; const float t16 = t4 + t14;
    const float t17 = t5 + t11; const float t18 = t6 + t12;
    const float t19 = t7 + t9; const float t20 = t8 + t10;
    const float t21 = t3 - t13; const float t22 = t4 - t14;
    const float t23 = t5 - t11; const float t24 = t6 - t12;
    const float t25 = t7 - t9; const float t26 = t8 - t10;
    const float t27 = t1 + t15 + t17 + t19; const float t28 = t2 + t16 + t18 + t20;
    const float t29 = fmaf(t19, -0.90096886790241903f, fmaf(t17, -0.22252093395631434f, fmaf(t15, 0.62348980185873359f, t1))); const float t30 = fmaf(t20, -0.90096886790241903f, fmaf(t18, -0.22252093395631434f, fmaf(t16, 0.62348980185873359f, t2)));
    const float t31 = fmaf(t25, 0.43388373911755823f, fmaf(t23, 0.97492791218182362f, t21 * 0.7818314824680298f)); const float t32 = fmaf(t26, 0.43388373911755823f, fmaf(t24, 0.97492791218182362f, t22 * 0.7818314824680298f));
    const float t33 = t29 - t32; const float t34 = t30 + t31;
    const float t35 = t29 + t32; const float t36 = t30 - t31;
    const float t37 = fmaf(t19, 0.62348980185873337f, fmaf(t17, -0.90096886790241915f, fmaf(t15, -0.22252093395631434f, t1))); const float t38 = fmaf(t20, 0.62348980185873337f, fmaf(t18, -0.90096886790241915f, fmaf(t16, -0.22252093395631434f, t2)));
    const float t39 = fmaf(t25, -0.78183148246802991f, fmaf(t23, -0.43388373911755801f, t21 * 0.97492791218182362f)); const float t40 = fmaf(t26, -0.78183148246802991f, fmaf(t24, -0.43388373911755801f, t22 * 0.97492791218182362f));
    const float t41 = t37 - t40; const float t42 = t38 + t39;
    const float t43 = t37 + t40; const float t44 = t38 - t39;
    const float t45 = fmaf(t19, -0.22252093395631409f, fmaf(t17, 0.62348980185873337f, fmaf(t15, -0.90096886790241903f, t1))); const float t46 = fmaf(t20, -0.22252093395631409f, fmaf(t18, 0.62348980185873337f, fmaf(t16, -0.90096886790241903f, t2)));
    const float t47 = fmaf(t25, 0.97492791218182373f, fmaf(t23, -0.78183148246802991f, t21 * 0.43388373911755823f)); const float t48 = fmaf(t26, 0.97492791218182373f, fmaf(t24, -0.78183148246802991f, t22 * 0.43388373911755823f));
    const float t49 = t45 - t48; const float t50 = t46 + t47;
    const float t51 = t45 + t48; const float t52 = t46 - t47;
    v[0] = make_float2(t27, t28);
    v[1] = make_float2(t33, t34);
    v[2] = make_float2(t41, t42);
    v[3] = make_float2(t49, t50);
    v[4] = make_float2(t51, t52);
    v[5] = make_float2(t43, t44);
    v[6] = make_float2(t35, t36);
  }
};

template <> struct Dft<8, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[8]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = t1 + t9; const float t18 = t2 + t10;
    const float t19 = t1 - t9; const float t20 = t2 - t10;
    const float t21 = t5 + t13; const float t22 = t6 + t14;
    const float t23 = t5 - t13; const float t24 = t6 - t14;
    const float t25 = t24; const float t26 = -t23;
    const float t27 = t17 + t21; const float t28 = t18 + t22;
    const float t29 = t17 - t21; const float t30 = t18 - t22;
    const float t31 = t19 + t25; const float t32 = t20 + t26;
    const float t33 = t19 - t25; const float t34 = t20 - t26;
    const float t35 = t3 + t11; const float t36 = t4 + t12;
    const float t37 = t3 - t11; const float t38 = t4 - t12;
    const float t39 = t7 + t15; const float t40 = t8 + t16;
    const float t41 = t7 - t15; const float t42 = t8 - t16;
    const float t43 = t42; const float t44 = -t41;
    const float t45 = t35 + t39; const float t46 = t36 + t40;
    const float t47 = t35 - t39; const float t48 = t36 - t40;
    const float t49 = t37 + t43; const float t50 = t38 + t44;
    const float t51 = t37 - t43; const float t52 = t38 - t44;
    const float t53 = 0.70710678118654752f * (t49 + t50); const float t54 = 0.70710678118654752f * (t50 - t49);
    const float t55 = t48; const float t56 = -t47;
    const float t57 = 0.70710678118654752f * (t52 - t51); const float t58 = -0.70710678118654752f * (t51 + t52);
    const float t59 = t27 + t45; const float t60 = t28 + t46;
    const float t61 = t27 - t45; const float t62 = t28 - t46;
    const float t63 = t31 + t53; const float t64 = t32 + t54;
    const float t65 = t31 - t53; const float t66 = t32 - t54;
    const float t67 = t29 + t55; const float t68 = t30 + t56;
    const float t69 = t29 - t55; const float t70 = t30 - t56;
    const float t71 = t33 + t57; const float t72 = t34 + t58;
    const float t73 = t33 - t57; const float t74 = t34 - t58;
    v[0] = make_float2(t59, t60);
    v[1] = make_float2(t63, t64);
    v[2] = make_float2(t67, t68);
    v[3] = make_float2(t71, t72);
    v[4] = make_float2(t61, t62);
    v[5] = make_float2(t65, t66);
    v[6] = make_float2(t69, t70);
    v[7] = make_float2(t73, t74);
  }
};

template <> struct Dft<8, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[8]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = t1 + t9; const float t18 = t2 + t10;
    const float t19 = t1 - t9; const float t20 = t2 - t10;
    const float t21 = t5 + t13; const float t22 = t6 + t14;
    const float t23 = t5 - t13; const float t24 = t6 - t14;
    const float t25 = -t24; const float t26 = t23;
    const float t27 = t17 + t21; const float t28 = t18 + t22;
    const float t29 = t17 - t21; const float t30 = t18 - t22;
    const float t31 = t19 + t25; const float t32 = t20 + t26;
    const float t33 = t19 - t25; const float t34 = t20 - t26;
    const float t35 = t3 + t11; const float t36 = t4 + t12;
    const float t37 = t3 - t11; const float t38 = t4 - t12;
    const float t39 = t7 + t15; const float t40 = t8 + t16;
    const float t41 = t7 - t15; const float t42 = t8 - t16;
    const float t43 = -t42; const float t44 = t41;
    const float t45 = t35 + t39; const float t46 = t36 + t40;
    const float t47 = t35 - t39; const float t48 = t36 - t40;
    const float t49 = t37 + t43; const float t50 = t38 + t44;
    const float t51 = t37 - t43; const float t52 = t38 - t44;
    const float t53 = 0.70710678118654752f * (t49 - t50); const float t54 = 0.70710678118654752f * (t49 + t50);
    const float t55 = -t48; const float t56 = t47;
    const float t57 = -0.70710678118654752f * (t51 + t52); const float t58 = 0.70710678118654752f * (t51 - t52);
    const float t59 = t27 + t45; const float t60 = t28 + t46;
    const float t61 = t27 - t45; const float t62 = t28 - t46;
    const float t63 = t31 + t53; const float t64 = t32 + t54;
    const float t65 = t31 - t53; const float t66 = t32 - t54;
    const float t67 = t29 + t55; const float t68 = t30 + t56;
    const float t69 = t29 - t55; const float t70 = t30 - t56;
    const float t71 = t33 + t57; const float t72 = t34 + t58;
    const float t73 = t33 - t57; const float t74 = t34 - t58;
    v[0] = make_float2(t59, t60);
    v[1] = make_float2(t63, t64);
    v[2] = make_float2(t67, t68);
    v[3] = make_float2(t71, t72);
    v[4] = make_float2(t61, t62);
    v[5] = make_float2(t65, t66);
    v[6] = make_float2(t69, t70);
    v[7] = make_float2(t73, t74);
  }
};

template <> struct Dft<9, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[9]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = t7 + t13; const float t20 = t8 + t14;
    const float t21 = t7 - t13; const float t22 = t8 - t14;
    const float t23 = t1 + t19; const float t24 = t2 + t20;
    const float t25 = fmaf(t19, -0.49999999999999978f, t1); const float t26 = fmaf(t20, -0.49999999999999978f, t2);
    const float t27 = t21 * 0.86602540378443871f; const float t28 = t22 * 0.86602540378443871f;
    const float t29 = t25 + t28; const float t30 = t26 - t27;
    const float t31 = t25 - t28; const float t32 = t26 + t27;
    const float t33 = t9 + t15; const float t34 = t10 + t16;
    const float t35 = t9 - t15; const float t36 = t10 - t16;
    const float t37 = t3 + t33; const float t38 = t4 + t34;
    const float t39 = fmaf(t33, -0.49999999999999978f, t3); const float t40 = fmaf(t34, -0.49999999999999978f, t4);
    const float t41 = t35 * 0.86602540378443871f; const float t42 = t36 * 0.86602540378443871f;
    const float t43 = t39 + t42; const float t44 = t40 - t41;
    const float t45 = t39 - t42; const float t46 = t40 + t41;
    const float t47 = fmaf(t43, 0.76604444311897801f, -t44 * -0.64278760968653925f); const float t48 = fmaf(t43, -0.64278760968653925f, t44 * 0.76604444311897801f);
    const float t49 = fmaf(t45, 0.17364817766693041f, -t46 * -0.98480775301220802f); const float t50 = fmaf(t45, -0.98480775301220802f, t46 * 0.17364817766693041f);
    const float t51 = t11 + t17; const float t52 = t12 + t18;
    const float t53 = t11 - t17; const float t54 = t12 - t18;
    const float t55 = t5 + t51; const float t56 = t6 + t52;
    const float t57 = fmaf(t51, -0.49999999999999978f, t5); const float t58 = fmaf(t52, -0.49999999999999978f, t6);
    const float t59 = t53 * 0.86602540378443871f; const float t60 = t54 * 0.86602540378443871f;
    const float t61 = t57 + t60; const float t62 = t58 - t59;
    const float t63 = t57 - t60; const float t64 = t58 + t59;
    const float t65 = fmaf(t61, 0.17364817766693041f, -t62 * -0.98480775301220802f); const float t66 = fmaf(t61, -0.98480775301220802f, t62 * 0.17364817766693041f);
    const float t67 = fmaf(t63, -0.93969262078590832f, -t64 * -0.34202014332566888f); const float t68 = fmaf(t63, -0.34202014332566888f, t64 * -0.93969262078590832f);
    const float t69 = t37 + t55; const float t70 = t38 + t56;
    const float t71 = t37 - t55; const float t72 = t38 - t56;
    const float t73 = t23 + t69; const float t74 = t24 + t70;
    const float t75 = fmaf(t69, -0.49999999999999978f, t23); const float t76 = fmaf(t70, -0.49999999999999978f, t24);
    const float t77 = t71 * 0.86602540378443871f; const float t78 = t72 * 0.86602540378443871f;
    const float t79 = t75 + t78; const float t80 = t76 - t77;
    const float t81 = t75 - t78; const float t82 = t76 + t77;
    const float t83 = t47 + t65; const float t84 = t48 + t66;
    const float t85 = t47 - t65; const float t86 = t48 - t66;
    const float t87 = t29 + t83; const float t88 = t30 + t84;
    const float t89 = fmaf(t83, -0.49999999999999978f, t29); const float t90 = fmaf(t84, -0.49999999999999978f, t30);
    const float t91 = t85 * 0.86602540378443871f; const float t92 = t86 * 0.86602540378443871f;
    const float t93 = t89 + t92; const float t94 = t90 - t91;
    const float t95 = t89 - t92; const float t96 = t90 + t91;
    const float t97 = t49 + t67; const float t98 = t50 + t68;
    const float t99 = t49 - t67; const float t100 = t50 - t68;
    const float t101 = t31 + t97; const float t102 = t32 + t98;
    const float t103 = fmaf(t97, -0.49999999999999978f, t31); const float t104 = fmaf(t98, -0.49999999999999978f, t32);
    const float t105 = t99 * 0.86602540378443871f; const float t106 = t100 * 0.86602540378443871f;
    const float t107 = t103 + t106; const float t108 = t104 - t105;
    const float t109 = t103 - t106; const float t110 = t104 + t105;
    v[0] = make_float2(t73, t74);
    v[1] = make_float2(t87, t88);
    v[2] = make_float2(t101, t102);
    v[3] = make_float2(t79, t80);
    v[4] = make_float2(t93, t94);
    v[5] = make_float2(t107, t108);
    v[6] = make_float2(t81, t82);
    v[7] = make_float2(t95, t96);
    v[8] = make_float2(t109, t110);
  }
};

template <> struct Dft<9, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[9]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = t7 + t13; const float t20 = t8 + t14;
    const float t21 = t7 - t13; const float t22 = t8 - t14;
    const float t23 = t1 + t19; const float t24 = t2 + t20;
    const float t25 = fmaf(t19, -0.49999999999999978f, t1); const float t26 = fmaf(t20, -0.49999999999999978f, t2);
    const float t27 = t21 * 0.86602540378443871f; const float t28 = t22 * 0.86602540378443871f;
    const float t29 = t25 - t28; const float t30 = t26 + t27;
    const float t31 = t25 + t28; const float t32 = t26 - t27;
    const float t33 = t9 + t15; const float t34 = t10 + t16;
    const float t35 = t9 - t15; const float t36 = t10 - t16;
    const float t37 = t3 + t33; const float t38 = t4 + t34;
    const float t39 = fmaf(t33, -0.49999999999999978f, t3); const float t40 = fmaf(t34, -0.49999999999999978f, t4);
    const float t41 = t35 * 0.86602540378443871f; const float t42 = t36 * 0.86602540378443871f;
    const float t43 = t39 - t42; const float t44 = t40 + t41;
    const float t45 = t39 + t42; const float t46 = t40 - t41;
    const float t47 = fmaf(t43, 0.76604444311897801f, -t44 * 0.64278760968653925f); const float t48 = fmaf(t43, 0.64278760968653925f, t44 * 0.76604444311897801f);
    const float t49 = fmaf(t45, 0.17364817766693041f, -t46 * 0.98480775301220802f); const float t50 = fmaf(t45, 0.98480775301220802f, t46 * 0.17364817766693041f);
    const float t51 = t11 + t17; const float t52 = t12 + t18;
    const float t53 = t11 - t17; const float t54 = t12 - t18;
    const float t55 = t5 + t51; const float t56 = t6 + t52;
    const float t57 = fmaf(t51, -0.49999999999999978f, t5); const float t58 = fmaf(t52, -0.49999999999999978f, t6);
    const float t59 = t53 * 0.86602540378443871f; const float t60 = t54 * 0.86602540378443871f;
    const float t61 = t57 - t60; const float t62 = t58 + t59;
    const float t63 = t57 + t60; const float t64 = t58 - t59;
    const float t65 = fmaf(t61, 0.17364817766693041f, -t62 * 0.98480775301220802f); const float t66 = fmaf(t61, 0.98480775301220802f, t62 * 0.17364817766693041f);
    const float t67 = fmaf(t63, -0.93969262078590832f, -t64 * 0.34202014332566888f); const float t68 = fmaf(t63, 0.34202014332566888f, t64 * -0.93969262078590832f);
    const float t69 = t37 + t55; const float t70 = t38 + t56;
    const float t71 = t37 - t55; const float t72 = t38 - t56;
    const float t73 = t23 + t69; const float t74 = t24 + t70;
    const float t75 = fmaf(t69, -0.49999999999999978f, t23); const float t76 = fmaf(t70, -0.49999999999999978f, t24);
    const float t77 = t71 * 0.86602540378443871f; const float t78 = t72 * 0.86602540378443871f;
    const float t79 = t75 - t78; const float t80 = t76 + t77;
    const float t81 = t75 + t78; const float t82 = t76 - t77;
    const float t83 = t47 + t65; const float t84 = t48 + t66;
    const float t85 = t47 - t65; const float t86 = t48 - t66;
    const float t87 = t29 + t83; const float t88 = t30 + t84;
    const float t89 = fmaf(t83, -0.49999999999999978f, t29); const float t90 = fmaf(t84, -0.49999999999999978f, t30);
    const float t91 = t85 * 0.86602540378443871f; const float t92 = t86 * 0.86602540378443871f;
    const float t93 = t89 - t92; const float t94 = t90 + t91;
    const float t95 = t89 + t92; const float t96 = t90 - t91;
    const float t97 = t49 + t67; const float t98 = t50 + t68;
    const float t99 = t49 - t67; const float t100 = t50 - t68;
    const float t101 = t31 + t97; const float t102 = t32 + t98;
    const float t103 = fmaf(t97, -0.49999999999999978f, t31); const float t104 = fmaf(t98, -0.49999999999999978f, t32);
    const float t105 = t99 * 0.86602540378443871f; const float t106 = t100 * 0.86602540378443871f;
    const float t107 = t103 - t106; const float t108 = t104 + t105;
    const float t109 = t103 + t106; const float t110 = t104 - t105;
    v[0] = make_float2(t73, t74);
    v[1] = make_float2(t87, t88);
    v[2] = make_float2(t101, t102);
    v[3] = make_float2(t79, t80);
    v[4] = make_float2(t93, t94);
    v[5] = make_float2(t107, t108);
    v[6] = make_float2(t81, t82);
    v[7] = make_float2(t95, t96);
    v[8] = make_float2(t109, t110);
  }
};

template <> struct Dft<10, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[10]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = t1 + t11; const float t22 = t2 + t12;
    const float t23 = t1 - t11; const float t24 = t2 - t12;
    const float t25 = t3 + t13; const float t26 = t4 + t14;
    const float t27 = t3 - t13; const float t28 = t4 - t14;
    const float t29 = fmaf(t27, 0.80901699437494745f, -t28 * -0.58778525229247314f); const float t30 = fmaf(t27, -0.58778525229247314f, t28 * 0.80901699437494745f);
    const float t31 = t5 + t15; const float t32 = t6 + t16;
    const float t33 = t5 - t15; const float t34 = t6 - t16;
    const float t35 = fmaf(t33, 0.30901699437494745f, -t34 * -0.95105651629515353f); const float t36 = fmaf(t33, -0.95105651629515353f, t34 * 0.30901699437494745f);
    const float t37 = t7 + t17; const float t38 = t8 + t18;
    const float t39 = t7 - t17; const float t40 = t8 - t18;
    const float t41 = fmaf(t39, -0.30901699437494734f, -t40 * -0.95105651629515364f); const float t42 = fmaf(t39, -0.95105651629515364f, t40 * -0.30901699437494734f);
    const float t43 = t9 + t19; const float t44 = t10 + t20;
    const float t45 = t9 - t19; const float t46 = t10 - t20;
    const float t47 = fmaf(t45, -0.80901699437494734f, -t46 * -0.58778525229247325f); const float t48 = fmaf(t45, -0.58778525229247325f, t46 * -0.80901699437494734f);
    const float t49 = t25 + t43; const float t50 = t26 + t44;
    const float t51 = t31 + t37; const float t52 = t32 + t38;
    const float t53 = t25 - t43; const float t54 = t26 - t44;
    const float t55 = t31 - t37; const float t56 = t32 - t38;
    const float t57 = t21 + t49 + t51; const float t58 = t22 + t50 + t52;
    const float t59 = fmaf(t51, -0.80901699437494734f, fmaf(t49, 0.30901699437494745f, t21)); const float t60 = fmaf(t52, -0.80901699437494734f, fmaf(t50, 0.30901699437494745f, t22));
    const float t61 = fmaf(t55, 0.58778525229247325f, t53 * 0.95105651629515353f); const float t62 = fmaf(t56, 0.58778525229247325f, t54 * 0.95105651629515353f);
    const float t63 = t59 + t62; const float t64 = t60 - t61;
    const float t65 = t59 - t62; const float t66 = t60 + t61;
    const float t67 = fmaf(t51, 0.30901699437494723f, fmaf(t49, -0.80901699437494734f, t21)); const float t68 = fmaf(t52, 0.30901699437494723f, fmaf(t50, -0.80901699437494734f, t22));
    const float t69 = fmaf(t55, -0.95105651629515364f, t53 * 0.58778525229247325f); const float t70 = fmaf(t56, -0.95105651629515364f, t54 * 0.58778525229247325f);
    const float t71 = t67 + t70; const float t72 = t68 - t69;
    const float t73 = t67 - t70; const float t74 = t68 + t69;
    const float t75 = t29 + t47; const float t76 = t30 + t48;
    const float t77 = t35 + t41; const float t78 = t36 + t42;
    const float t79 = t29 - t47; const float t80 = t30 - t48;
    const float t81 = t35 - t41; const float t82 = t36 - t42;
    const float t83 = t23 + t75 + t77; const float t84 = t24 + t76 + t78;
    const float t85 = fmaf(t77, -0.80901699437494734f, fmaf(t75, 0.30901699437494745f, t23)); const float t86 = fmaf(t78, -0.80901699437494734f, fmaf(t76, 0.30901699437494745f, t24));
    const float t87 = fmaf(t81, 0.58778525229247325f, t79 * 0.95105651629515353f); const float t88 = fmaf(t82, 0.58778525229247325f, t80 * 0.95105651629515353f);
    const float t89 = t85 + t88; const float t90 = t86 - t87;
    const float t91 = t85 - t88; const float t92 = t86 + t87;
    const float t93 = fmaf(t77, 0.30901699437494723f, fmaf(t75, -0.80901699437494734f, t23)); const float t94 = fmaf(t78, 0.30901699437494723f, fmaf(t76, -0.80901699437494734f, t24));
    const float t95 = fmaf(t81, -0.95105651629515364f, t79 * 0.58778525229247325f); const float t96 = fmaf(t82, -0.95105651629515364f, t80 * 0.58778525229247325f);
    const float t97 = t93 + t96; const float t98 = t94 - t95;
    const float t99 = t93 - t96; const float t100 = t94 + t95;
    v[0] = make_float2(t57, t58);
    v[1] = make_float2(t83, t84);
    v[2] = make_float2(t63, t64);
    v[3] = make_float2(t89, t90);
    v[4] = make_float2(t71, t72);
    v[5] = make_float2(t97, t98);
    v[6] = make_float2(t73, t74);
    v[7] = make_float2(t99, t100);
    v[8] = make_float2(t65, t66);
    v[9] = make_float2(t91, t92);
  }
};

template <> struct Dft<10, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[10]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = t1 + t11; const float t22 = t2 + t12;
    const float t23 = t1 - t11; const float t24 = t2 - t12;
    const float t25 = t3 + t13; const float t26 = t4 + t14;
    const float t27 = t3 - t13; const float t28 = t4 - t14;
    const float t29 = fmaf(t27, 0.80901699437494745f, -t28 * 0.58778525229247314f); const float t30 = fmaf(t27, 0.58778525229247314f, t28 * 0.80901699437494745f);
    const float t31 = t5 + t15; const float t32 = t6 + t16;
    const float t33 = t5 - t15; const float t34 = t6 - t16;
    const float t35 = fmaf(t33, 0.30901699437494745f, -t34 * 0.95105651629515353f); const float t36 = fmaf(t33, 0.95105651629515353f, t34 * 0.30901699437494745f);
    const float t37 = t7 + t17; const float t38 = t8 + t18;
    const float t39 = t7 - t17; const float t40 = t8 - t18;
    const float t41 = fmaf(t39, -0.30901699437494734f, -t40 * 0.95105651629515364f); const float t42 = fmaf(t39, 0.95105651629515364f, t40 * -0.30901699437494734f);
    const float t43 = t9 + t19; const float t44 = t10 + t20;
    const float t45 = t9 - t19; const float t46 = t10 - t20;
    const float t47 = fmaf(t45, -0.80901699437494734f, -t46 * 0.58778525229247325f); const float t48 = fmaf(t45, 0.58778525229247325f, t46 * -0.80901699437494734f);
    const float t49 = t25 + t43; const float t50 = t26 + t44;
    const float t51 = t31 + t37; const float t52 = t32 + t38;
    const float t53 = t25 - t43; const float t54 = t26 - t44;
    const float t55 = t31 - t37; const float t56 = t32 - t38;
    const float t57 = t21 + t49 + t51; const float t58 = t22 + t50 + t52;
    const float t59 = fmaf(t51, -0.80901699437494734f, fmaf(t49, 0.30901699437494745f, t21)); const float t60 = fmaf(t52, -0.80901699437494734f, fmaf(t50, 0.30901699437494745f, t22));
    const float t61 = fmaf(t55, 0.58778525229247325f, t53 * 0.95105651629515353f); const float t62 = fmaf(t56, 0.58778525229247325f, t54 * 0.95105651629515353f);
    const float t63 = t59 - t62; const float t64 = t60 + t61;
    const float t65 = t59 + t62; const float t66 = t60 - t61;
    const float t67 = fmaf(t51, 0.30901699437494723f, fmaf(t49, -0.80901699437494734f, t21)); const float t68 = fmaf(t52, 0.30901699437494723f, fmaf(t50, -0.80901699437494734f, t22));
    const float t69 = fmaf(t55, -0.95105651629515364f, t53 * 0.58778525229247325f); const float t70 = fmaf(t56, -0.95105651629515364f, t54 * 0.58778525229247325f);
    const float t71 = t67 - t70; const float t72 = t68 + t69;
    const float t73 = t67 + t70; const float t74 = t68 - t69;
    const float t75 = t29 + t47; const float t76 = t30 + t48;
    const float t77 = t35 + t41; const float t78 = t36 + t42;
    const float t79 = t29 - t47; const float t80 = t30 - t48;
    const float t81 = t35 - t41; const float t82 = t36 - t42;
    const float t83 = t23 + t75 + t77; const float t84 = t24 + t76 + t78;
    const float t85 = fmaf(t77, -0.80901699437494734f, fmaf(t75, 0.30901699437494745f, t23)); const float t86 = fmaf(t78, -0.80901699437494734f, fmaf(t76, 0.30901699437494745f, t24));
    const float t87 = fmaf(t81, 0.58778525229247325f, t79 * 0.95105651629515353f); const float t88 = fmaf(t82, 0.58778525229247325f, t80 * 0.95105651629515353f);
    const float t89 = t85 - t88; const float t90 = t86 + t87;
    const float t91 = t85 + t88; const float t92 = t86 - t87;
    const float t93 = fmaf(t77, 0.30901699437494723f, fmaf(t75, -0.80901699437494734f, t23)); const float t94 = fmaf(t78, 0.30901699437494723f, fmaf(t76, -0.80901699437494734f, t24));
    const float t95 = fmaf(t81, -0.95105651629515364f, t79 * 0.58778525229247325f); const float t96 = fmaf(t82, -0.95105651629515364f, t80 * 0.58778525229247325f);
    const float t97 = t93 - t96; const float t98 = t94 + t95;
    const float t99 = t93 + t96; const float t100 = t94 - t95;
    v[0] = make_float2(t57, t58);
    v[1] = make_float2(t83, t84);
    v[2] = make_float2(t63, t64);
    v[3] = make_float2(t89, t90);
    v[4] = make_float2(t71, t72);
    v[5] = make_float2(t97, t98);
    v[6] = make_float2(t73, t74);
    v[7] = make_float2(t99, t100);
    v[8] = make_float2(t65, t66);
    v[9] = make_float2(t91, t92);
  }
};

template <> struct Dft<11, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[11]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = t3 + t21; const float t24 = t4 + t22;
    const float t25 = t5 + t19; const float t26 = t6 + t20;
    const float t27 = t7 + t17; const float t28 = t8 + t18;
    const float t29 = t9 + t15; const float t30 = t10 + t16;
    const float t31 = t11 + t13; const float t32 = t12 + t14;
    const float t33 = t3 - t21; const float t34 = t4 - t22;
    const float t35 = t5 - t19; const float t36 = t6 - t20;
    const float t37 = t7 - t17; const float t38 = t8 - t18;
    const float t39 = t9 - t15; const float t40 = t10 - t16;
    const float t41 = t11 - t13; const float t42 = t12 - t14;
    const float t43 = t1 + t23 + t25 + t27 + t29 + t31; const float t44 = t2 + t24 + t26 + t28 + t30 + t32;
    const float t45 = fmaf(t31, -0.95949297361449737f, fmaf(t29, -0.65486073394528499f, fmaf(t27, -0.142314838273285f, fmaf(t25, 0.41541501300188644f, fmaf(t23, 0.84125353283118121f, t1))))); const float t46 = fmaf(t32, -0.95949297361449737f, fmaf(t30, -0.65486073394528499f, fmaf(t28, -0.142314838273285f, fmaf(t26, 0.41541501300188644f, fmaf(t24, 0.84125353283118121f, t2)))));
    const float t47 = fmaf(t41, 0.28173255684142967f, fmaf(t39, 0.75574957435425827f, fmaf(t37, 0.9898214418809328f, fmaf(t35, 0.90963199535451833f, t33 * 0.54064081745559756f)))); const float t48 = fmaf(t42, 0.28173255684142967f, fmaf(t40, 0.75574957435425827f, fmaf(t38, 0.9898214418809328f, fmaf(t36, 0.90963199535451833f, t34 * 0.54064081745559756f))));
    const float t49 = t45 + t48; const float t50 = t46 - t47;
    const float t51 = t45 - t48; const float t52 = t46 + t47;
    const float t53 = fmaf(t31, 0.84125353283118121f, fmaf(t29, -0.14231483827328523f, fmaf(t27, -0.95949297361449748f, fmaf(t25, -0.65486073394528499f, fmaf(t23, 0.41541501300188644f, t1))))); const float t54 = fmaf(t32, 0.84125353283118121f, fmaf(t30, -0.14231483827328523f, fmaf(t28, -0.95949297361449748f, fmaf(t26, -0.65486073394528499f, fmaf(t24, 0.41541501300188644f, t2)))));
    const float t55 = fmaf(t41, -0.54064081745559744f, fmaf(t39, -0.98982144188093268f, fmaf(t37, -0.28173255684142939f, fmaf(t35, 0.75574957435425827f, t33 * 0.90963199535451833f)))); const float t56 = fmaf(t42, -0.54064081745559744f, fmaf(t40, -0.98982144188093268f, fmaf(t38, -0.28173255684142939f, fmaf(t36, 0.75574957435425827f, t34 * 0.90963199535451833f))));
    const float t57 = t53 + t56; const float t58 = t54 - t55;
    const float t59 = t53 - t56; const float t60 = t54 + t55;
    const float t61 = fmaf(t31, -0.65486073394528388f, fmaf(t29, 0.84125353283118154f, fmaf(t27, 0.41541501300188605f, fmaf(t25, -0.95949297361449748f, fmaf(t23, -0.142314838273285f, t1))))); const float t62 = fmaf(t32, -0.65486073394528388f, fmaf(t30, 0.84125353283118154f, fmaf(t28, 0.41541501300188605f, fmaf(t26, -0.95949297361449748f, fmaf(t24, -0.142314838273285f, t2)))));
    const float t63 = fmaf(t41, 0.75574957435425938f, fmaf(t39, 0.54064081745559711f, fmaf(t37, -0.90963199535451855f, fmaf(t35, -0.28173255684142939f, t33 * 0.9898214418809328f)))); const float t64 = fmaf(t42, 0.75574957435425938f, fmaf(t40, 0.54064081745559711f, fmaf(t38, -0.90963199535451855f, fmaf(t36, -0.28173255684142939f, t34 * 0.9898214418809328f))));
    const float t65 = t61 + t64; const float t66 = t62 - t63;
    const float t67 = t61 - t64; const float t68 = t62 + t63;
    const float t69 = fmaf(t31, 0.4154150130018866f, fmaf(t29, -0.95949297361449737f, fmaf(t27, 0.84125353283118154f, fmaf(t25, -0.14231483827328523f, fmaf(t23, -0.65486073394528499f, t1))))); const float t70 = fmaf(t32, 0.4154150130018866f, fmaf(t30, -0.95949297361449737f, fmaf(t28, 0.84125353283118154f, fmaf(t26, -0.14231483827328523f, fmaf(t24, -0.65486073394528499f, t2)))));
    const float t71 = fmaf(t41, -0.90963199535451833f, fmaf(t39, 0.28173255684142989f, fmaf(t37, 0.54064081745559711f, fmaf(t35, -0.98982144188093268f, t33 * 0.75574957435425827f)))); const float t72 = fmaf(t42, -0.90963199535451833f, fmaf(t40, 0.28173255684142989f, fmaf(t38, 0.54064081745559711f, fmaf(t36, -0.98982144188093268f, t34 * 0.75574957435425827f))));
    const float t73 = t69 + t72; const float t74 = t70 - t71;
    const float t75 = t69 - t72; const float t76 = t70 + t71;
    const float t77 = fmaf(t31, -0.14231483827328539f, fmaf(t29, 0.4154150130018866f, fmaf(t27, -0.65486073394528388f, fmaf(t25, 0.84125353283118121f, fmaf(t23, -0.95949297361449737f, t1))))); const float t78 = fmaf(t32, -0.14231483827328539f, fmaf(t30, 0.4154150130018866f, fmaf(t28, -0.65486073394528388f, fmaf(t26, 0.84125353283118121f, fmaf(t24, -0.95949297361449737f, t2)))));
    const float t79 = fmaf(t41, 0.98982144188093268f, fmaf(t39, -0.90963199535451833f, fmaf(t37, 0.75574957435425938f, fmaf(t35, -0.54064081745559744f, t33 * 0.28173255684142967f)))); const float t80 = fmaf(t42, 0.98982144188093268f, fmaf(t40, -0.90963199535451833f, fmaf(t38, 0.75574957435425938f, fmaf(t36, -0.54064081745559744f, t34 * 0.28173255684142967f))));
    const float t81 = t77 + t80; const float t82 = t78 - t79;
    const float t83 = t77 - t80; const float t84 = t78 + t79;
    v[0] = make_float2(t43, t44);
    v[1] = make_float2(t49, t50);
    v[2] = make_float2(t57, t58);
    v[3] = make_float2(t65, t66);
    v[4] = make_float2(t73, t74);
    v[5] = make_float2(t81, t82);
    v[6] = make_float2(t83, t84);
    v[7] = make_float2(t75, t76);
    v[8] = make_float2(t67, t68);
    v[9] = make_float2(t59, t60);
    v[10] = make_float2(t51, t52);
  }
};

template <> struct Dft<11, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[11]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = t3 + t21; const float t24 = t4 + t22;
    const float t25 = t5 + t19; const float t26 = t6 + t20;
    const float t27 = t7 + t17; const float t28 = t8 + t18;
    const float t29 = t9 + t15; const float t30 = t10 + t16;
    const float t31 = t11 + t13; const float t32 = t12 + t14;
    const float t33 = t3 - t21; const float t34 = t4 - t22;
    const float t35 = t5 - t19; const float t36 = t6 - t20;
    const float t37 = t7 - t17; const float t38 = t8 - t18;
    const float t39 = t9 - t15; const float t40 = t10 - t16;
    const float t41 = t11 - t13; const float t42 = t12 - t14;
    const float t43 = t1 + t23 + t25 + t27 + t29 + t31; const float t44 = t2 + t24 + t26 + t28 + t30 + t32;
    const float t45 = fmaf(t31, -0.95949297361449737f, fmaf(t29, -0.65486073394528499f, fmaf(t27, -0.142314838273285f, fmaf(t25, 0.41541501300188644f, fmaf(t23, 0.84125353283118121f, t1))))); const float t46 = fmaf(t32, -0.95949297361449737f, fmaf(t30, -0.65486073394528499f, fmaf(t28, -0.142314838273285f, fmaf(t26, 0.41541501300188644f, fmaf(t24, 0.84125353283118121f, t2)))));
    const float t47 = fmaf(t41, 0.28173255684142967f, fmaf(t39, 0.75574957435425827f, fmaf(t37, 0.9898214418809328f, fmaf(t35, 0.90963199535451833f, t33 * 0.54064081745559756f)))); const float t48 = fmaf(t42, 0.28173255684142967f, fmaf(t40, 0.75574957435425827f, fmaf(t38, 0.9898214418809328f, fmaf(t36, 0.90963199535451833f, t34 * 0.54064081745559756f))));
    const float t49 = t45 - t48; const float t50 = t46 + t47;
    const float t51 = t45 + t48; const float t52 = t46 - t47;
    const float t53 = fmaf(t31, 0.84125353283118121f, fmaf(t29, -0.14231483827328523f, fmaf(t27, -0.95949297361449748f, fmaf(t25, -0.65486073394528499f, fmaf(t23, 0.41541501300188644f, t1))))); const float t54 = fmaf(t32, 0.84125353283118121f, fmaf(t30, -0.14231483827328523f, fmaf(t28, -0.95949297361449748f, fmaf(t26, -0.65486073394528499f, fmaf(t24, 0.41541501300188644f, t2)))));
    const float t55 = fmaf(t41, -0.54064081745559744f, fmaf(t39, -0.98982144188093268f, fmaf(t37, -0.28173255684142939f, fmaf(t35, 0.75574957435425827f, t33 * 0.90963199535451833f)))); const float t56 = fmaf(t42, -0.54064081745559744f, fmaf(t40, -0.98982144188093268f, fmaf(t38, -0.28173255684142939f, fmaf(t36, 0.75574957435425827f, t34 * 0.90963199535451833f))));
    const float t57 = t53 - t56; const float t58 = t54 + t55;
    const float t59 = t53 + t56; const float t60 = t54 - t55;
    const float t61 = fmaf(t31, -0.65486073394528388f, fmaf(t29, 0.84125353283118154f, fmaf(t27, 0.41541501300188605f, fmaf(t25, -0.95949297361449748f, fmaf(t23, -0.142314838273285f, t1))))); const float t62 = fmaf(t32, -0.65486073394528388f, fmaf(t30, 0.84125353283118154f, fmaf(t28, 0.41541501300188605f, fmaf(t26, -0.95949297361449748f, fmaf(t24, -0.142314838273285f, t2)))));
    const float t63 = fmaf(t41, 0.75574957435425938f, fmaf(t39, 0.54064081745559711f, fmaf(t37, -0.90963199535451855f, fmaf(t35, -0.28173255684142939f, t33 * 0.9898214418809328f)))); const float t64 = fmaf(t42, 0.75574957435425938f, fmaf(t40, 0.54064081745559711f, fmaf(t38, -0.90963199535451855f, fmaf(t36, -0.28173255684142939f, t34 * 0.9898214418809328f))));
    const float t65 = t61 - t64; const float t66 = t62 + t63;
    const float t67 = t61 + t64; const float t68 = t62 - t63;
    const float t69 = fmaf(t31, 0.4154150130018866f, fmaf(t29, -0.95949297361449737f, fmaf(t27, 0.84125353283118154f, fmaf(t25, -0.14231483827328523f, fmaf(t23, -0.65486073394528499f, t1))))); const float t70 = fmaf(t32, 0.4154150130018866f, fmaf(t30, -0.95949297361449737f, fmaf(t28, 0.84125353283118154f, fmaf(t26, -0.14231483827328523f, fmaf(t24, -0.65486073394528499f, t2)))));
    const float t71 = fmaf(t41, -0.90963199535451833f, fmaf(t39, 0.28173255684142989f, fmaf(t37, 0.54064081745559711f, fmaf(t35, -0.98982144188093268f, t33 * 0.75574957435425827f)))); const float t72 = fmaf(t42, -0.90963199535451833f, fmaf(t40, 0.28173255684142989f, fmaf(t38, 0.54064081745559711f, fmaf(t36, -0.98982144188093268f, t34 * 0.75574957435425827f))));
    const float t73 = t69 - t72; const float t74 = t70 + t71;
    const float t75 = t69 + t72; const float t76 = t70 - t71;
    const float t77 = fmaf(t31, -0.14231483827328539f, fmaf(t29, 0.4154150130018866f, fmaf(t27, -0.65486073394528388f, fmaf(t25, 0.84125353283118121f, fmaf(t23, -0.95949297361449737f, t1))))); const float t78 = fmaf(t32, -0.14231483827328539f, fmaf(t30, 0.4154150130018866f, fmaf(t28, -0.65486073394528388f, fmaf(t26, 0.84125353283118121f, fmaf(t24, -0.95949297361449737f, t2)))));
    const float t79 = fmaf(t41, 0.98982144188093268f, fmaf(t39, -0.90963199535451833f, fmaf(t37, 0.75574957435425938f, fmaf(t35, -0.54064081745559744f, t33 * 0.28173255684142967f)))); const float t80 = fmaf(t42, 0.98982144188093268f, fmaf(t40, -0.90963199535451833f, fmaf(t38, 0.75574957435425938f, fmaf(t36, -0.54064081745559744f, t34 * 0.28173255684142967f))));
    const float t81 = t77 - t80; const float t82 = t78 + t79;
    const float t83 = t77 + t80; const float t84 = t78 - t79;
    v[0] = make_float2(t43, t44);
    v[1] = make_float2(t49, t50);
    v[2] = make_float2(t57, t58);
    v[3] = make_float2(t65, t66);
    v[4] = make_float2(t73, t74);
    v[5] = make_float2(t81, t82);
    v[6] = make_float2(t83, t84);
    v[7] = make_float2(t75, t76);
    v[8] = make_float2(t67, t68);
    v[9] = make_float2(t59, t60);
    v[10] = make_float2(t51, t52);
  }
};

template <> struct Dft<12, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[12]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = t1 + t13; const float t26 = t2 + t14;
    const float t27 = t1 - t13; const float t28 = t2 - t14;
    const float t29 = t7 + t19; const float t30 = t8 + t20;
    const float t31 = t7 - t19; const float t32 = t8 - t20;
    const float t33 = t32; const float t34 = -t31;
    const float t35 = t25 + t29; const float t36 = t26 + t30;
    const float t37 = t25 - t29; const float t38 = t26 - t30;
    const float t39 = t27 + t33; const float t40 = t28 + t34;
    const float t41 = t27 - t33; const float t42 = t28 - t34;
    const float t43 = t3 + t15; const float t44 = t4 + t16;
    const float t45 = t3 - t15; const float t46 = t4 - t16;
    const float t47 = t9 + t21; const float t48 = t10 + t22;
    const float t49 = t9 - t21; const float t50 = t10 - t22;
    const float t51 = t50; const float t52 = -t49;
    const float t53 = t43 + t47; const float t54 = t44 + t48;
    const float t55 = t43 - t47; const float t56 = t44 - t48;
    const float t57 = t45 + t51; const float t58 = t46 + t52;
    const float t59 = t45 - t51; const float t60 = t46 - t52;
    const float t61 = fmaf(t57, 0.86602540378443871f, -t58 * -0.49999999999999994f); const float t62 = fmaf(t57, -0.49999999999999994f, t58 * 0.86602540378443871f);
    const float t63 = fmaf(t55, 0.50000000000000011f, -t56 * -0.8660254037844386f); const float t64 = fmaf(t55, -0.8660254037844386f, t56 * 0.50000000000000011f);
    const float t65 = t60; const float t66 = -t59;
    const float t67 = t5 + t17; const float t68 = t6 + t18;
    const float t69 = t5 - t17; const float t70 = t6 - t18;
    const float t71 = t11 + t23; const float t72 = t12 + t24;
    const float t73 = t11 - t23; const float t74 = t12 - t24;
    const float t75 = t74; const float t76 = -t73;
    const float t77 = t67 + t71; const float t78 = t68 + t72;
    const float t79 = t67 - t71; const float t80 = t68 - t72;
    const float t81 = t69 + t75; const float t82 = t70 + t76;
    const float t83 = t69 - t75; const float t84 = t70 - t76;
    const float t85 = fmaf(t81, 0.50000000000000011f, -t82 * -0.8660254037844386f); const float t86 = fmaf(t81, -0.8660254037844386f, t82 * 0.50000000000000011f);
    const float t87 = fmaf(t79, -0.49999999999999978f, -t80 * -0.86602540378443871f); const float t88 = fmaf(t79, -0.86602540378443871f, t80 * -0.49999999999999978f);
    const float t89 = -t83; const float t90 = -t84;
    const float t91 = t53 + t77; const float t92 = t54 + t78;
    const float t93 = t53 - t77; const float t94 = t54 - t78;
    const float t95 = t35 + t91; const float t96 = t36 + t92;
    const float t97 = fmaf(t91, -0.49999999999999978f, t35); const float t98 = fmaf(t92, -0.49999999999999978f, t36);
    const float t99 = t93 * 0.86602540378443871f; const float t100 = t94 * 0.86602540378443871f;
    const float t101 = t97 + t100; const float t102 = t98 - t99;
    const float t103 = t97 - t100; const float t104 = t98 + t99;
    const float t105 = t61 + t85; const float t106 = t62 + t86;
    const float t107 = t61 - t85; const float t108 = t62 - t86;
    const float t109 = t39 + t105; const float t110 = t40 + t106;
    const float t111 = fmaf(t105, -0.49999999999999978f, t39); const float t112 = fmaf(t106, -0.49999999999999978f, t40);
    const float t113 = t107 * 0.86602540378443871f; const float t114 = t108 * 0.86602540378443871f;
    const float t115 = t111 + t114; const float t116 = t112 - t113;
    const float t117 = t111 - t114; const float t118 = t112 + t113;
    const float t119 = t63 + t87; const float t120 = t64 + t88;
    const float t121 = t63 - t87; const float t122 = t64 - t88;
    const float t123 = t37 + t119; const float t124 = t38 + t120;
    const float t125 = fmaf(t119, -0.49999999999999978f, t37); const float t126 = fmaf(t120, -0.49999999999999978f, t38);
    const float t127 = t121 * 0.86602540378443871f; const float t128 = t122 * 0.86602540378443871f;
    const float t129 = t125 + t128; const float t130 = t126 - t127;
    const float t131 = t125 - t128; const float t132 = t126 + t127;
    const float t133 = t65 + t89; const float t134 = t66 + t90;
    const float t135 = t65 - t89; const float t136 = t66 - t90;
    const float t137 = t41 + t133; const float t138 = t42 + t134;
    const float t139 = fmaf(t133, -0.49999999999999978f, t41); const float t140 = fmaf(t134, -0.49999999999999978f, t42);
    const float t141 = t135 * 0.86602540378443871f; const float t142 = t136 * 0.86602540378443871f;
    const float t143 = t139 + t142; const float t144 = t140 - t141;
    const float t145 = t139 - t142; const float t146 = t140 + t141;
    v[0] = make_float2(t95, t96);
    v[1] = make_float2(t109, t110);
    v[2] = make_float2(t123, t124);
    v[3] = make_float2(t137, t138);
    v[4] = make_float2(t101, t102);
    v[5] = make_float2(t115, t116);
    v[6] = make_float2(t129, t130);
    v[7] = make_float2(t143, t144);
    v[8] = make_float2(t103, t104);
    v[9] = make_float2(t117, t118);
    v[10] = make_float2(t131, t132);
    v[11] = make_float2(t145, t146);
  }
};

template <> struct Dft<12, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[12]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = t1 + t13; const float t26 = t2 + t14;
    const float t27 = t1 - t13; const float t28 = t2 - t14;
    const float t29 = t7 + t19; const float t30 = t8 + t20;
    const float t31 = t7 - t19; const float t32 = t8 - t20;
    const float t33 = -t32; const float t34 = t31;
    const float t35 = t25 + t29; const float t36 = t26 + t30;
    const float t37 = t25 - t29; const float t38 = t26 - t30;
    const float t39 = t27 + t33; const float t40 = t28 + t34;
    const float t41 = t27 - t33; const float t42 = t28 - t34;
    const float t43 = t3 + t15; const float t44 = t4 + t16;
    const float t45 = t3 - t15; const float t46 = t4 - t16;
    const float t47 = t9 + t21; const float t48 = t10 + t22;
    const float t49 = t9 - t21; const float t50 = t10 - t22;
    const float t51 = -t50; const float t52 = t49;
    const float t53 = t43 + t47; const float t54 = t44 + t48;
    const float t55 = t43 - t47; const float t56 = t44 - t48;
    const float t57 = t45 + t51; const float t58 = t46 + t52;
    const float t59 = t45 - t51; const float t60 = t46 - t52;
    const float t61 = fmaf(t57, 0.86602540378443871f, -t58 * 0.49999999999999994f); const float t62 = fmaf(t57, 0.49999999999999994f, t58 * 0.86602540378443871f);
    const float t63 = fmaf(t55, 0.50000000000000011f, -t56 * 0.8660254037844386f); const float t64 = fmaf(t55, 0.8660254037844386f, t56 * 0.50000000000000011f);
    const float t65 = -t60; const float t66 = t59;
    const float t67 = t5 + t17; const float t68 = t6 + t18;
    const float t69 = t5 - t17; const float t70 = t6 - t18;
    const float t71 = t11 + t23; const float t72 = t12 + t24;
    const float t73 = t11 - t23; const float t74 = t12 - t24;
    const float t75 = -t74; const float t76 = t73;
    const float t77 = t67 + t71; const float t78 = t68 + t72;
    const float t79 = t67 - t71; const float t80 = t68 - t72;
    const float t81 = t69 + t75; const float t82 = t70 + t76;
    const float t83 = t69 - t75; const float t84 = t70 - t76;
    const float t85 = fmaf(t81, 0.50000000000000011f, -t82 * 0.8660254037844386f); const float t86 = fmaf(t81, 0.8660254037844386f, t82 * 0.50000000000000011f);
    const float t87 = fmaf(t79, -0.49999999999999978f, -t80 * 0.86602540378443871f); const float t88 = fmaf(t79, 0.86602540378443871f, t80 * -0.49999999999999978f);
    const float t89 = -t83; const float t90 = -t84;
    const float t91 = t53 + t77; const float t92 = t54 + t78;
    const float t93 = t53 - t77; const float t94 = t54 - t78;
    const float t95 = t35 + t91; const float t96 = t36 + t92;
    const float t97 = fmaf(t91, -0.49999999999999978f, t35); const float t98 = fmaf(t92, -0.49999999999999978f, t36);
    const float t99 = t93 * 0.86602540378443871f; const float t100 = t94 * 0.86602540378443871f;
    const float t101 = t97 - t100; const float t102 = t98 + t99;
    const float t103 = t97 + t100; const float t104 = t98 - t99;
    const float t105 = t61 + t85; const float t106 = t62 + t86;
    const float t107 = t61 - t85; const float t108 = t62 - t86;
    const float t109 = t39 + t105; const float t110 = t40 + t106;
    const float t111 = fmaf(t105, -0.49999999999999978f, t39); const float t112 = fmaf(t106, -0.49999999999999978f, t40);
    const float t113 = t107 * 0.86602540378443871f; const float t114 = t108 * 0.86602540378443871f;
    const float t115 = t111 - t114; const float t116 = t112 + t113;
    const float t117 = t111 + t114; const float t118 = t112 - t113;
    const float t119 = t63 + t87; const float t120 = t64 + t88;
    const float t121 = t63 - t87; const float t122 = t64 - t88;
    const float t123 = t37 + t119; const float t124 = t38 + t120;
    const float t125 = fmaf(t119, -0.49999999999999978f, t37); const float t126 = fmaf(t120, -0.49999999999999978f, t38);
    const float t127 = t121 * 0.86602540378443871f; const float t128 = t122 * 0.86602540378443871f;
    const float t129 = t125 - t128; const float t130 = t126 + t127;
    const float t131 = t125 + t128; const float t132 = t126 - t127;
    const float t133 = t65 + t89; const float t134 = t66 + t90;
    const float t135 = t65 - t89; const float t136 = t66 - t90;
    const float t137 = t41 + t133; const float t138 = t42 + t134;
    const float t139 = fmaf(t133, -0.49999999999999978f, t41); const float t140 = fmaf(t134, -0.49999999999999978f, t42);
    const float t141 = t135 * 0.86602540378443871f; const float t142 = t136 * 0.86602540378443871f;
    const float t143 = t139 - t142; const float t144 = t140 + t141;
    const float t145 = t139 + t142; const float t146 = t140 - t141;
    v[0] = make_float2(t95, t96);
    v[1] = make_float2(t109, t110);
    v[2] = make_float2(t123, t124);
    v[3] = make_float2(t137, t138);
    v[4] = make_float2(t101, t102);
    v[5] = make_float2(t115, t116);
    v[6] = make_float2(t129, t130);
    v[7] = make_float2(t143, t144);
    v[8] = make_float2(t103, t104);
    v[9] = make_float2(t117, t118);
    v[10] = make_float2(t131, t132);
    v[11] = make_float2(t145, t146);
  }
};

template <> struct Dft<13, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[13]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = t3 + t25; const float t28 = t4 + t26;
    const float t29 = t5 + t23; const float t30 = t6 + t24;
    const float t31 = t7 + t21; const float t32 = t8 + t22;
    const float t33 = t9 + t19; const float t34 = t10 + t20;
    const float t35 = t11 + t17; const float t36 = t12 + t18;
    const float t37 = t13 + t15; const float t38 = t14 + t16;
    const float t39 = t3 - t25; const float t40 = t4 - t26;
    const float t41 = t5 - t23; const float t42 = t6 - t24;
    const float t43 = t7 - t21; const float t44 = t8 - t22;
    const float t45 = t9 - t19; const float t46 = t10 - t20;
    const float t47 = t11 - t17; const float t48 = t12 - t18;
    const float t49 = t13 - t15; const float t50 = t14 - t16;
    const float t51 = t1 + t27 + t29 + t31 + t33 + t35 + t37; const float t52 = t2 + t28 + t30 + t32 + t34 + t36 + t38;
    const float t53 = fmaf(t37, -0.97094181742605201f, fmaf(t35, -0.74851074817110119f, fmaf(t33, -0.35460488704253545f, fmaf(t31, 0.12053668025532301f, fmaf(t29, 0.56806474673115592f, fmaf(t27, 0.88545602565320991f, t1)))))); const float t54 = fmaf(t38, -0.97094181742605201f, fmaf(t36, -0.74851074817110119f, fmaf(t34, -0.35460488704253545f, fmaf(t32, 0.12053668025532301f, fmaf(t30, 0.56806474673115592f, fmaf(t28, 0.88545602565320991f, t2))))));
    const float t55 = fmaf(t49, 0.23931566428755768f, fmaf(t47, 0.66312265824079519f, fmaf(t45, 0.93501624268541483f, fmaf(t43, 0.99270887409805397f, fmaf(t41, 0.82298386589365635f, t39 * 0.46472317204376851f))))); const float t56 = fmaf(t50, 0.23931566428755768f, fmaf(t48, 0.66312265824079519f, fmaf(t46, 0.93501624268541483f, fmaf(t44, 0.99270887409805397f, fmaf(t42, 0.82298386589365635f, t40 * 0.46472317204376851f)))));
    const float t57 = t53 + t56; const float t58 = t54 - t55;
    const float t59 = t53 - t56; const float t60 = t54 + t55;
    const float t61 = fmaf(t37, 0.88545602565321002f, fmaf(t35, 0.1205366802553232f, fmaf(t33, -0.7485107481711013f, fmaf(t31, -0.97094181742605201f, fmaf(t29, -0.35460488704253545f, fmaf(t27, 0.56806474673115592f, t1)))))); const float t62 = fmaf(t38, 0.88545602565321002f, fmaf(t36, 0.1205366802553232f, fmaf(t34, -0.7485107481711013f, fmaf(t32, -0.97094181742605201f, fmaf(t30, -0.35460488704253545f, fmaf(t28, 0.56806474673115592f, t2))))));
    const float t63 = fmaf(t49, -0.4647231720437684f, fmaf(t47, -0.99270887409805397f, fmaf(t45, -0.66312265824079497f, fmaf(t43, 0.23931566428755768f, fmaf(t41, 0.93501624268541483f, t39 * 0.82298386589365635f))))); const float t64 = fmaf(t50, -0.4647231720437684f, fmaf(t48, -0.99270887409805397f, fmaf(t46, -0.66312265824079497f, fmaf(t44, 0.23931566428755768f, fmaf(t42, 0.93501624268541483f, t40 * 0.82298386589365635f)))));
    const float t65 = t61 + t64; const float t66 = t62 - t63;
    const float t67 = t61 - t64; const float t68 = t62 + t63;
    const float t69 = fmaf(t37, -0.74851074817110064f, fmaf(t35, 0.5680647467311567f, fmaf(t33, 0.88545602565321002f, fmaf(t31, -0.3546048870425359f, fmaf(t29, -0.97094181742605201f, fmaf(t27, 0.12053668025532301f, t1)))))); const float t70 = fmaf(t38, -0.74851074817110064f, fmaf(t36, 0.5680647467311567f, fmaf(t34, 0.88545602565321002f, fmaf(t32, -0.3546048870425359f, fmaf(t30, -0.97094181742605201f, fmaf(t28, 0.12053668025532301f, t2))))));
    const float t71 = fmaf(t49, 0.66312265824079564f, fmaf(t47, 0.8229838658936558f, fmaf(t45, -0.4647231720437684f, fmaf(t43, -0.93501624268541472f, fmaf(t41, 0.23931566428755768f, t39 * 0.99270887409805397f))))); const float t72 = fmaf(t50, 0.66312265824079564f, fmaf(t48, 0.8229838658936558f, fmaf(t46, -0.4647231720437684f, fmaf(t44, -0.93501624268541472f, fmaf(t42, 0.23931566428755768f, t40 * 0.99270887409805397f)))));
    const float t73 = t69 + t72; const float t74 = t70 - t71;
    const float t75 = t69 - t72; const float t76 = t70 + t71;
    const float t77 = fmaf(t37, 0.56806474673115614f, fmaf(t35, -0.9709418174260519f, fmaf(t33, 0.12053668025532369f, fmaf(t31, 0.88545602565321002f, fmaf(t29, -0.7485107481711013f, fmaf(t27, -0.35460488704253545f, t1)))))); const float t78 = fmaf(t38, 0.56806474673115614f, fmaf(t36, -0.9709418174260519f, fmaf(t34, 0.12053668025532369f, fmaf(t32, 0.88545602565321002f, fmaf(t30, -0.7485107481711013f, fmaf(t28, -0.35460488704253545f, t2))))));
    const float t79 = fmaf(t49, -0.82298386589365613f, fmaf(t47, -0.23931566428755807f, fmaf(t45, 0.99270887409805386f, fmaf(t43, -0.4647231720437684f, fmaf(t41, -0.66312265824079497f, t39 * 0.93501624268541483f))))); const float t80 = fmaf(t50, -0.82298386589365613f, fmaf(t48, -0.23931566428755807f, fmaf(t46, 0.99270887409805386f, fmaf(t44, -0.4647231720437684f, fmaf(t42, -0.66312265824079497f, t40 * 0.93501624268541483f)))));
    const float t81 = t77 + t80; const float t82 = t78 - t79;
    const float t83 = t77 - t80; const float t84 = t78 + t79;
    const float t85 = fmaf(t37, -0.35460488704253357f, fmaf(t35, 0.88545602565320991f, fmaf(t33, -0.9709418174260519f, fmaf(t31, 0.5680647467311567f, fmaf(t29, 0.1205366802553232f, fmaf(t27, -0.74851074817110119f, t1)))))); const float t86 = fmaf(t38, -0.35460488704253357f, fmaf(t36, 0.88545602565320991f, fmaf(t34, -0.9709418174260519f, fmaf(t32, 0.5680647467311567f, fmaf(t30, 0.1205366802553232f, fmaf(t28, -0.74851074817110119f, t2))))));
    const float t87 = fmaf(t49, 0.93501624268541561f, fmaf(t47, -0.46472317204376862f, fmaf(t45, -0.23931566428755807f, fmaf(t43, 0.8229838658936558f, fmaf(t41, -0.99270887409805397f, t39 * 0.66312265824079519f))))); const float t88 = fmaf(t50, 0.93501624268541561f, fmaf(t48, -0.46472317204376862f, fmaf(t46, -0.23931566428755807f, fmaf(t44, 0.8229838658936558f, fmaf(t42, -0.99270887409805397f, t40 * 0.66312265824079519f)))));
    const float t89 = t85 + t88; const float t90 = t86 - t87;
    const float t91 = t85 - t88; const float t92 = t86 + t87;
    const float t93 = fmaf(t37, 0.12053668025532184f, fmaf(t35, -0.35460488704253357f, fmaf(t33, 0.56806474673115614f, fmaf(t31, -0.74851074817110064f, fmaf(t29, 0.88545602565321002f, fmaf(t27, -0.97094181742605201f, t1)))))); const float t94 = fmaf(t38, 0.12053668025532184f, fmaf(t36, -0.35460488704253357f, fmaf(t34, 0.56806474673115614f, fmaf(t32, -0.74851074817110064f, fmaf(t30, 0.88545602565321002f, fmaf(t28, -0.97094181742605201f, t2))))));
    const float t95 = fmaf(t49, -0.99270887409805419f, fmaf(t47, 0.93501624268541561f, fmaf(t45, -0.82298386589365613f, fmaf(t43, 0.66312265824079564f, fmaf(t41, -0.4647231720437684f, t39 * 0.23931566428755768f))))); const float t96 = fmaf(t50, -0.99270887409805419f, fmaf(t48, 0.93501624268541561f, fmaf(t46, -0.82298386589365613f, fmaf(t44, 0.66312265824079564f, fmaf(t42, -0.4647231720437684f, t40 * 0.23931566428755768f)))));
    const float t97 = t93 + t96; const float t98 = t94 - t95;
    const float t99 = t93 - t96; const float t100 = t94 + t95;
    v[0] = make_float2(t51, t52);
    v[1] = make_float2(t57, t58);
    v[2] = make_float2(t65, t66);
    v[3] = make_float2(t73, t74);
    v[4] = make_float2(t81, t82);
    v[5] = make_float2(t89, t90);
    v[6] = make_float2(t97, t98);
    v[7] = make_float2(t99, t100);
    v[8] = make_float2(t91, t92);
    v[9] = make_float2(t83, t84);
    v[10] = make_float2(t75, t76);
    v[11] = make_float2(t67, t68);
    v[12] = make_float2(t59, t60);
  }
};

template <> struct Dft<13, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[13]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = t3 + t25; const float t28 = t4 + t26;
    const float t29 = t5 + t23; const float t30 = t6 + t24;
    const float t31 = t7 + t21; const float t32 = t8 + t22;
    const float t33 = t9 + t19; const float t34 = t10 + t20;
    const float t35 = t11 + t17; const float t36 = t12 + t18;
    const float t37 = t13 + t15; const float t38 = t14 + t16;
    const float t39 = t3 - t25; const float t40 = t4 - t26;
    const float t41 = t5 - t23; const float t42 = t6 - t24;
    const float t43 = t7 - t21; const float t44 = t8 - t22;
    const float t45 = t9 - t19; const float t46 = t10 - t20;
    const float t47 = t11 - t17; const float t48 = t12 - t18;
    const float t49 = t13 - t15; const float t50 = t14 - t16;
    const float t51 = t1 + t27 + t29 + t31 + t33 + t35 + t37; const float t52 = t2 + t28 + t30 + t32 + t34 + t36 + t38;
    const float t53 = fmaf(t37, -0.97094181742605201f, fmaf(t35, -0.74851074817110119f, fmaf(t33, -0.35460488704253545f, fmaf(t31, 0.12053668025532301f, fmaf(t29, 0.56806474673115592f, fmaf(t27, 0.88545602565320991f, t1)))))); const float t54 = fmaf(t38, -0.97094181742605201f, fmaf(t36, -0.74851074817110119f, fmaf(t34, -0.35460488704253545f, fmaf(t32, 0.12053668025532301f, fmaf(t30, 0.56806474673115592f, fmaf(t28, 0.88545602565320991f, t2))))));
    const float t55 = fmaf(t49, 0.23931566428755768f, fmaf(t47, 0.66312265824079519f, fmaf(t45, 0.93501624268541483f, fmaf(t43, 0.99270887409805397f, fmaf(t41, 0.82298386589365635f, t39 * 0.46472317204376851f))))); const float t56 = fmaf(t50, 0.23931566428755768f, fmaf(t48, 0.66312265824079519f, fmaf(t46, 0.93501624268541483f, fmaf(t44, 0.99270887409805397f, fmaf(t42, 0.82298386589365635f, t40 * 0.46472317204376851f)))));
    const float t57 = t53 - t56; const float t58 = t54 + t55;
    const float t59 = t53 + t56; const float t60 = t54 - t55;
    const float t61 = fmaf(t37, 0.88545602565321002f, fmaf(t35, 0.1205366802553232f, fmaf(t33, -0.7485107481711013f, fmaf(t31, -0.97094181742605201f, fmaf(t29, -0.35460488704253545f, fmaf(t27, 0.56806474673115592f, t1)))))); const float t62 = fmaf(t38, 0.88545602565321002f, fmaf(t36, 0.1205366802553232f, fmaf(t34, -0.7485107481711013f, fmaf(t32, -0.97094181742605201f, fmaf(t30, -0.35460488704253545f, fmaf(t28, 0.56806474673115592f, t2))))));
    const float t63 = fmaf(t49, -0.4647231720437684f, fmaf(t47, -0.99270887409805397f, fmaf(t45, -0.66312265824079497f, fmaf(t43, 0.23931566428755768f, fmaf(t41, 0.93501624268541483f, t39 * 0.82298386589365635f))))); const float t64 = fmaf(t50, -0.4647231720437684f, fmaf(t48, -0.99270887409805397f, fmaf(t46, -0.66312265824079497f, fmaf(t44, 0.23931566428755768f, fmaf(t42, 0.93501624268541483f, t40 * 0.82298386589365635f)))));
    const float t65 = t61 - t64; const float t66 = t62 + t63;
    const float t67 = t61 + t64; const float t68 = t62 - t63;
    const float t69 = fmaf(t37, -0.74851074817110064f, fmaf(t35, 0.5680647467311567f, fmaf(t33, 0.88545602565321002f, fmaf(t31, -0.3546048870425359f, fmaf(t29, -0.97094181742605201f, fmaf(t27, 0.12053668025532301f, t1)))))); const float t70 = fmaf(t38, -0.74851074817110064f, fmaf(t36, 0.5680647467311567f, fmaf(t34, 0.88545602565321002f, fmaf(t32, -0.3546048870425359f, fmaf(t30, -0.97094181742605201f, fmaf(t28, 0.12053668025532301f, t2))))));
    const float t71 = fmaf(t49, 0.66312265824079564f, fmaf(t47, 0.8229838658936558f, fmaf(t45, -0.4647231720437684f, fmaf(t43, -0.93501624268541472f, fmaf(t41, 0.23931566428755768f, t39 * 0.99270887409805397f))))); const float t72 = fmaf(t50, 0.66312265824079564f, fmaf(t48, 0.8229838658936558f, fmaf(t46, -0.4647231720437684f, fmaf(t44, -0.93501624268541472f, fmaf(t42, 0.23931566428755768f, t40 * 0.99270887409805397f)))));
    const float t73 = t69 - t72; const float t74 = t70 + t71;
    const float t75 = t69 + t72; const float t76 = t70 - t71;
    const float t77 = fmaf(t37, 0.56806474673115614f, fmaf(t35, -0.9709418174260519f, fmaf(t33, 0.12053668025532369f, fmaf(t31, 0.88545602565321002f, fmaf(t29, -0.7485107481711013f, fmaf(t27, -0.35460488704253545f, t1)))))); const float t78 = fmaf(t38, 0.56806474673115614f, fmaf(t36, -0.9709418174260519f, fmaf(t34, 0.12053668025532369f, fmaf(t32, 0.88545602565321002f, fmaf(t30, -0.7485107481711013f, fmaf(t28, -0.35460488704253545f, t2))))));
    const float t79 = fmaf(t49, -0.82298386589365613f, fmaf(t47, -0.23931566428755807f, fmaf(t45, 0.99270887409805386f, fmaf(t43, -0.4647231720437684f, fmaf(t41, -0.66312265824079497f, t39 * 0.93501624268541483f))))); const float t80 = fmaf(t50, -0.82298386589365613f, fmaf(t48, -0.23931566428755807f, fmaf(t46, 0.99270887409805386f, fmaf(t44, -0.4647231720437684f, fmaf(t42, -0.66312265824079497f, t40 * 0.93501624268541483f)))));
    const float t81 = t77 - t80; const float t82 = t78 + t79;
    const float t83 = t77 + t80; const float t84 = t78 - t79;
    const float t85 = fmaf(t37, -0.35460488704253357f, fmaf(t35, 0.88545602565320991f, fmaf(t33, -0.9709418174260519f, fmaf(t31, 0.5680647467311567f, fmaf(t29, 0.1205366802553232f, fmaf(t27, -0.74851074817110119f, t1)))))); const float t86 = fmaf(t38, -0.35460488704253357f, fmaf(t36, 0.88545602565320991f, fmaf(t34, -0.9709418174260519f, fmaf(t32, 0.5680647467311567f, fmaf(t30, 0.1205366802553232f, fmaf(t28, -0.74851074817110119f, t2))))));
    const float t87 = fmaf(t49, 0.93501624268541561f, fmaf(t47, -0.46472317204376862f, fmaf(t45, -0.23931566428755807f, fmaf(t43, 0.8229838658936558f, fmaf(t41, -0.99270887409805397f, t39 * 0.66312265824079519f))))); const float t88 = fmaf(t50, 0.93501624268541561f, fmaf(t48, -0.46472317204376862f, fmaf(t46, -0.23931566428755807f, fmaf(t44, 0.8229838658936558f, fmaf(t42, -0.99270887409805397f, t40 * 0.66312265824079519f)))));
    const float t89 = t85 - t88; const float t90 = t86 + t87;
    const float t91 = t85 + t88; const float t92 = t86 - t87;
    const float t93 = fmaf(t37, 0.12053668025532184f, fmaf(t35, -0.35460488704253357f, fmaf(t33, 0.56806474673115614f, fmaf(t31, -0.74851074817110064f, fmaf(t29, 0.88545602565321002f, fmaf(t27, -0.97094181742605201f, t1)))))); const float t94 = fmaf(t38, 0.12053668025532184f, fmaf(t36, -0.35460488704253357f, fmaf(t34, 0.56806474673115614f, fmaf(t32, -0.74851074817110064f, fmaf(t30, 0.88545602565321002f, fmaf(t28, -0.97094181742605201f, t2))))));
    const float t95 = fmaf(t49, -0.99270887409805419f, fmaf(t47, 0.93501624268541561f, fmaf(t45, -0.82298386589365613f, fmaf(t43, 0.66312265824079564f, fmaf(t41, -0.4647231720437684f, t39 * 0.23931566428755768f))))); const float t96 = fmaf(t50, -0.99270887409805419f, fmaf(t48, 0.93501624268541561f, fmaf(t46, -0.82298386589365613f, fmaf(t44, 0.66312265824079564f, fmaf(t42, -0.4647231720437684f, t40 * 0.23931566428755768f)))));
    const float t97 = t93 - t96; const float t98 = t94 + t95;
    const float t99 = t93 + t96; const float t100 = t94 - t95;
    v[0] = make_float2(t51, t52);
    v[1] = make_float2(t57, t58);
    v[2] = make_float2(t65, t66);
    v[3] = make_float2(t73, t74);
    v[4] = make_float2(t81, t82);
    v[5] = make_float2(t89, t90);
    v[6] = make_float2(t97, t98);
    v[7] = make_float2(t99, t100);
    v[8] = make_float2(t91, t92);
    v[9] = make_float2(t83, t84);
    v[10] = make_float2(t75, t76);
    v[11] = make_float2(t67, t68);
    v[12] = make_float2(t59, t60);
  }
};

template <> struct Dft<14, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[14]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = v[13].x; const float t28 = v[13].y;
    const float t29 = t1 + t15; const float t30 = t2 + t16;
    const float t31 = t1 - t15; const float t32 = t2 - t16;
    const float t33 = t3 + t17; const float t34 = t4 + t18;
    const float t35 = t3 - t17; const float t36 = t4 - t18;
    const float t37 = fmaf(t35, 0.90096886790241915f, -t36 * -0.43388373911755812f); const float t38 = fmaf(t35, -0.43388373911755812f, t36 * 0.90096886790241915f);
    const float t39 = t5 + t19; const float t40 = t6 + t20;
    const float t41 = t5 - t19; const float t42 = t6 - t20;
    const float t43 = fmaf(t41, 0.62348980185873359f, -t42 * -0.7818314824680298f); const float t44 = fmaf(t41, -0.7818314824680298f, t42 * 0.62348980185873359f);
    const float t45 = t7 + t21; const float t46 = t8 + t22;
    const float t47 = t7 - t21; const float t48 = t8 - t22;
    const float t49 = fmaf(t47, 0.22252093395631445f, -t48 * -0.97492791218182362f); const float t50 = fmaf(t47, -0.97492791218182362f, t48 * 0.22252093395631445f);
    const float t51 = t9 + t23; const float t52 = t10 + t24;
    const float t53 = t9 - t23; const float t54 = t10 - t24;
    const float t55 = fmaf(t53, -0.22252093395631434f, -t54 * -0.97492791218182362f); const float t56 = fmaf(t53, -0.97492791218182362f, t54 * -0.22252093395631434f);
    const float t57 = t11 + t25; const float t58 = t12 + t26;
    const float t59 = t11 - t25; const float t60 = t12 - t26;
    const float t61 = fmaf(t59, -0.62348980185873348f, -t60 * -0.78183148246802991f); const float t62 = fmaf(t59, -0.78183148246802991f, t60 * -0.62348980185873348f);
    const float t63 = t13 + t27; const float t64 = t14 + t28;
    const float t65 = t13 - t27; const float t66 = t14 - t28;
    const float t67 = fmaf(t65, -0.90096886790241903f, -t66 * -0.43388373911755823f); const float t68 = fmaf(t65, -0.43388373911755823f, t66 * -0.90096886790241903f);
    const float t69 = t33 + t63; const float t70 = t34 + t64;
    const float t71 = t39 + t57; const float t72 = t40 + t58;
    const float t73 = t45 + t51; const float t74 = t46 + t52;
    const float t75 = t33 - t63; const float t76 = t34 - t64;
    const float t77 = t39 - t57; const float t78 = t40 - t58;
    const float t79 = t45 - t51; const float t80 = t46 - t52;
    const float t81 = t29 + t69 + t71 + t73; const float t82 = t30 + t70 + t72 + t74;
    const float t83 = fmaf(t73, -0.90096886790241903f, fmaf(t71, -0.22252093395631434f, fmaf(t69, 0.62348980185873359f, t29))); const float t84 = fmaf(t74, -0.90096886790241903f, fmaf(t72, -0.22252093395631434f, fmaf(t70, 0.62348980185873359f, t30)));
    const float t85 = fmaf(t79, 0.43388373911755823f, fmaf(t77, 0.97492791218182362f, t75 * 0.7818314824680298f)); const float t86 = fmaf(t80, 0.43388373911755823f, fmaf(t78, 0.97492791218182362f, t76 * 0.7818314824680298f));
    const float t87 = t83 + t86; const float t88 = t84 - t85;
    const float t89 = t83 - t86; const float t90 = t84 + t85;
    const float t91 = fmaf(t73, 0.62348980185873337f, fmaf(t71, -0.90096886790241915f, fmaf(t69, -0.22252093395631434f, t29))); const float t92 = fmaf(t74, 0.62348980185873337f, fmaf(t72, -0.90096886790241915f, fmaf(t70, -0.22252093395631434f, t30)));
    const float t93 = fmaf(t79, -0.78183148246802991f, fmaf(t77, -0.43388373911755801f, t75 * 0.97492791218182362f)); const float t94 = fmaf(t80, -0.78183148246802991f, fmaf(t78, -0.43388373911755801f, t76 * 0.97492791218182362f));
    const float t95 = t91 + t94; const float t96 = t92 - t93;
    const float t97 = t91 - t94; const float t98 = t92 + t93;
    const float t99 = fmaf(t73, -0.22252093395631409f, fmaf(t71, 0.62348980185873337f, fmaf(t69, -0.90096886790241903f, t29))); const float t100 = fmaf(t74, -0.22252093395631409f, fmaf(t72, 0.62348980185873337f, fmaf(t70, -0.90096886790241903f, t30)));
    const float t101 = fmaf(t79, 0.97492791218182373f, fmaf(t77, -0.78183148246802991f, t75 * 0.43388373911755823f)); const float t102 = fmaf(t80, 0.97492791218182373f, fmaf(t78, -0.78183148246802991f, t76 * 0.43388373911755823f));
    const float t103 = t99 + t102; const float t104 = t100 - t101;
    const float t105 = t99 - t102; const float t106 = t100 + t101;
    const float t107 = t37 + t67; const float t108 = t38 + t68;
    const float t109 = t43 + t61; const float t110 = t44 + t62;
    const float t111 = t49 + t55; const float t112 = t50 + t56;
    const float t113 = t37 - t67; const float t114 = t38 - t68;
    const float t115 = t43 - t61; const float t116 = t44 - t62;
    const float t117 = t49 - t55; const float t118 = t50 - t56;
    const float t119 = t31 + t107 + t109 + t111; const float t120 = t32 + t108 + t110 + t112;
    const float t121 = fmaf(t111, -0.90096886790241903f, fmaf(t109, -0.22252093395631434f, fmaf(t107, 0.62348980185873359f, t31))); const float t122 = fmaf(t112, -0.90096886790241903f, fmaf(t110, -0.22252093395631434f, fmaf(t108, 0.62348980185873359f, t32)));
    const float t123 = fmaf(t117, 0.43388373911755823f, fmaf(t115, 0.97492791218182362f, t113 * 0.7818314824680298f)); const float t124 = fmaf(t118, 0.43388373911755823f, fmaf(t116, 0.97492791218182362f, t114 * 0.7818314824680298f));
    const float t125 = t121 + t124; const float t126 = t122 - t123;
    const float t127 = t121 - t124; const float t128 = t122 + t123;
    const float t129 = fmaf(t111, 0.62348980185873337f, fmaf(t109, -0.90096886790241915f, fmaf(t107, -0.22252093395631434f, t31))); const float t130 = fmaf(t112, 0.62348980185873337f, fmaf(t110, -0.90096886790241915f, fmaf(t108, -0.22252093395631434f, t32)));
    const float t131 = fmaf(t117, -0.78183148246802991f, fmaf(t115, -0.43388373911755801f, t113 * 0.97492791218182362f)); const float t132 = fmaf(t118, -0.78183148246802991f, fmaf(t116, -0.43388373911755801f, t114 * 0.97492791218182362f));
    const float t133 = t129 + t132; const float t134 = t130 - t131;
    const float t135 = t129 - t132; const float t136 = t130 + t131;
    const float t137 = fmaf(t111, -0.22252093395631409f, fmaf(t109, 0.62348980185873337f, fmaf(t107, -0.90096886790241903f, t31))); const float t138 = fmaf(t112, -0.22252093395631409f, fmaf(t110, 0.62348980185873337f, fmaf(t108, -0.90096886790241903f, t32)));
    const float t139 = fmaf(t117, 0.97492791218182373f, fmaf(t115, -0.78183148246802991f, t113 * 0.43388373911755823f)); const float t140 = fmaf(t118, 0.97492791218182373f, fmaf(t116, -0.78183148246802991f, t114 * 0.43388373911755823f));
    const float t141 = t137 + t140; const float t142 = t138 - t139;
    const float t143 = t137 - t140; const float t144 = t138 + t139;
    v[0] = make_float2(t81, t82);
    v[1] = make_float2(t119, t120);
    v[2] = make_float2(t87, t88);
    v[3] = make_float2(t125, t126);
    v[4] = make_float2(t95, t96);
    v[5] = make_float2(t133, t134);
    v[6] = make_float2(t103, t104);
    v[7] = make_float2(t141, t142);
    v[8] = make_float2(t105, t106);
    v[9] = make_float2(t143, t144);
    v[10] = make_float2(t97, t98);
    v[11] = make_float2(t135, t136);
    v[12] = make_float2(t89, t90);
    v[13] = make_float2(t127, t128);
  }
};

template <> struct Dft<14, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[14]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = v[13].x; const float t28 = v[13].y;
    const float t29 = t1 + t15; const float t30 = t2 + t16;
    const float t31 = t1 - t15; const float t32 = t2 - t16;
    const float t33 = t3 + t17; const float t34 = t4 + t18;
    const float t35 = t3 - t17; const float t36 = t4 - t18;
    const float t37 = fmaf(t35, 0.90096886790241915f, -t36 * 0.43388373911755812f); const float t38 = fmaf(t35, 0.43388373911755812f, t36 * 0.90096886790241915f);
    const float t39 = t5 + t19; const float t40 = t6 + t20;
    const float t41 = t5 - t19; const float t42 = t6 - t20;
    const float t43 = fmaf(t41, 0.62348980185873359f, -t42 * 0.7818314824680298f); const float t44 = fmaf(t41, 0.7818314824680298f, t42 * 0.62348980185873359f);
    const float t45 = t7 + t21; const float t46 = t8 + t22;
    const float t47 = t7 - t21; const float t48 = t8 - t22;
    const float t49 = fmaf(t47, 0.22252093395631445f, -t48 * 0.97492791218182362f); const float t50 = fmaf(t47, 0.97492791218182362f, t48 * 0.22252093395631445f);
    const float t51 = t9 + t23; const float t52 = t10 + t24;
    const float t53 = t9 - t23; const float t54 = t10 - t24;
    const float t55 = fmaf(t53, -0.22252093395631434f, -t54 * 0.97492791218182362f); const float t56 = fmaf(t53, 0.97492791218182362f, t54 * -0.22252093395631434f);
    const float t57 = t11 + t25; const float t58 = t12 + t26;
    const float t59 = t11 - t25; const float t60 = t12 - t26;
    const float t61 = fmaf(t59, -0.62348980185873348f, -t60 * 0.78183148246802991f); const float t62 = fmaf(t59, 0.78183148246802991f, t60 * -0.62348980185873348f);
    const float t63 = t13 + t27; const float t64 = t14 + t28;
    const float t65 = t13 - t27; const float t66 = t14 - t28;
    const float t67 = fmaf(t65, -0.90096886790241903f, -t66 * 0.43388373911755823f); const float t68 = fmaf(t65, 0.43388373911755823f, t66 * -0.90096886790241903f);
    const float t69 = t33 + t63; const float t70 = t34 + t64;
    const float t71 = t39 + t57; const float t72 = t40 + t58;
    const float t73 = t45 + t51; const float t74 = t46 + t52;
    const float t75 = t33 - t63; const float t76 = t34 - t64;
    const float t77 = t39 - t57; const float t78 = t40 - t58;
    const float t79 = t45 - t51; const float t80 = t46 - t52;
    const float t81 = t29 + t69 + t71 + t73; const float t82 = t30 + t70 + t72 + t74;
    const float t83 = fmaf(t73, -0.90096886790241903f, fmaf(t71, -0.22252093395631434f, fmaf(t69, 0.62348980185873359f, t29))); const float t84 = fmaf(t74, -0.90096886790241903f, fmaf(t72, -0.22252093395631434f, fmaf(t70, 0.62348980185873359f, t30)));
    const float t85 = fmaf(t79, 0.43388373911755823f, fmaf(t77, 0.97492791218182362f, t75 * 0.7818314824680298f)); const float t86 = fmaf(t80, 0.43388373911755823f, fmaf(t78, 0.97492791218182362f, t76 * 0.7818314824680298f));
    const float t87 = t83 - t86; const float t88 = t84 + t85;
    const float t89 = t83 + t86; const float t90 = t84 - t85;
    const float t91 = fmaf(t73, 0.62348980185873337f, fmaf(t71, -0.90096886790241915f, fmaf(t69, -0.22252093395631434f, t29))); const float t92 = fmaf(t74, 0.62348980185873337f, fmaf(t72, -0.90096886790241915f, fmaf(t70, -0.22252093395631434f, t30)));
    const float t93 = fmaf(t79, -0.78183148246802991f, fmaf(t77, -0.43388373911755801f, t75 * 0.97492791218182362f)); const float t94 = fmaf(t80, -0.78183148246802991f, fmaf(t78, -0.43388373911755801f, t76 * 0.97492791218182362f));
    const float t95 = t91 - t94; const float t96 = t92 + t93;
    const float t97 = t91 + t94; const float t98 = t92 - t93;
    const float t99 = fmaf(t73, -0.22252093395631409f, fmaf(t71, 0.62348980185873337f, fmaf(t69, -0.90096886790241903f, t29))); const float t100 = fmaf(t74, -0.22252093395631409f, fmaf(t72, 0.62348980185873337f, fmaf(t70, -0.90096886790241903f, t30)));
    const float t101 = fmaf(t79, 0.97492791218182373f, fmaf(t77, -0.78183148246802991f, t75 * 0.43388373911755823f)); const float t102 = fmaf(t80, 0.97492791218182373f, fmaf(t78, -0.78183148246802991f, t76 * 0.43388373911755823f));
    const float t103 = t99 - t102; const float t104 = t100 + t101;
    const float t105 = t99 + t102; const float t106 = t100 - t101;
    const float t107 = t37 + t67; const float t108 = t38 + t68;
    const float t109 = t43 + t61; const float t110 = t44 + t62;
    const float t111 = t49 + t55; const float t112 = t50 + t56;
    const float t113 = t37 - t67; const float t114 = t38 - t68;
    const float t115 = t43 - t61; const float t116 = t44 - t62;
    const float t117 = t49 - t55; const float t118 = t50 - t56;
    const float t119 = t31 + t107 + t109 + t111; const float t120 = t32 + t108 + t110 + t112;
    const float t121 = fmaf(t111, -0.90096886790241903f, fmaf(t109, -0.22252093395631434f, fmaf(t107, 0.62348980185873359f, t31))); const float t122 = fmaf(t112, -0.90096886790241903f, fmaf(t110, -0.22252093395631434f, fmaf(t108, 0.62348980185873359f, t32)));
    const float t123 = fmaf(t117, 0.43388373911755823f, fmaf(t115, 0.97492791218182362f, t113 * 0.7818314824680298f)); const float t124 = fmaf(t118, 0.43388373911755823f, fmaf(t116, 0.97492791218182362f, t114 * 0.7818314824680298f));
    const float t125 = t121 - t124; const float t126 = t122 + t123;
    const float t127 = t121 + t124; const float t128 = t122 - t123;
    const float t129 = fmaf(t111, 0.62348980185873337f, fmaf(t109, -0.90096886790241915f, fmaf(t107, -0.22252093395631434f, t31))); const float t130 = fmaf(t112, 0.62348980185873337f, fmaf(t110, -0.90096886790241915f, fmaf(t108, -0.22252093395631434f, t32)));
    const float t131 = fmaf(t117, -0.78183148246802991f, fmaf(t115, -0.43388373911755801f, t113 * 0.97492791218182362f)); const float t132 = fmaf(t118, -0.78183148246802991f, fmaf(t116, -0.43388373911755801f, t114 * 0.97492791218182362f));
    const float t133 = t129 - t132; const float t134 = t130 + t131;
    const float t135 = t129 + t132; const float t136 = t130 - t131;
    const float t137 = fmaf(t111, -0.22252093395631409f, fmaf(t109, 0.62348980185873337f, fmaf(t107, -0.90096886790241903f, t31))); const float t138 = fmaf(t112, -0.22252093395631409f, fmaf(t110, 0.62348980185873337f, fmaf(t108, -0.90096886790241903f, t32)));
    const float t139 = fmaf(t117, 0.97492791218182373f, fmaf(t115, -0.78183148246802991f, t113 * 0.43388373911755823f)); const float t140 = fmaf(t118, 0.97492791218182373f, fmaf(t116, -0.78183148246802991f, t114 * 0.43388373911755823f));
    const float t141 = t137 - t140; const float t142 = t138 + t139;
    const float t143 = t137 + t140; const float t144 = t138 - t139;
    v[0] = make_float2(t81, t82);
    v[1] = make_float2(t119, t120);
    v[2] = make_float2(t87, t88);
    v[3] = make_float2(t125, t126);
    v[4] = make_float2(t95, t96);
    v[5] = make_float2(t133, t134);
    v[6] = make_float2(t103, t104);
    v[7] = make_float2(t141, t142);
    v[8] = make_float2(t105, t106);
    v[9] = make_float2(t143, t144);
    v[10] = make_float2(t97, t98);
    v[11] = make_float2(t135, t136);
    v[12] = make_float2(t89, t90);
    v[13] = make_float2(t127, t128);
  }
};

template <> struct Dft<15, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[15]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = v[13].x; const float t28 = v[13].y;
    const float t29 = v[14].x; const float t30 = v[14].y;
    const float t31 = t11 + t21; const float t32 = t12 + t22;
    const float t33 = t11 - t21; const float t34 = t12 - t22;
    const float t35 = t1 + t31; const float t36 = t2 + t32;
    const float t37 = fmaf(t31, -0.49999999999999978f, t1); const float t38 = fmaf(t32, -0.49999999999999978f, t2);
    const float t39 = t33 * 0.86602540378443871f; const float t40 = t34 * 0.86602540378443871f;
    const float t41 = t37 + t40; const float t42 = t38 - t39;
    const float t43 = t37 - t40; const float t44 = t38 + t39;
    const float t45 = t13 + t23; const float t46 = t14 + t24;
    const float t47 = t13 - t23; const float t48 = t14 - t24;
    const float t49 = t3 + t45; const float t50 = t4 + t46;
    const float t51 = fmaf(t45, -0.49999999999999978f, t3); const float t52 = fmaf(t46, -0.49999999999999978f, t4);
    const float t53 = t47 * 0.86602540378443871f; const float t54 = t48 * 0.86602540378443871f;
    const float t55 = t51 + t54; const float t56 = t52 - t53;
    const float t57 = t51 - t54; const float t58 = t52 + t53;
    const float t59 = fmaf(t55, 0.91354545764260087f, -t56 * -0.40673664307580015f); const float t60 = fmaf(t55, -0.40673664307580015f, t56 * 0.91354545764260087f);
    const float t61 = fmaf(t57, 0.66913060635885824f, -t58 * -0.74314482547739413f); const float t62 = fmaf(t57, -0.74314482547739413f, t58 * 0.66913060635885824f);
    const float t63 = t15 + t25; const float t64 = t16 + t26;
    const float t65 = t15 - t25; const float t66 = t16 - t26;
    const float t67 = t5 + t63; const float t68 = t6 + t64;
    const float t69 = fmaf(t63, -0.49999999999999978f, t5); const float t70 = fmaf(t64, -0.49999999999999978f, t6);
    const float t71 = t65 * 0.86602540378443871f; const float t72 = t66 * 0.86602540378443871f;
    const float t73 = t69 + t72; const float t74 = t70 - t71;
    const float t75 = t69 - t72; const float t76 = t70 + t71;
    const float t77 = fmaf(t73, 0.66913060635885824f, -t74 * -0.74314482547739413f); const float t78 = fmaf(t73, -0.74314482547739413f, t74 * 0.66913060635885824f);
    const float t79 = fmaf(t75, -0.10452846326765333f, -t76 * -0.9945218953682734f); const float t80 = fmaf(t75, -0.9945218953682734f, t76 * -0.10452846326765333f);
    const float t81 = t17 + t27; const float t82 = t18 + t28;
    const float t83 = t17 - t27; const float t84 = t18 - t28;
    const float t85 = t7 + t81; const float t86 = t8 + t82;
    const float t87 = fmaf(t81, -0.49999999999999978f, t7); const float t88 = fmaf(t82, -0.49999999999999978f, t8);
    const float t89 = t83 * 0.86602540378443871f; const float t90 = t84 * 0.86602540378443871f;
    const float t91 = t87 + t90; const float t92 = t88 - t89;
    const float t93 = t87 - t90; const float t94 = t88 + t89;
    const float t95 = fmaf(t91, 0.30901699437494745f, -t92 * -0.95105651629515353f); const float t96 = fmaf(t91, -0.95105651629515353f, t92 * 0.30901699437494745f);
    const float t97 = fmaf(t93, -0.80901699437494734f, -t94 * -0.58778525229247325f); const float t98 = fmaf(t93, -0.58778525229247325f, t94 * -0.80901699437494734f);
    const float t99 = t19 + t29; const float t100 = t20 + t30;
    const float t101 = t19 - t29; const float t102 = t20 - t30;
    const float t103 = t9 + t99; const float t104 = t10 + t100;
    const float t105 = fmaf(t99, -0.49999999999999978f, t9); const float t106 = fmaf(t100, -0.49999999999999978f, t10);
    const float t107 = t101 * 0.86602540378443871f; const float t108 = t102 * 0.86602540378443871f;
    const float t109 = t105 + t108; const float t110 = t106 - t107;
    const float t111 = t105 - t108; const float t112 = t106 + t107;
    const float t113 = fmaf(t109, -0.10452846326765333f, -t110 * -0.9945218953682734f); const float t114 = fmaf(t109, -0.9945218953682734f, t110 * -0.10452846326765333f);
    const float t115 = fmaf(t111, -0.97814760073380569f, -t112 * 0.20791169081775907f); const float t116 = fmaf(t111, 0.20791169081775907f, t112 * -0.97814760073380569f);
    const float t117 = t49 + t103; const float t118 = t50 + t104;
    const float t119 = t67 + t85; const float t120 = t68 + t86;
    const float t121 = t49 - t103; const float t122 = t50 - t104;
    const float t123 = t67 - t85; const float t124 = t68 - t86;
    const float t125 = t35 + t117 + t119; const float t126 = t36 + t118 + t120;
    const float t127 = fmaf(t119, -0.80901699437494734f, fmaf(t117, 0.30901699437494745f, t35)); const float t128 = fmaf(t120, -0.80901699437494734f, fmaf(t118, 0.30901699437494745f, t36));
    const float t129 = fmaf(t123, 0.58778525229247325f, t121 * 0.95105651629515353f); const float t130 = fmaf(t124, 0.58778525229247325f, t122 * 0.95105651629515353f);
    const float t131 = t127 + t130; const float t132 = t128 - t129;
    const float t133 = t127 - t130; const float t134 = t128 + t129;
    const float t135 = fmaf(t119, 0.30901699437494723f, fmaf(t117, -0.80901699437494734f, t35)); const float t136 = fmaf(t120, 0.30901699437494723f, fmaf(t118, -0.80901699437494734f, t36));
    const float t137 = fmaf(t123, -0.95105651629515364f, t121 * 0.58778525229247325f); const float t138 = fmaf(t124, -0.95105651629515364f, t122 * 0.58778525229247325f);
    const float t139 = t135 + t138; const float t140 = t136 - t137;
    const float t141 = t135 - t138; const float t142 = t136 + t137;
    const float t143 = t59 + t113; const float t144 = t60 + t114;
    const float t145 = t77 + t95; const float t146 = t78 + t96;
    const float t147 = t59 - t113; const float t148 = t60 - t114;
    const float t149 = t77 - t95; const float t150 = t78 - t96;
    const float t151 = t41 + t143 + t145; const float t152 = t42 + t144 + t146;
    const float t153 = fmaf(t145, -0.80901699437494734f, fmaf(t143, 0.30901699437494745f, t41)); const float t154 = fmaf(t146, -0.80901699437494734f, fmaf(t144, 0.30901699437494745f, t42));
    const float t155 = fmaf(t149, 0.58778525229247325f, t147 * 0.95105651629515353f); const float t156 = fmaf(t150, 0.58778525229247325f, t148 * 0.95105651629515353f);
    const float t157 = t153 + t156; const float t158 = t154 - t155;
    const float t159 = t153 - t156; const float t160 = t154 + t155;
    const float t161 = fmaf(t145, 0.30901699437494723f, fmaf(t143, -0.80901699437494734f, t41)); const float t162 = fmaf(t146, 0.30901699437494723f, fmaf(t144, -0.80901699437494734f, t42));
    const float t163 = fmaf(t149, -0.95105651629515364f, t147 * 0.58778525229247325f); const float t164 = fmaf(t150, -0.95105651629515364f, t148 * 0.58778525229247325f);
    const float t165 = t161 + t164; const float t166 = t162 - t163;
    const float t167 = t161 - t164; const float t168 = t162 + t163;
    const float t169 = t61 + t115; const float t170 = t62 + t116;
    const float t171 = t79 + t97; const float t172 = t80 + t98;
    const float t173 = t61 - t115; const float t174 = t62 - t116;
    const float t175 = t79 - t97; const float t176 = t80 - t98;
    const float t177 = t43 + t169 + t171; const float t178 = t44 + t170 + t172;
    const float t179 = fmaf(t171, -0.80901699437494734f, fmaf(t169, 0.30901699437494745f, t43)); const float t180 = fmaf(t172, -0.80901699437494734f, fmaf(t170, 0.30901699437494745f, t44));
    const float t181 = fmaf(t175, 0.58778525229247325f, t173 * 0.95105651629515353f); const float t182 = fmaf(t176, 0.58778525229247325f, t174 * 0.95105651629515353f);
    const float t183 = t179 + t182; const float t184 = t180 - t181;
    const float t185 = t179 - t182; const float t186 = t180 + t181;
    const float t187 = fmaf(t171, 0.30901699437494723f, fmaf(t169, -0.80901699437494734f, t43)); const float t188 = fmaf(t172, 0.30901699437494723f, fmaf(t170, -0.80901699437494734f, t44));
    const float t189 = fmaf(t175, -0.95105651629515364f, t173 * 0.58778525229247325f); const float t190 = fmaf(t176, -0.95105651629515364f, t174 * 0.58778525229247325f);
    const float t191 = t187 + t190; const float t192 = t188 - t189;
    const float t193 = t187 - t190; const float t194 = t188 + t189;
    v[0] = make_float2(t125, t126);
    v[1] = make_float2(t151, t152);
    v[2] = make_float2(t177, t178);
    v[3] = make_float2(t131, t132);
    v[4] = make_float2(t157, t158);
    v[5] = make_float2(t183, t184);
    v[6] = make_float2(t139, t140);
    v[7] = make_float2(t165, t166);
    v[8] = make_float2(t191, t192);
    v[9] = make_float2(t141, t142);
    v[10] = make_float2(t167, t168);
    v[11] = make_float2(t193, t194);
    v[12] = make_float2(t133, t134);
    v[13] = make_float2(t159, t160);
    v[14] = make_float2(t185, t186);
  }
};

template <> struct Dft<15, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[15]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = v[13].x; const float t28 = v[13].y;
    const float t29 = v[14].x; const float t30 = v[14].y;
    const float t31 = t11 + t21; const float t32 = t12 + t22;
    const float t33 = t11 - t21; const float t34 = t12 - t22;
    const float t35 = t1 + t31; const float t36 = t2 + t32;
    const float t37 = fmaf(t31, -0.49999999999999978f, t1); const float t38 = fmaf(t32, -0.49999999999999978f, t2);
    const float t39 = t33 * 0.86602540378443871f; const float t40 = t34 * 0.86602540378443871f;
    const float t41 = t37 - t40; const float t42 = t38 + t39;
    const float t43 = t37 + t40; const float t44 = t38 - t39;
    const float t45 = t13 + t23; const float t46 = t14 + t24;
    const float t47 = t13 - t23; const float t48 = t14 - t24;
    const float t49 = t3 + t45; const float t50 = t4 + t46;
    const float t51 = fmaf(t45, -0.49999999999999978f, t3); const float t52 = fmaf(t46, -0.49999999999999978f, t4);
    const float t53 = t47 * 0.86602540378443871f; const float t54 = t48 * 0.86602540378443871f;
    const float t55 = t51 - t54; const float t56 = t52 + t53;
    const float t57 = t51 + t54; const float t58 = t52 - t53;
    const float t59 = fmaf(t55, 0.91354545764260087f, -t56 * 0.40673664307580015f); const float t60 = fmaf(t55, 0.40673664307580015f, t56 * 0.91354545764260087f);
    const float t61 = fmaf(t57, 0.66913060635885824f, -t58 * 0.74314482547739413f); const float t62 = fmaf(t57, 0.74314482547739413f, t58 * 0.66913060635885824f);
    const float t63 = t15 + t25; const float t64 = t16 + t26;
    const float t65 = t15 - t25; const float t66 = t16 - t26;
    const float t67 = t5 + t63; const float t68 = t6 + t64;
    const float t69 = fmaf(t63, -0.49999999999999978f, t5); const float t70 = fmaf(t64, -0.49999999999999978f, t6);
    const float t71 = t65 * 0.86602540378443871f; const float t72 = t66 * 0.86602540378443871f;
    const float t73 = t69 - t72; const float t74 = t70 + t71;
    const float t75 = t69 + t72; const float t76 = t70 - t71;
    const float t77 = fmaf(t73, 0.66913060635885824f, -t74 * 0.74314482547739413f); const float t78 = fmaf(t73, 0.74314482547739413f, t74 * 0.66913060635885824f);
    const float t79 = fmaf(t75, -0.10452846326765333f, -t76 * 0.9945218953682734f); const float t80 = fmaf(t75, 0.9945218953682734f, t76 * -0.10452846326765333f);
    const float t81 = t17 + t27; const float t82 = t18 + t28;
    const float t83 = t17 - t27; const float t84 = t18 - t28;
    const float t85 = t7 + t81; const float t86 = t8 + t82;
    const float t87 = fmaf(t81, -0.49999999999999978f, t7); const float t88 = fmaf(t82, -0.49999999999999978f, t8);
    const float t89 = t83 * 0.86602540378443871f; const float t90 = t84 * 0.86602540378443871f;
    const float t91 = t87 - t90; const float t92 = t88 + t89;
    const float t93 = t87 + t90; const float t94 = t88 - t89;
    const float t95 = fmaf(t91, 0.30901699437494745f, -t92 * 0.95105651629515353f); const float t96 = fmaf(t91, 0.95105651629515353f, t92 * 0.30901699437494745f);
    const float t97 = fmaf(t93, -0.80901699437494734f, -t94 * 0.58778525229247325f); const float t98 = fmaf(t93, 0.58778525229247325f, t94 * -0.80901699437494734f);
    const float t99 = t19 + t29; const float t100 = t20 + t30;
    const float t101 = t19 - t29; const float t102 = t20 - t30;
    const float t103 = t9 + t99; const float t104 = t10 + t100;
    const float t105 = fmaf(t99, -0.49999999999999978f, t9); const float t106 = fmaf(t100, -0.49999999999999978f, t10);
    const float t107 = t101 * 0.86602540378443871f; const float t108 = t102 * 0.86602540378443871f;
    const float t109 = t105 - t108; const float t110 = t106 + t107;
    const float t111 = t105 + t108; const float t112 = t106 - t107;
    const float t113 = fmaf(t109, -0.10452846326765333f, -t110 * 0.9945218953682734f); const float t114 = fmaf(t109, 0.9945218953682734f, t110 * -0.10452846326765333f);
    const float t115 = fmaf(t111, -0.97814760073380569f, -t112 * -0.20791169081775907f); const float t116 = fmaf(t111, -0.20791169081775907f, t112 * -0.97814760073380569f);
    const float t117 = t49 + t103; const float t118 = t50 + t104;
    const float t119 = t67 + t85; const float t120 = t68 + t86;
    const float t121 = t49 - t103; const float t122 = t50 - t104;
    const float t123 = t67 - t85; const float t124 = t68 - t86;
    const float t125 = t35 + t117 + t119; const float t126 = t36 + t118 + t120;
    const float t127 = fmaf(t119, -0.80901699437494734f, fmaf(t117, 0.30901699437494745f, t35)); const float t128 = fmaf(t120, -0.80901699437494734f, fmaf(t118, 0.30901699437494745f, t36));
    const float t129 = fmaf(t123, 0.58778525229247325f, t121 * 0.95105651629515353f); const float t130 = fmaf(t124, 0.58778525229247325f, t122 * 0.95105651629515353f);
    const float t131 = t127 - t130; const float t132 = t128 + t129;
    const float t133 = t127 + t130; const float t134 = t128 - t129;
    const float t135 = fmaf(t119, 0.30901699437494723f, fmaf(t117, -0.80901699437494734f, t35)); const float t136 = fmaf(t120, 0.30901699437494723f, fmaf(t118, -0.80901699437494734f, t36));
    const float t137 = fmaf(t123, -0.95105651629515364f, t121 * 0.58778525229247325f); const float t138 = fmaf(t124, -0.95105651629515364f, t122 * 0.58778525229247325f);
    const float t139 = t135 - t138; const float t140 = t136 + t137;
    const float t141 = t135 + t138; const float t142 = t136 - t137;
    const float t143 = t59 + t113; const float t144 = t60 + t114;
    const float t145 = t77 + t95; const float t146 = t78 + t96;
    const float t147 = t59 - t113; const float t148 = t60 - t114;
    const float t149 = t77 - t95; const float t150 = t78 - t96;
    const float t151 = t41 + t143 + t145; const float t152 = t42 + t144 + t146;
    const float t153 = fmaf(t145, -0.80901699437494734f, fmaf(t143, 0.30901699437494745f, t41)); const float t154 = fmaf(t146, -0.80901699437494734f, fmaf(t144, 0.30901699437494745f, t42));
    const float t155 = fmaf(t149, 0.58778525229247325f, t147 * 0.95105651629515353f); const float t156 = fmaf(t150, 0.58778525229247325f, t148 * 0.95105651629515353f);
    const float t157 = t153 - t156; const float t158 = t154 + t155;
    const float t159 = t153 + t156; const float t160 = t154 - t155;
    const float t161 = fmaf(t145, 0.30901699437494723f, fmaf(t143, -0.80901699437494734f, t41)); const float t162 = fmaf(t146, 0.30901699437494723f, fmaf(t144, -0.80901699437494734f, t42));
    const float t163 = fmaf(t149, -0.95105651629515364f, t147 * 0.58778525229247325f); const float t164 = fmaf(t150, -0.95105651629515364f, t148 * 0.58778525229247325f);
    const float t165 = t161 - t164; const float t166 = t162 + t163;
    const float t167 = t161 + t164; const float t168 = t162 - t163;
    const float t169 = t61 + t115; const float t170 = t62 + t116;
    const float t171 = t79 + t97; const float t172 = t80 + t98;
    const float t173 = t61 - t115; const float t174 = t62 - t116;
    const float t175 = t79 - t97; const float t176 = t80 - t98;
    const float t177 = t43 + t169 + t171; const float t178 = t44 + t170 + t172;
    const float t179 = fmaf(t171, -0.80901699437494734f, fmaf(t169, 0.30901699437494745f, t43)); const float t180 = fmaf(t172, -0.80901699437494734f, fmaf(t170, 0.30901699437494745f, t44));
    const float t181 = fmaf(t175, 0.58778525229247325f, t173 * 0.95105651629515353f); const float t182 = fmaf(t176, 0.58778525229247325f, t174 * 0.95105651629515353f);
    const float t183 = t179 - t182; const float t184 = t180 + t181;
    const float t185 = t179 + t182; const float t186 = t180 - t181;
    const float t187 = fmaf(t171, 0.30901699437494723f, fmaf(t169, -0.80901699437494734f, t43)); const float t188 = fmaf(t172, 0.30901699437494723f, fmaf(t170, -0.80901699437494734f, t44));
    const float t189 = fmaf(t175, -0.95105651629515364f, t173 * 0.58778525229247325f); const float t190 = fmaf(t176, -0.95105651629515364f, t174 * 0.58778525229247325f);
    const float t191 = t187 - t190; const float t192 = t188 + t189;
    const float t193 = t187 + t190; const float t194 = t188 - t189;
    v[0] = make_float2(t125, t126);
    v[1] = make_float2(t151, t152);
    v[2] = make_float2(t177, t178);
    v[3] = make_float2(t131, t132);
    v[4] = make_float2(t157, t158);
    v[5] = make_float2(t183, t184);
    v[6] = make_float2(t139, t140);
    v[7] = make_float2(t165, t166);
    v[8] = make_float2(t191, t192);
    v[9] = make_float2(t141, t142);
    v[10] = make_float2(t167, t168);
    v[11] = make_float2(t193, t194);
    v[12] = make_float2(t133, t134);
    v[13] = make_float2(t159, t160);
    v[14] = make_float2(t185, t186);
  }
};

template <> struct Dft<16, false> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[16]) {  // fwd
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = v[13].x; const float t28 = v[13].y;
    const float t29 = v[14].x; const float t30 = v[14].y;
    const float t31 = v[15].x; const float t32 = v[15].y;
    const float t33 = t1 + t17; const float t34 = t2 + t18;
    const float t35 = t1 - t17; const float t36 = t2 - t18;
    const float t37 = t9 + t25; const float t38 = t10 + t26;
    const float t39 = t9 - t25; const float t40 = t10 - t26;
    const float t41 = t40; const float t42 = -t39;
    const float t43 = t33 + t37; const float t44 = t34 + t38;
    const float t45 = t33 - t37; const float t46 = t34 - t38;
    const float t47 = t35 + t41; const float t48 = t36 + t42;
    const float t49 = t35 - t41; const float t50 = t36 - t42;
    const float t51 = t3 + t19; const float t52 = t4 + t20;
    const float t53 = t3 - t19; const float t54 = t4 - t20;
    const float t55 = t11 + t27; const float t56 = t12 + t28;
    const float t57 = t11 - t27; const float t58 = t12 - t28;
    const float t59 = t58; const float t60 = -t57;
    const float t61 = t51 + t55; const float t62 = t52 + t56;
    const float t63 = t51 - t55; const float t64 = t52 - t56;
    const float t65 = t53 + t59; const float t66 = t54 + t60;
    const float t67 = t53 - t59; const float t68 = t54 - t60;
    const float t69 = fmaf(t65, 0.92387953251128674f, -t66 * -0.38268343236508978f); const float t70 = fmaf(t65, -0.38268343236508978f, t66 * 0.92387953251128674f);
    const float t71 = 0.70710678118654752f * (t63 + t64); const float t72 = 0.70710678118654752f * (t64 - t63);
    const float t73 = fmaf(t67, 0.38268343236508984f, -t68 * -0.92387953251128674f); const float t74 = fmaf(t67, -0.92387953251128674f, t68 * 0.38268343236508984f);
    const float t75 = t5 + t21; const float t76 = t6 + t22;
    const float t77 = t5 - t21; const float t78 = t6 - t22;
    const float t79 = t13 + t29; const float t80 = t14 + t30;
    const float t81 = t13 - t29; const float t82 = t14 - t30;
    const float t83 = t82; const float t84 = -t81;
    const float t85 = t75 + t79; const float t86 = t76 + t80;
    const float t87 = t75 - t79; const float t88 = t76 - t80;
    const float t89 = t77 + t83; const float t90 = t78 + t84;
    const float t91 = t77 - t83; const float t92 = t78 - t84;
    const float t93 = 0.70710678118654752f * (t89 + t90); const float t94 = 0.70710678118654752f * (t90 - t89);
    const float t95 = t88; const float t96 = -t87;
    const float t97 = 0.70710678118654752f * (t92 - t91); const float t98 = -0.70710678118654752f * (t91 + t92);
    const float t99 = t7 + t23; const float t100 = t8 + t24;
    const float t101 = t7 - t23; const float t102 = t8 - t24;
    const float t103 = t15 + t31; const float t104 = t16 + t32;
    const float t105 = t15 - t31; const float t106 = t16 - t32;
    const float t107 = t106; const float t108 = -t105;
    const float t109 = t99 + t103; const float t110 = t100 + t104;
    const float t111 = t99 - t103; const float t112 = t100 - t104;
    const float t113 = t101 + t107; const float t114 = t102 + t108;
    const float t115 = t101 - t107; const float t116 = t102 - t108;
    const float t117 = fmaf(t113, 0.38268343236508984f, -t114 * -0.92387953251128674f); const float t118 = fmaf(t113, -0.92387953251128674f, t114 * 0.38268343236508984f);
    const float t119 = 0.70710678118654752f * (t112 - t111); const float t120 = -0.70710678118654752f * (t111 + t112);
    const float t121 = fmaf(t115, -0.92387953251128685f, -t116 * 0.38268343236508967f); const float t122 = fmaf(t115, 0.38268343236508967f, t116 * -0.92387953251128685f);
    const float t123 = t43 + t85; const float t124 = t44 + t86;
    const float t125 = t43 - t85; const float t126 = t44 - t86;
    const float t127 = t61 + t109; const float t128 = t62 + t110;
    const float t129 = t61 - t109; const float t130 = t62 - t110;
    const float t131 = t130; const float t132 = -t129;
    const float t133 = t123 + t127; const float t134 = t124 + t128;
    const float t135 = t123 - t127; const float t136 = t124 - t128;
    const float t137 = t125 + t131; const float t138 = t126 + t132;
    const float t139 = t125 - t131; const float t140 = t126 - t132;
    const float t141 = t47 + t93; const float t142 = t48 + t94;
    const float t143 = t47 - t93; const float t144 = t48 - t94;
    const float t145 = t69 + t117; const float t146 = t70 + t118;
    const float t147 = t69 - t117; const float t148 = t70 - t118;
    const float t149 = t148; const float t150 = -t147;
    const float t151 = t141 + t145; const float t152 = t142 + t146;
    const float t153 = t141 - t145; const float t154 = t142 - t146;
    const float t155 = t143 + t149; const float t156 = t144 + t150;
    const float t157 = t143 - t149; const float t158 = t144 - t150;
    const float t159 = t45 + t95; const float t160 = t46 + t96;
    const float t161 = t45 - t95; const float t162 = t46 - t96;
    const float t163 = t71 + t119; const float t164 = t72 + t120;
    const float t165 = t71 - t119; const float t166 = t72 - t120;
    const float t167 = t166; const float t168 = -t165;
    const float t169 = t159 + t163; const float t170 = t160 + t164;
    const float t171 = t159 - t163; const float t172 = t160 - t164;
    const float t173 = t161 + t167; const float t174 = t162 + t168;
    const float t175 = t161 - t167; const float t176 = t162 - t168;
    const float t177 = t49 + t97; const float t178 = t50 + t98;
    const float t179 = t49 - t97; const float t180 = t50 - t98;
    const float t181 = t73 + t121; const float t182 = t74 + t122;
    const float t183 = t73 - t121; const float t184 = t74 - t122;
    const float t185 = t184; const float t186 = -t183;
    const float t187 = t177 + t181; const float t188 = t178 + t182;
    const float t189 = t177 - t181; const float t190 = t178 - t182;
    const float t191 = t179 + t185; const float t192 = t180 + t186;
    const float t193 = t179 - t185; const float t194 = t180 - t186;
    v[0] = make_float2(t133, t134);
    v[1] = make_float2(t151, t152);
    v[2] = make_float2(t169, t170);
    v[3] = make_float2(t187, t188);
    v[4] = make_float2(t137, t138);
    v[5] = make_float2(t155, t156);
    v[6] = make_float2(t173, t174);
    v[7] = make_float2(t191, t192);
    v[8] = make_float2(t135, t136);
    v[9] = make_float2(t153, t154);
    v[10] = make_float2(t171, t172);
    v[11] = make_float2(t189, t190);
    v[12] = make_float2(t139, t140);
    v[13] = make_float2(t157, t158);
    v[14] = make_float2(t175, t176);
    v[15] = make_float2(t193, t194);
  }
};

template <> struct Dft<16, true> {
  static __host__ __device__ __forceinline__ void run(float2 (&v)[16]) {  // inv
    const float t1 = v[0].x; const float t2 = v[0].y;
    const float t3 = v[1].x; const float t4 = v[1].y;
    const float t5 = v[2].x; const float t6 = v[2].y;
    const float t7 = v[3].x; const float t8 = v[3].y;
    const float t9 = v[4].x; const float t10 = v[4].y;
    const float t11 = v[5].x; const float t12 = v[5].y;
    const float t13 = v[6].x; const float t14 = v[6].y;
    const float t15 = v[7].x; const float t16 = v[7].y;
    const float t17 = v[8].x; const float t18 = v[8].y;
    const float t19 = v[9].x; const float t20 = v[9].y;
    const float t21 = v[10].x; const float t22 = v[10].y;
    const float t23 = v[11].x; const float t24 = v[11].y;
    const float t25 = v[12].x; const float t26 = v[12].y;
    const float t27 = v[13].x; const float t28 = v[13].y;
    const float t29 = v[14].x; const float t30 = v[14].y;
    const float t31 = v[15].x; const float t32 = v[15].y;
    const float t33 = t1 + t17; const float t34 = t2 + t18;
    const float t35 = t1 - t17; const float t36 = t2 - t18;
    const float t37 = t9 + t25; const float t38 = t10 + t26;
    const float t39 = t9 - t25; const float t40 = t10 - t26;
    const float t41 = -t40; const float t42 = t39;
    const float t43 = t33 + t37; const float t44 = t34 + t38;
    const float t45 = t33 - t37; const float t46 = t34 - t38;
    const float t47 = t35 + t41; const float t48 = t36 + t42;
    const float t49 = t35 - t41; const float t50 = t36 - t42;
    const float t51 = t3 + t19; const float t52 = t4 + t20;
    const float t53 = t3 - t19; const float t54 = t4 - t20;
    const float t55 = t11 + t27; const float t56 = t12 + t28;
    const float t57 = t11 - t27; const float t58 = t12 - t28;
    const float t59 = -t58; const float t60 = t57;
    const float t61 = t51 + t55; const float t62 = t52 + t56;
    const float t63 = t51 - t55; const float t64 = t52 - t56;
    const float t65 = t53 + t59; const float t66 = t54 + t60;
    const float t67 = t53 - t59; const float t68 = t54 - t60;
    const float t69 = fmaf(t65, 0.92387953251128674f, -t66 * 0.38268343236508978f); const float t70 = fmaf(t65, 0.38268343236508978f, t66 * 0.92387953251128674f);
    const float t71 = 0.70710678118654752f * (t63 - t64); const float t72 = 0.70710678118654752f * (t63 + t64);
    const float t73 = fmaf(t67, 0.38268343236508984f, -t68 * 0.92387953251128674f); const float t74 = fmaf(t67, 0.92387953251128674f, t68 * 0.38268343236508984f);
    const float t75 = t5 + t21; const float t76 = t6 + t22;
    const float t77 = t5 - t21; const float t78 = t6 - t22;
    const float t79 = t13 + t29; const float t80 = t14 + t30;
    const float t81 = t13 - t29; const float t82 = t14 - t30;
    const float t83 = -t82; const float t84 = t81;
    const float t85 = t75 + t79; const float t86 = t76 + t80;
    const float t87 = t75 - t79; const float t88 = t76 - t80;
    const float t89 = t77 + t83; const float t90 = t78 + t84;
    const float t91 = t77 - t83; const float t92 = t78 - t84;
    const float t93 = 0.70710678118654752f * (t89 - t90); const float t94 = 0.70710678118654752f * (t89 + t90);
    const float t95 = -t88; const float t96 = t87;
    const float t97 = -0.70710678118654752f * (t91 + t92); const float t98 = 0.70710678118654752f * (t91 - t92);
    const float t99 = t7 + t23; const float t100 = t8 + t24;
    const float t101 = t7 - t23; const float t102 = t8 - t24;
    const float t103 = t15 + t31; const float t104 = t16 + t32;
    const float t105 = t15 - t31; const float t106 = t16 - t32;
    const float t107 = -t106; const float t108 = t105;
    const float t109 = t99 + t103; const float t110 = t100 + t104;
    const float t111 = t99 - t103; const float t112 = t100 - t104;
    const float t113 = t101 + t107; const float t114 = t102 + t108;
    const float t115 = t101 - t107; const float t116 = t102 - t108;
    const float t117 = fmaf(t113, 0.38268343236508984f, -t114 * 0.92387953251128674f); const float t118 = fmaf(t113, 0.92387953251128674f, t114 * 0.38268343236508984f);
    const float t119 = -0.70710678118654752f * (t111 + t112); const float t120 = 0.70710678118654752f * (t111 - t112);
    const float t121 = fmaf(t115, -0.92387953251128685f, -t116 * -0.38268343236508967f); const float t122 = fmaf(t115, -0.38268343236508967f, t116 * -0.92387953251128685f);
    const float t123 = t43 + t85; const float t124 = t44 + t86;
    const float t125 = t43 - t85; const float t126 = t44 - t86;
    const float t127 = t61 + t109; const float t128 = t62 + t110;
    const float t129 = t61 - t109; const float t130 = t62 - t110;
    const float t131 = -t130; const float t132 = t129;
    const float t133 = t123 + t127; const float t134 = t124 + t128;
    const float t135 = t123 - t127; const float t136 = t124 - t128;
    const float t137 = t125 + t131; const float t138 = t126 + t132;
    const float t139 = t125 - t131; const float t140 = t126 - t132;
    const float t141 = t47 + t93; const float t142 = t48 + t94;
    const float t143 = t47 - t93; const float t144 = t48 - t94;
    const float t145 = t69 + t117; const float t146 = t70 + t118;
    const float t147 = t69 - t117; const float t148 = t70 - t118;
    const float t149 = -t148; const float t150 = t147;
    const float t151 = t141 + t145; const float t152 = t142 + t146;
    const float t153 = t141 - t145; const float t154 = t142 - t146;
    const float t155 = t143 + t149; const float t156 = t144 + t150;
    const float t157 = t143 - t149; const float t158 = t144 - t150;
    const float t159 = t45 + t95; const float t160 = t46 + t96;
    const float t161 = t45 - t95; const float t162 = t46 - t96;
    const float t163 = t71 + t119; const float t164 = t72 + t120;
    const float t165 = t71 - t119; const float t166 = t72 - t120;
    const float t167 = -t166; const float t168 = t165;
    const float t169 = t159 + t163; const float t170 = t160 + t164;
    const float t171 = t159 - t163; const float t172 = t160 - t164;
    const float t173 = t161 + t167; const float t174 = t162 + t168;
    const float t175 = t161 - t167; const float t176 = t162 - t168;
    const float t177 = t49 + t97; const float t178 = t50 + t98;
    const float t179 = t49 - t97; const float t180 = t50 - t98;
    const float t181 = t73 + t121; const float t182 = t74 + t122;
    const float t183 = t73 - t121; const float t184 = t74 - t122;
    const float t185 = -t184; const float t186 = t183;
    const float t187 = t177 + t181; const float t188 = t178 + t182;
    const float t189 = t177 - t181; const float t190 = t178 - t182;
    const float t191 = t179 + t185; const float t192 = t180 + t186;
    const float t193 = t179 - t185; const float t194 = t180 - t186;
    v[0] = make_float2(t133, t134);
    v[1] = make_float2(t151, t152);
    v[2] = make_float2(t169, t170);
    v[3] = make_float2(t187, t188);
    v[4] = make_float2(t137, t138);
    v[5] = make_float2(t155, t156);
    v[6] = make_float2(t173, t174);
    v[7] = make_float2(t191, t192);
    v[8] = make_float2(t135, t136);
    v[9] = make_float2(t153, t154);
    v[10] = make_float2(t171, t172);
    v[11] = make_float2(t189, t190);
    v[12] = make_float2(t139, t140);
    v[13] = make_float2(t157, t158);
    v[14] = make_float2(t175, t176);
    v[15] = make_float2(t193, t194);
  }
};

constexpr int kNumRadices = 15;
constexpr int kRadices[kNumRadices] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16};

// The butterflies' constants are rounded to single precision: the real part of their matrices' relative error,
// averaged; which = 0, 1: the forward one by input i, by output i; 2, 3: the inverse one.
inline double butterfly_gain(int which, int R, int i) {
  constexpr double g[4][17][16] = {
      {
          {},
          {},
          {0, 0},
          {0, -8.974116e-09, -8.974116e-09},
          {0, 0, 0, 0},
          {0, 1.074062e-08, 1.074062e-08, 1.074062e-08, 1.074062e-08},
          {0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08},
          {0, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09},
          {0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09},
          {0, -1.240993e-08, -1.670447e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08},
          {0, 1.162006e-08, 2.328697e-08, 2.328697e-08, 1.162006e-08, 0, 1.162006e-08, 2.328697e-08, 2.328697e-08, 1.162006e-08},
          {0, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09},
          {0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08},
          {0, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10},
          {0, -1.632419e-08, 1.124557e-09, -1.040063e-08, -1.040063e-08, 1.124557e-09, -1.632419e-08, 0, -1.632419e-08, 1.124557e-09, -1.040063e-08, -1.040063e-08, 1.124557e-09, -1.632419e-08},
          {0, 2.107566e-09, 1.759304e-08, 1.969114e-08, 2.540721e-08, -8.974116e-09, -6.866550e-09, 8.618926e-09, 1.071703e-08, 1.643310e-08, -8.974116e-09, -6.866550e-09, 8.618926e-09, 1.071703e-08, 1.643310e-08},
          {0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08},
      },
      {
          {},
          {},
          {0, 0},
          {0, -8.974116e-09, -8.974116e-09},
          {0, 0, 0, 0},
          {0, 1.074062e-08, 1.074062e-08, 1.074062e-08, 1.074062e-08},
          {0, -8.974116e-09, -8.974116e-09, -1.794823e-08, -8.974116e-09, -1.794823e-08},
          {0, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09},
          {0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09},
          {0, -1.240993e-08, -1.670447e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08},
          {0, 1.074062e-08, 1.074062e-08, 2.148125e-08, 1.074062e-08, 2.148125e-08, 1.074062e-08, 2.148125e-08, 1.074062e-08, 2.148125e-08},
          {0, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09},
          {0, -8.974116e-09, -8.974116e-09, 0, -8.974116e-09, -1.794823e-08, -1.794823e-08, -8.974116e-09, -8.974116e-09, -1.794823e-08, -1.794823e-08, -8.974116e-09},
          {0, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10},
          {0, -5.389529e-09, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08},
          {0, -5.025859e-09, 1.795115e-10, 1.074062e-08, 5.714763e-09, 1.092013e-08, 1.074062e-08, 5.714763e-09, 1.092013e-08, 1.074062e-08, 5.714763e-09, 1.092013e-08, 1.074062e-08, 5.714763e-09, 1.092013e-08},
          {0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08},
      },
      {
          {},
          {},
          {0, 0},
          {0, -8.974116e-09, -8.974116e-09},
          {0, 0, 0, 0},
          {0, 1.074062e-08, 1.074062e-08, 1.074062e-08, 1.074062e-08},
          {0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08},
          {0, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09},
          {0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09},
          {0, -1.240993e-08, -1.670447e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08},
          {0, 1.162006e-08, 2.328697e-08, 2.328697e-08, 1.162006e-08, 0, 1.162006e-08, 2.328697e-08, 2.328697e-08, 1.162006e-08},
          {0, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09},
          {0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08, 0, -1.570470e-08, -1.570470e-08},
          {0, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10},
          {0, -1.632419e-08, 1.124557e-09, -1.040063e-08, -1.040063e-08, 1.124557e-09, -1.632419e-08, 0, -1.632419e-08, 1.124557e-09, -1.040063e-08, -1.040063e-08, 1.124557e-09, -1.632419e-08},
          {0, 2.107566e-09, 1.759304e-08, 1.969114e-08, 2.540721e-08, -8.974116e-09, -6.866550e-09, 8.618926e-09, 1.071703e-08, 1.643310e-08, -8.974116e-09, -6.866550e-09, 8.618926e-09, 1.071703e-08, 1.643310e-08},
          {0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08},
      },
      {
          {},
          {},
          {0, 0},
          {0, -8.974116e-09, -8.974116e-09},
          {0, 0, 0, 0},
          {0, 1.074062e-08, 1.074062e-08, 1.074062e-08, 1.074062e-08},
          {0, -8.974116e-09, -8.974116e-09, -1.794823e-08, -8.974116e-09, -1.794823e-08},
          {0, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09, -5.389529e-09},
          {0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09, 0, -8.557136e-09},
          {0, -1.240993e-08, -1.670447e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08, -8.974116e-09, -2.138405e-08, -2.567859e-08},
          {0, 1.074062e-08, 1.074062e-08, 2.148125e-08, 1.074062e-08, 2.148125e-08, 1.074062e-08, 2.148125e-08, 1.074062e-08, 2.148125e-08},
          {0, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09, -3.575949e-09},
          {0, -8.974116e-09, -8.974116e-09, 0, -8.974116e-09, -1.794823e-08, -1.794823e-08, -8.974116e-09, -8.974116e-09, -1.794823e-08, -1.794823e-08, -8.974116e-09},
          {0, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10, 6.025156e-10},
          {0, -5.389529e-09, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08, -5.389529e-09, -1.077906e-08},
          {0, -5.025859e-09, 1.795115e-10, 1.074062e-08, 5.714763e-09, 1.092013e-08, 1.074062e-08, 5.714763e-09, 1.092013e-08, 1.074062e-08, 5.714763e-09, 1.092013e-08, 1.074062e-08, 5.714763e-09, 1.092013e-08},
          {0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08, 0, -1.854571e-08, -8.557136e-09, -1.854571e-08},
      },
  };
  return g[which][R][i];
}
// Forward and inverse butterflies in a row multiply by R (1 + gain), apart from what they mix in of the others:
// side 0 the gain of frequency i (inverse, then forward), 1 that of input i (forward, then inverse).  A literal
// where R and i are known.
__host__ __device__ constexpr double round_trip(int side, int R, int i) {
  constexpr double g[2][17][16] = {
      {
          {},
          {},
          {0, 0},
          {0, -1.794823e-08, -1.794823e-08},
          {0, 0, 0, 0},
          {0, 2.148125e-08, 2.148125e-08, 2.148125e-08, 2.148125e-08},
          {0, -2.467882e-08, -2.467882e-08, -1.794823e-08, -2.467882e-08, -3.365293e-08},
          {0, -1.077906e-08, -1.077906e-08, -1.077906e-08, -1.077906e-08, -1.077906e-08, -1.077906e-08},
          {0, -1.711427e-08, 0, -1.711427e-08, 0, -1.711427e-08, 0, -1.711427e-08},
          {0, -2.481987e-08, -3.340894e-08, -1.794823e-08, -4.276810e-08, -5.135717e-08, -1.794823e-08, -4.276810e-08, -5.135717e-08},
          {0, 2.236068e-08, 3.402759e-08, 4.476821e-08, 2.236068e-08, 2.148125e-08, 2.236068e-08, 4.476821e-08, 3.402759e-08, 3.310130e-08},
          {0, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09},
          {0, -2.467882e-08, -2.467882e-08, 0, -2.467882e-08, -3.365293e-08, -1.794823e-08, -2.467882e-08, -2.467882e-08, -1.794823e-08, -3.365293e-08, -2.467882e-08},
          {0, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09},
          {0, -2.171372e-08, -4.264971e-09, -2.117969e-08, -1.579016e-08, -9.654500e-09, -2.171372e-08, -1.077906e-08, -2.171372e-08, -9.654500e-09, -1.579016e-08, -2.117969e-08, -4.264971e-09, -2.710325e-08},
          {0, -2.918294e-09, 1.777255e-08, 3.043176e-08, 3.112198e-08, 1.946019e-09, 3.874073e-09, 1.433369e-08, 2.163716e-08, 2.717372e-08, -3.259352e-09, 4.053584e-09, 1.935955e-08, 1.643179e-08, 2.735323e-08},
          {0, -3.709142e-08, -1.711427e-08, -3.709142e-08, 0, -3.709142e-08, -1.711427e-08, -3.709142e-08, 0, -3.709142e-08, -1.711427e-08, -3.709142e-08, 0, -3.709142e-08, -1.711427e-08, -3.709142e-08},
      },
      {
          {},
          {},
          {0, 0},
          {0, -1.794823e-08, -1.794823e-08},
          {0, 0, 0, 0},
          {0, 2.148125e-08, 2.148125e-08, 2.148125e-08, 2.148125e-08},
          {0, -2.467882e-08, -2.467882e-08, -1.794823e-08, -2.467882e-08, -3.365293e-08},
          {0, -1.077906e-08, -1.077906e-08, -1.077906e-08, -1.077906e-08, -1.077906e-08, -1.077906e-08},
          {0, -1.711427e-08, 0, -1.711427e-08, 0, -1.711427e-08, 0, -1.711427e-08},
          {0, -2.481987e-08, -3.340894e-08, -1.794823e-08, -4.276810e-08, -5.135717e-08, -1.794823e-08, -4.276810e-08, -5.135717e-08},
          {0, 2.236068e-08, 3.402759e-08, 4.476821e-08, 2.236068e-08, 2.148125e-08, 2.236068e-08, 4.476821e-08, 3.402759e-08, 3.310130e-08},
          {0, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09, -7.151898e-09},
          {0, -2.467882e-08, -2.467882e-08, 0, -2.467882e-08, -3.365293e-08, -1.794823e-08, -2.467882e-08, -2.467882e-08, -1.794823e-08, -3.365293e-08, -2.467882e-08},
          {0, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09, 1.205031e-09},
          {0, -2.171372e-08, -4.264971e-09, -2.117969e-08, -1.579016e-08, -9.654500e-09, -2.171372e-08, -1.077906e-08, -2.171372e-08, -9.654500e-09, -1.579016e-08, -2.117969e-08, -4.264971e-09, -2.710325e-08},
          {0, -2.918294e-09, 1.777255e-08, 3.043176e-08, 3.112198e-08, 1.946019e-09, 3.874073e-09, 1.433369e-08, 2.163716e-08, 2.717372e-08, -3.259352e-09, 4.053584e-09, 1.935955e-08, 1.643179e-08, 2.735323e-08},
          {0, -3.709142e-08, -1.711427e-08, -3.709142e-08, 0, -3.709142e-08, -1.711427e-08, -3.709142e-08, 0, -3.709142e-08, -1.711427e-08, -3.709142e-08, 0, -3.709142e-08, -1.711427e-08, -3.709142e-08},
      },
  };
  return g[side][R][i];
}

}  // namespace ws
