// rve_modes.cuh -- the stencil operator of the batched solve in element-mode
// form, marched along z, and a per-load-case solve that keeps its search
// direction on chip.
//
// Element modes.  All elements of an RVE mesh are equal boxes.  In the Walsh
// basis of the 8 corners (sums and differences along x, y and z) the element
// stiffness K = H^T Khat H of an isotropic material has 21 diagonal entries
// and 12 couplings instead of 576 entries (the modes are the orthogonal
// polynomials 1, x, y, z, xy, ... of the trilinear element, and the 2x2x2
// Gauss rule of micro/src/assembly.c:97-108 integrates their products
// exactly).  The transforms along x and y are shared by the elements above
// and below a face, the one along z is a running pair of faces, so an
// operator application costs about 140 packed additions and FMAs per element
// and pair of values instead of the 243 FMAs and 27 block loads per node of
// the assembled stencil.  Differences are formed before they are multiplied,
// so the FP32 operator annihilates rigid motions exactly.
//
// March.  A thread owns one element column (face f = ex + nex*ey) and steps
// through z; F0/F1 are the x-y modes of the face below and above the current
// layer.  The mode forces of a plane are turned back to nodes along x by a
// shuffle (lane 0 of a warp repeats the last column of the previous warp)
// and along y through shared memory, one barrier a plane.  The column's node
// (ex, ey) belongs to the same thread, which updates its vectors.
//
// Packing.  FP32 values travel in pairs: plane i of the lower half of the
// interior planes with plane i + h of the upper half, h = ceil(mz / 2), so
// every addition and FMA is one packed instruction for two layers.  One
// layer (the seam) is computed by both halves.
//
// Boundary nodes carry zeros (the unknown is the fluctuation w of
// u = eps.x + w).  Node (i, j) of a plane lies at index i + nex*j, i in
// [0, nex), j in [0, ney): the nodes at i = 0 and j = 0 are the zero padding
// that the last column's and row's faces read too.
#pragma once

#include "rve_device.cuh"

namespace sp {

// ------------------------------------------------------ packed FP32 pairs ---

struct F2 {
  float2 v;
};
__device__ __forceinline__ F2 mk2(float a, float b) { return F2{make_float2(a, b)}; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return F2{__fadd2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  return F2{__ffma2_rn(b.v, make_float2(-1.f, -1.f), a.v)};
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return F2{__fmul2_rn(a.v, b.v)}; }
__device__ __forceinline__ F2 mad(F2 a, F2 b, F2 c) { return F2{__ffma2_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ F2 up1(F2 a) {
  return mk2(__shfl_up_sync(0xffffffffu, a.v.x, 1), __shfl_up_sync(0xffffffffu, a.v.y, 1));
}
__device__ __forceinline__ double up1(double a) { return __shfl_up_sync(0xffffffffu, a, 1); }
__device__ __forceinline__ F2 zero_of(F2) { return mk2(0.f, 0.f); }
__device__ __forceinline__ double zero_of(double) { return 0.0; }

// ------------------------------------------------------------ coefficients ---

// Khat of one material: entries of the mode matrix, c0 = volume / 16,
// L = lambda + 2 mu, a = 1 / h.
enum ModeCoef {
  MC_AXX, MC_AYY, MC_AZZ,           // c0 L a_i^2
  MC_BXY, MC_BXZ, MC_BYZ,           // c0 lambda a_i a_j
  MC_MXX, MC_MYY, MC_MZZ,           // c0 mu a_i^2
  MC_MXY, MC_MXZ, MC_MYZ,           // c0 mu a_i a_j
  MC_U110, MC_W011, MC_U101, MC_V011, MC_V110, MC_W101,  // bilinear modes of normal strains
  MC_B3XY, MC_B3XZ, MC_B3YZ,        // their lambda couplings
  MC_U011, MC_V101, MC_W110,        // twist modes
  MC_M3XY, MC_M3XZ, MC_M3YZ,        // their mu couplings
  MC_U111, MC_V111, MC_W111,
  MC_N
};

__device__ inline double mode_coef(int i, double lam, double mu, double c0, const double *a) {
  const double L = lam + 2.0 * mu;
  const double xx = a[0] * a[0], yy = a[1] * a[1], zz = a[2] * a[2];
  const double xy = a[0] * a[1], xz = a[0] * a[2], yz = a[1] * a[2];
  const double c1 = c0 / 3.0, c2 = c0 / 9.0;
  switch (i) {
    case MC_AXX: return c0 * L * xx;
    case MC_AYY: return c0 * L * yy;
    case MC_AZZ: return c0 * L * zz;
    case MC_BXY: return c0 * lam * xy;
    case MC_BXZ: return c0 * lam * xz;
    case MC_BYZ: return c0 * lam * yz;
    case MC_MXX: return c0 * mu * xx;
    case MC_MYY: return c0 * mu * yy;
    case MC_MZZ: return c0 * mu * zz;
    case MC_MXY: return c0 * mu * xy;
    case MC_MXZ: return c0 * mu * xz;
    case MC_MYZ: return c0 * mu * yz;
    case MC_U110: return c1 * (L * xx + mu * yy);
    case MC_W011: return c1 * (L * zz + mu * yy);
    case MC_U101: return c1 * (L * xx + mu * zz);
    case MC_V011: return c1 * (L * yy + mu * zz);
    case MC_V110: return c1 * (L * yy + mu * xx);
    case MC_W101: return c1 * (L * zz + mu * xx);
    case MC_B3XY: return c1 * lam * xy;
    case MC_B3XZ: return c1 * lam * xz;
    case MC_B3YZ: return c1 * lam * yz;
    case MC_U011: return c1 * mu * (yy + zz);
    case MC_V101: return c1 * mu * (xx + zz);
    case MC_W110: return c1 * mu * (xx + yy);
    case MC_M3XY: return c1 * mu * xy;
    case MC_M3XZ: return c1 * mu * xz;
    case MC_M3YZ: return c1 * mu * yz;
    case MC_U111: return c2 * (L * xx + mu * (yy + zz));
    case MC_V111: return c2 * (L * yy + mu * (xx + zz));
    default: return c2 * (L * zz + mu * (xx + yy));
  }
}

// diagonal of the element stiffness for component c (the same at every
// corner: the sum of the component's diagonal mode entries)
__device__ inline double mode_diag(const double *C, int c) {
  if (c == 0)
    return C[MC_AXX] + C[MC_MYY] + C[MC_MZZ] + C[MC_U110] + C[MC_U101] + C[MC_U011] + C[MC_U111];
  if (c == 1)
    return C[MC_AYY] + C[MC_MXX] + C[MC_MZZ] + C[MC_V110] + C[MC_V011] + C[MC_V101] + C[MC_V111];
  return C[MC_AZZ] + C[MC_MXX] + C[MC_MYY] + C[MC_W101] + C[MC_W011] + C[MC_W110] + C[MC_W111];
}

// --------------------------------------------------------------- one layer ---

// x-y modes of a face from its corner values raw[c][corner], corners
// (0,0), (1,0), (0,1), (1,1); modes 00, 10, 01, 11 (sum/difference along x,
// then along y)
template <typename V>
__device__ __forceinline__ void face_modes(const V (&raw)[3][4], V (&F)[3][4]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const V s0 = raw[c][1] + raw[c][0], d0 = raw[c][1] - raw[c][0];
    const V s1 = raw[c][3] + raw[c][2], d1 = raw[c][3] - raw[c][2];
    F[c][0] = s1 + s0;
    F[c][1] = d1 + d0;
    F[c][2] = s1 - s0;
    F[c][3] = d1 - d0;
  }
}

// f = Khat m for a box element; S[c] = modes 100, 010, 110, D[c] = modes 001,
// 101, 011, 111 of component c, overwritten by the mode forces.  C(i):
// coefficient i.
template <typename V, typename CF>
__device__ __forceinline__ void modes_box(V (&S)[3][3], V (&D)[3][4], const CF &C) {
  {
    const V a = S[0][0], b = S[1][1], c = D[2][0];
    const V bxy = C(MC_BXY), bxz = C(MC_BXZ), byz = C(MC_BYZ);
    S[0][0] = mad(bxz, c, mad(bxy, b, C(MC_AXX) * a));
    S[1][1] = mad(byz, c, mad(bxy, a, C(MC_AYY) * b));
    D[2][0] = mad(byz, b, mad(bxz, a, C(MC_AZZ) * c));
  }
  {
    const V mxx = C(MC_MXX), myy = C(MC_MYY), mzz = C(MC_MZZ);
    {
      const V a = S[0][1], b = S[1][0], m = C(MC_MXY);
      S[0][1] = mad(m, b, myy * a);
      S[1][0] = mad(m, a, mxx * b);
    }
    {
      const V a = D[0][0], b = S[2][0], m = C(MC_MXZ);
      D[0][0] = mad(m, b, mzz * a);
      S[2][0] = mad(m, a, mxx * b);
    }
    {
      const V a = D[1][0], b = S[2][1], m = C(MC_MYZ);
      D[1][0] = mad(m, b, mzz * a);
      S[2][1] = mad(m, a, myy * b);
    }
  }
  {
    const V a = S[0][2], b = D[2][2], m = C(MC_B3XZ);
    S[0][2] = mad(m, b, C(MC_U110) * a);
    D[2][2] = mad(m, a, C(MC_W011) * b);
  }
  {
    const V a = D[0][1], b = D[1][2], m = C(MC_B3XY);
    D[0][1] = mad(m, b, C(MC_U101) * a);
    D[1][2] = mad(m, a, C(MC_V011) * b);
  }
  {
    const V a = S[1][2], b = D[2][1], m = C(MC_B3YZ);
    S[1][2] = mad(m, b, C(MC_V110) * a);
    D[2][1] = mad(m, a, C(MC_W101) * b);
  }
  {
    const V a = D[0][2], b = D[1][1], c = S[2][2];
    const V mxy = C(MC_M3XY), mxz = C(MC_M3XZ), myz = C(MC_M3YZ);
    D[0][2] = mad(mxz, c, mad(mxy, b, C(MC_U011) * a));
    D[1][1] = mad(myz, c, mad(mxy, a, C(MC_V101) * b));
    S[2][2] = mad(myz, b, mad(mxz, a, C(MC_W110) * c));
  }
  D[0][3] = C(MC_U111) * D[0][3];
  D[1][3] = C(MC_V111) * D[1][3];
  D[2][3] = C(MC_W111) * D[2][3];
}

// the same for a cube, whose coefficients are six numbers: 35 instead of 45
// operations and no coefficient loads
enum CubeCoefIndex { CC_LAM, CC_MU, CC_MU2, CC_LAM3, CC_MU3, CC_K9, CC_N };
// C(i): lambda, mu, 2 mu, lambda/3, mu/3, (lambda + 4 mu)/9, read where used
template <typename V, typename CF>
__device__ __forceinline__ void modes_cube(V (&S)[3][3], V (&D)[3][4], const CF &C) {
  const V mu = C(CC_MU);
  {
    const V t = C(CC_LAM) * (S[0][0] + S[1][1] + D[2][0]);
    const V mu2 = C(CC_MU2);
    S[0][0] = mad(mu2, S[0][0], t);
    S[1][1] = mad(mu2, S[1][1], t);
    D[2][0] = mad(mu2, D[2][0], t);
  }

  S[0][1] = S[1][0] = mu * (S[0][1] + S[1][0]);
  D[0][0] = S[2][0] = mu * (D[0][0] + S[2][0]);
  D[1][0] = S[2][1] = mu * (D[1][0] + S[2][1]);
  {
    const V lam3 = C(CC_LAM3);
    {
      const V t = lam3 * (S[0][2] + D[2][2]);
      S[0][2] = mad(mu, S[0][2], t);
      D[2][2] = mad(mu, D[2][2], t);
    }
    {
      const V t = lam3 * (D[0][1] + D[1][2]);
      D[0][1] = mad(mu, D[0][1], t);
      D[1][2] = mad(mu, D[1][2], t);
    }
    {
      const V t = lam3 * (S[1][2] + D[2][1]);
      S[1][2] = mad(mu, S[1][2], t);
      D[2][1] = mad(mu, D[2][1], t);
    }
  }

  {
    const V mu3 = C(CC_MU3);
    const V t = mu3 * (D[0][2] + D[1][1] + S[2][2]);
    D[0][2] = mad(mu3, D[0][2], t);
    D[1][1] = mad(mu3, D[1][1], t);
    S[2][2] = mad(mu3, S[2][2], t);
  }
  const V k9 = C(CC_K9);
#pragma unroll
  for (int c = 0; c < 3; c++) D[c][3] = k9 * D[c][3];
}

// Mode differences of a layer from its two faces
template <typename V>
__device__ __forceinline__ void layer_modes(const V (&F0)[3][4], const V (&F1)[3][4], V (&S)[3][3],
                                            V (&D)[3][4]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
#pragma unroll
    for (int m = 0; m < 3; m++) S[c][m] = F1[c][m + 1] + F0[c][m + 1];
#pragma unroll
    for (int m = 0; m < 4; m++) D[c][m] = F1[c][m] - F0[c][m];
  }
}

// One component's mode forces of a plane turned back to nodes: low/high = the
// force of the column's nodes in row ey / row ey + 1, the left column's share
// taken from the lane below.
template <typename V>
__device__ __forceinline__ void plane_back(V t0, V t1, V t2, V t3, V &low, V &high) {
  const V m0 = (t0 - t1) + up1(t0 + t1);
  const V m1 = (t2 - t3) + up1(t2 + t3);
  low = m0 - m1;
  high = m0 + m1;
}

// Mode forces of the plane below the layer (acc + this layer's part) turned
// back to nodes; acc becomes the layer's part of the plane above.
template <typename V>
__device__ __forceinline__ void layer_back(const V (&S)[3][3], const V (&D)[3][4], V (&acc)[3][4],
                                           V (&low)[3], V (&high)[3]) {
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const V t0 = acc[c][0] - D[c][0];
    const V t1 = acc[c][1] + (S[c][0] - D[c][1]);
    const V t2 = acc[c][2] + (S[c][1] - D[c][2]);
    const V t3 = acc[c][3] + (S[c][2] - D[c][3]);
    acc[c][0] = D[c][0];
    acc[c][1] = S[c][0] + D[c][1];
    acc[c][2] = S[c][1] + D[c][2];
    acc[c][3] = S[c][2] + D[c][3];
    plane_back(t0, t1, t2, t3, low[c], high[c]);
  }
}

}  // namespace sp
