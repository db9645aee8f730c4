// sma_solo.cuh -- the element loop with one thread per HEX08 element.
//
// k_element gives each element 8 lanes, one per Gauss point; what the lanes
// share (the gathered nodes, the material, the scatter) is then formed eight
// times or passed through shuffles and shared memory.  Here one thread walks
// its element's 8 Gauss points:
//   - connectivity, material record and addresses once per element;
//   - the gathered nodes transformed once in registers (solo_wht), the 42
//     trilinear coefficients kept in the thread's own row of shared memory;
//   - the two Gauss points of a pair (s = -p, +p at the same t, z) share
//     du/ds, dX/ds and the parts of the other derivatives that do not depend
//     on s: 30 operations per point instead of 54;
//   - the element forces summed in the transformed space too: 28 operations
//     per point instead of 72 and no exchange between lanes; one transform
//     back at the end;
//   - lanes of a warp hold neighbouring elements, so the node gathers, the
//     state (tiles of 32 elements, state_index) and the scatter's atomics are
//     coalesced;
//   - FP32: the two Gauss points of a pair go through packed instructions.
//
// Bound: instruction issue and dependent latency (ncu, FP32, 250 k-element
// cylinder section: 416 thread-instructions per Gauss point where k_element
// executes 1,100; 44-50 % of issue slots at 10.5 resident warps per SM; DRAM
// 1.1 TB/s).  Per launch, 8 lanes per element -> one thread per element:
//   2.0 M-element cylinder, a material per element, FP32    704 -> 334 us
//   640 k-element cantilever, one material, FP32 / FP64     180 -> 120, 318 -> 205
//   250 k-element cylinder FP32 / FP64                       78 -> 52, 146 -> 90
//   24-specimen ensemble (294 k) FP32 / FP64                111 -> 63, 163 -> 107
// The steps on the way, cylinder FP32: scalar arithmetic, both points of a
// pair interleaved by the compiler 471; packed with the rare forms called
// inside the loop (300 bytes of spills) 506; the rare forms moved behind the
// loop 364; tiled state, transforms and derivatives packed over components
// 341; connectivity prefetch 334.
#pragma once

#include "sma_kernels.cuh"

namespace sma {

// material of an element: the launch's one material, its compact record, or
// the material table
constexpr int SOLO_ONE = 0, SOLO_COMPACT = 1, SOLO_TABLE = 2;

constexpr int SOLO_BLOCK = 64;                                   // largest block

// Resident 64-thread blocks per SM the register cap allows: FP32 6 (168
// registers, 12 warps; no spills with one material), FP64 4 (255 registers, 8
// warps).  FP32 at 8 blocks (128 registers, 200-270 bytes of spills) lost 25 %
// on the 640 k-element cantilever and the 2.0 M-element cylinder, FP64 at 6
// blocks (168 registers, 600 bytes) 30 %.
template <typename T>
constexpr int solo_min_blocks() {
  return sizeof(T) == 4 ? 6 : 4;
}

// a thread's row of shared memory: the 48 coefficients (solo_gather; entry 0
// of each unused), padded to an odd multiple of 16 bytes so that the 128-bit
// accesses of a quarter warp hit distinct banks
template <typename T>
struct SoloRow {
  static constexpr int STRIDE = 48 + 16 / (int)sizeof(T);
};
template <typename T>
inline size_t solo_smem_bytes(int block) {
  return (size_t)block * SoloRow<T>::STRIDE * sizeof(T);
}

// ---------------------------------------------------------------------------
// Two values, one per Gauss point of a pair.  FP32: one register pair and
// the packed f32x2 instructions, which do both multiply-adds in one issue
// slot (the FP32 element loop is bound by instruction issue, and 61 % of its
// instructions are FP32 multiply-adds).  FP64: two scalars.
// ---------------------------------------------------------------------------
struct f2 {
  unsigned long long v;
};
struct d2 {
  double x, y;
};
__device__ __forceinline__ f2 mk2(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float lo(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return x;
}
__device__ __forceinline__ float hi(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return y;
}
__device__ __forceinline__ f2 operator+(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a) { return a * mk2(-1.0f, -1.0f); }
__device__ __forceinline__ d2 mk2(double x, double y) { return d2{x, y}; }
__device__ __forceinline__ double lo(d2 a) { return a.x; }
__device__ __forceinline__ double hi(d2 a) { return a.y; }
__device__ __forceinline__ d2 operator+(d2 a, d2 b) { return d2{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ d2 operator-(d2 a, d2 b) { return d2{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ d2 operator*(d2 a, d2 b) { return d2{a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ d2 vfma(d2 a, d2 b, d2 c) { return d2{fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)}; }
__device__ __forceinline__ d2 operator-(d2 a) { return d2{-a.x, -a.y}; }
template <typename T> struct PairOf;
template <> struct PairOf<float> { using type = f2; };
template <> struct PairOf<double> { using type = d2; };

// adjugate of 3x3 (row-major M[3 i + j]): C[3 j + i] = cofactor of M[3 i + j],
// so M^-1 = C / det.  Returns det.  Products that enter with a minus sign
// take one of six negated entries (packed operands carry no sign).
template <typename V>
__device__ __forceinline__ V adj3(const V* M, V* C) {
  const V n5 = -M[5], n0 = -M[0], n3 = -M[3], n1 = -M[1], n4 = -M[4], n2 = -M[2];
  C[0] = vfma(M[4], M[8], n5 * M[7]);
  C[3] = vfma(M[5], M[6], n3 * M[8]);
  C[6] = vfma(M[3], M[7], n4 * M[6]);
  C[1] = vfma(M[2], M[7], n1 * M[8]);
  C[4] = vfma(M[0], M[8], n2 * M[6]);
  C[7] = vfma(M[1], M[6], n0 * M[7]);
  C[2] = vfma(M[1], M[5], n4 * M[2]);
  C[5] = vfma(M[2], M[3], n5 * M[0]);
  C[8] = vfma(M[0], M[4], n3 * M[1]);
  return vfma(M[0], C[0], vfma(M[1], C[3], M[2] * C[6]));
}

// log1p of the pair's two symmetric matrices by the polynomial of sym_log1p
// (i2 from the traces).  False: a strain beyond its range, L meaningless.
template <typename T, typename V>
__device__ __forceinline__ bool pair_log1p(const V* A, V* L) {
  const V s00 = vfma(A[0], A[0], vfma(A[3], A[3], A[5] * A[5]));
  const V s11 = vfma(A[3], A[3], vfma(A[1], A[1], A[4] * A[4]));
  const V s22 = vfma(A[5], A[5], vfma(A[4], A[4], A[2] * A[2]));
  const V fro = s00 + s11 + s22;
  const bool ok = lo(fro) <= T(0.0625) && hi(fro) <= T(0.0625);
  const V s01 = vfma(A[0], A[3], vfma(A[3], A[1], A[5] * A[4]));
  const V s12 = vfma(A[3], A[5], vfma(A[1], A[4], A[4] * A[2]));
  const V s02 = vfma(A[0], A[5], vfma(A[3], A[4], A[5] * A[2]));
  const V i1 = A[0] + A[1] + A[2];
  const V half = mk2(T(0.5), T(0.5)), nhalf = mk2(T(-0.5), T(-0.5));
  const V ni2 = vfma(i1 * nhalf, i1, half * fro);
  const V n3 = -A[3], n4 = -A[4], n5 = -A[5];
  const V c00 = vfma(A[1], A[2], n4 * A[4]);
  const V c01 = vfma(A[4], A[5], n3 * A[2]);
  const V c02 = vfma(A[3], A[4], n5 * A[1]);
  const V i3 = vfma(A[0], c00, vfma(A[3], c01, A[5] * c02));
  constexpr int N = LogPoly<T>::N;
  auto cst = [](int k) { return mk2(LogPoly<T>::c(k), LogPoly<T>::c(k)); };
  // the first two Horner steps from (q[N-1], 0, 0)
  V al = cst(N - 3), be = cst(N - 2), ga = cst(N - 1);
#pragma unroll
  for (int k = N - 4; k >= 0; --k) {
    const V al1 = vfma(ga, i3, cst(k));
    const V be1 = vfma(ga, ni2, al);
    ga = vfma(ga, i1, be);
    al = al1;
    be = be1;
  }
  const V c0 = ga * i3, c1 = vfma(ga, ni2, al), c2 = vfma(ga, i1, be);   // the last product with A
  L[0] = vfma(c1, A[0], vfma(c2, s00, c0));
  L[1] = vfma(c1, A[1], vfma(c2, s11, c0));
  L[2] = vfma(c1, A[2], vfma(c2, s22, c0));
  L[3] = vfma(c1, A[3], c2 * s01);
  L[4] = vfma(c1, A[4], c2 * s12);
  L[5] = vfma(c1, A[5], c2 * s02);
  return ok;
}

// The scalar part of law 160 for one Gauss point (law160_from_A): from the
// trace theta, |e|^2 of the logarithmic strain and the state of the previous
// step to the new state, pv = K (theta - 3 alpha eL xS) and kappa.  False:
// the return map needs its iteration (return_map_closed).
template <typename T>
__device__ __forceinline__ bool law160_scalars(const MatC& m, T theta_t, T en2, double tmp, double& xS, double& F_AS,
                                              double& F_SA, T& pv, T& kp, int& flag) {
  const bool pos = en2 > T(0);
  const T ie = rsqrt(pos ? en2 : T(1));
  const T en_t = pos ? en2 * ie : T(0);
  double K = m.K, G = m.G, G_1 = m.G1;
  if (m.ext_E) {
    const double E = 1.0 / ((1.0 - xS) * m.iEA + xS * m.iEM);
    K = E * m.kK;
    G = E * m.kG;
    G_1 = (2.0 * G + 9.0 * (m.alfa * m.alfa) * K) * m.eL;
  }
  const double theta = (double)theta_t, e_n = (double)en_t;
  flag = NR_NONE;
  const bool ok = return_map_closed<sizeof(T) == 8>(m, K, G, G_1, theta, e_n, tmp, xS, F_AS, F_SA, flag);
  pv = (T)(K * (theta - 3.0 * m.alfa * m.eL * xS));
  const T twoG = (T)(2.0 * G);
  kp = (en_t > T(2.220446049250313e-16)) ? twoG * (T(1) - (T)(m.eL * xS) * ie) : twoG;
  return ok;
}

// Walsh-Hadamard transform of 8 values, w[k] = sum_a v[a] (-1)^popc(a & k),
// with w[2], w[3] and w[4] negated (the signs the derivatives take them with;
// the operands' order does it)
template <typename V>
__device__ __forceinline__ void solo_wht(V* w) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const V p = w[k], q = w[k + 1];
    w[k] = p + q;
    w[k + 1] = p - q;
  }
#pragma unroll
  for (int k = 0; k < 8; k += 4)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const V p = w[k + j], q = w[k + j + 2];
      w[k + j] = p + q;
      w[k + j + 2] = q - p;
    }
  const V p0 = w[0], p1 = w[1], p2 = w[2], p3 = w[3];
  w[0] = p0 + w[4];
  w[4] = w[4] - p0;
  w[1] = p1 + w[5];
  w[5] = p1 - w[5];
  w[2] = p2 + w[6];
  w[6] = w[6] - p2;
  w[3] = p3 + w[7];
  w[7] = w[7] - p3;
}

// two values to and from shared memory
__device__ __forceinline__ void ld2x2(const float* p, f2& a, f2& b) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  a.v = v.x;
  b.v = v.y;
}
__device__ __forceinline__ void st2x2(float* p, f2 a, f2 b) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a.v, b.v);
}
__device__ __forceinline__ void ld2x2(const double* p, d2& a, d2& b) {
  const double2 u = *reinterpret_cast<const double2*>(p), v = *reinterpret_cast<const double2*>(p + 2);
  a = d2{u.x, u.y};
  b = d2{v.x, v.y};
}
__device__ __forceinline__ void st2x2(double* p, d2 a, d2 b) {
  *reinterpret_cast<double2*>(p) = make_double2(a.x, a.y);
  *reinterpret_cast<double2*>(p + 2) = make_double2(b.x, b.y);
}

template <typename T>
__device__ __forceinline__ void solo_nodes(const ElemArgs<T>& a, int64_t ec, int* nid) {
  const int4* ln = reinterpret_cast<const int4*>(a.lnods + 8 * ec);
  const int4 p = __ldg(ln), q = __ldg(ln + 1);
  nid[0] = p.x; nid[1] = p.y; nid[2] = p.z; nid[3] = p.w;
  nid[4] = q.x; nid[5] = q.y; nid[6] = q.z; nid[7] = q.w;
}

// the element's node values relative to its first node, formed in FP64 and
// transformed, into the thread's row: [3][8][2], two of x, y, z, ux, uy, uz
// side by side
template <typename T>
__device__ __forceinline__ void solo_gather(const ElemArgs<T>& a, int64_t ec, T* row) {
  using V = typename PairOf<T>::type;
  int nid[8];
  solo_nodes(a, ec, nid);
  pdl_wait();                                                    // displacement, state, residual
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double* s0 = c == 0 ? a.coord : (c == 1 ? a.coord + 2 * a.npad : a.u + a.npad);
    const double* s1 = c == 0 ? a.coord + a.npad : (c == 1 ? a.u : a.u + 2 * a.npad);
    double v0[8], v1[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v0[k] = c == 2 ? ldcur(s0 + nid[k]) : __ldg(s0 + nid[k]);
      v1[k] = c == 0 ? __ldg(s1 + nid[k]) : ldcur(s1 + nid[k]);
    }
    V w[8];
    w[0] = mk2(T(0), T(0));
#pragma unroll
    for (int k = 1; k < 8; ++k) w[k] = mk2((T)(v0[k] - v0[0]), (T)(v1[k] - v1[0]));
    solo_wht(w);
#pragma unroll
    for (int k = 0; k < 8; k += 2) st2x2(row + 16 * c + 2 * k, w[k], w[k + 1]);
  }
}

template <typename T, int MAT>
__device__ __forceinline__ MatC solo_mat(const ElemArgs<T>& a, int64_t ec, double* tmp) {
  if constexpr (MAT == SOLO_COMPACT) {
    return compact_mat<T>(a, ec, tmp);
  } else {
    *tmp = a.tempe ? __ldg(a.tempe + ec) : 0.0;
    if constexpr (MAT == SOLO_TABLE) return a.mats[__ldg(a.lmate + ec)];
    else return a.mat0;
  }
}

// One element by the general forms (any strain, both transformations, det F
// <= 0 counted), a Gauss point at a time: what the loop below hands over when
// a point leaves the range of its short forms.  Out of line and called where
// nothing else is live, so it costs the loop no registers.
template <typename T, int MAT>
__device__ __noinline__ void solo_element_any(const ElemArgs<T>* ap, int64_t ec) {
  const ElemArgs<T>& a = *ap;
  double tmp;
  const MatC mat = solo_mat<T, MAT>(a, ec, &tmp);
  __align__(16) T nod[48], tr[48];                               // read and written in 128-bit pieces
  T f[8][3];
  solo_gather(a, ec, tr);
  for (int c = 0; c < 6; ++c)                                    // as stage_node_rows leaves them
    for (int k = 0; k < 8; ++k) nod[8 * c + k] = (k >= 2 && k <= 4 ? T(-1) : T(1)) * tr[16 * (c / 2) + 2 * k + (c & 1)];
  for (int k = 0; k < 24; ++k) f[k / 3][k % 3] = T(0);
  for (int g = 0; g < 8; ++g) {
    T Ji[9], H[9], Jc[9], B[9], tau[6], N[8], dN[24];
    const T detJ = gp_kinematics<T>(nod, g, Ji, H, Jc);
    const int64_t at = state_at(a, ec, g);
    double xS = (double)a.sold[at], F_AS = (double)a.sold[a.sst + at], F_SA = (double)a.sold[2 * a.sst + at];
    const int flag = law160_tau<T>(mat, H, tmp, xS, F_AS, F_SA, tau);
    a.snew[at] = (T)xS;
    a.snew[a.sst + at] = (T)F_AS;
    a.snew[2 * a.sst + at] = (T)F_SA;
    const T detFJ = inv3(Jc, B);
    const T w = T(8) * detJ;                                     // dV (F J)^-1 = w B
    hex8_gp<T>(g, N, dN);
    const T tf[9] = {tau[0], tau[3], tau[5], tau[3], tau[1], tau[4], tau[5], tau[4], tau[2]};
    for (int i = 0; i < 3; ++i) {
      T q[3];
      for (int m = 0; m < 3; ++m)
        q[m] = w * (tf[3 * i] * B[3 * m] + tf[3 * i + 1] * B[3 * m + 1] + tf[3 * i + 2] * B[3 * m + 2]);
      for (int k = 0; k < 8; ++k) f[k][i] -= q[0] * dN[3 * k] + q[1] * dN[3 * k + 1] + q[2] * dN[3 * k + 2];
    }
    if (flag & (NR_CONVERGED | NR_FAILED)) atomicAdd(a.cnt + CNT_NR_ACTIVE, 1ull);
    if (flag & NR_FAILED) atomicAdd(a.cnt + CNT_NR_FAILED, 1ull);
    if (flag & NR_BOTH) atomicAdd(a.cnt + CNT_NR_BOTH, 1ull);
    if (!(detFJ * detJ > T(0))) {
      atomicAdd(a.cnt + CNT_NEG_DET, 1ull);
      atomicMin(a.cnt + CNT_DETMIN, detmin_key((float)(detFJ / (T(512) * detJ)), ec));
    }
  }
  int nid[8];
  solo_nodes(a, ec, nid);
  for (int i = 0; i < 3; ++i)
    for (int k = 0; k < 8; ++k) atomicAdd(a.f + i * a.npad + nid[k], (double)f[k][i]);
}

template <typename T, int MAT>
__global__ void __launch_bounds__(SOLO_BLOCK, (solo_min_blocks<T>())) k_element_solo(const __grid_constant__ ElemArgs<T> a) {
  using V = typename PairOf<T>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* row = reinterpret_cast<T*>(smem_raw) + threadIdx.x * SoloRow<T>::STRIDE;
  const int64_t e = (int64_t)a.beg + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = e < a.end;
  const int64_t ec = valid ? e : (int64_t)a.end - 1;
  pdl_launch();
  if (time_block(a)) return;

  // the connectivity of the element one resident wave ahead, into L2
  if (e + a.pf_ahead < a.end) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.lnods + 8 * (e + a.pf_ahead)));
  double tmp;
  MatC mx;
  if constexpr (MAT == SOLO_COMPACT) mx = compact_mat<T>(a, ec, &tmp);
  else tmp = a.tempe ? __ldg(a.tempe + ec) : 0.0;
  const MatC& mat = MAT == SOLO_ONE ? a.mat0 : (MAT == SOLO_TABLE ? a.mats[__ldg(a.lmate + ec)] : mx);

  solo_gather(a, ec, row);

  // ---- Gauss points -------------------------------------------------------
  const T p = T(0.577350269189626);
  V F2[8];                                                       // force sums of x and y,
  T F1[8];                                                       // of z; [0] stays 0
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    F2[k] = mk2(T(0), T(0));
    F1[k] = T(0);
  }
  int active = 0;
  bool ok = true;                                                // false: redo by solo_element_any
  // state of the warp's tile: every access an immediate offset from here
  const T* so = a.sold + state_at(a, ec, 0);
  T* sn = a.snew + state_at(a, ec, 0);
  T st[2][3];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int c = 0; c < 3; ++c) st[h][c] = so[c * ST_C + 4 * h * ST_G];
  // pair (t, z): Gauss points g = tz (s = -p) and tz + 4 (s = +p)
#pragma unroll 1
  for (int tz = 0; tz < 4; ++tz) {
    const T t = (tz & 2) ? p : -p, z = (tz & 1) ? p : -p;
    const V tt = mk2(t, t), zz = mk2(z, z), nt = mk2(-t, -t), nz = mk2(-z, -z);
    // 8 d/ds, 8 d/dt, 8 d/dz at the pair of two of x, y, z, ux, uy, uz
    auto deriv = [&](int c, V* o, V* o2) {
      V w[8];
#pragma unroll
      for (int k = 0; k < 8; k += 2) ld2x2(row + 16 * c + 2 * k, w[k], w[k + 1]);
      const V b = vfma(nz, w[5], w[1]), d = vfma(nt, w[5], w[7]);
      const V ds = vfma(w[7], zz, vfma(b, tt, w[3]));
      const V dt = vfma(w[6], zz, w[2]), dz = vfma(w[6], tt, w[4]);
      o[0] = mk2(lo(ds), lo(ds));
      o[1] = mk2(fma(-p, lo(b), lo(dt)), fma(p, lo(b), lo(dt)));
      o[2] = mk2(fma(-p, lo(d), lo(dz)), fma(p, lo(d), lo(dz)));
      o2[0] = mk2(hi(ds), hi(ds));
      o2[1] = mk2(fma(-p, hi(b), hi(dt)), fma(p, hi(b), hi(dt)));
      o2[2] = mk2(fma(-p, hi(d), hi(dz)), fma(p, hi(d), hi(dz)));
    };
    V B[9], J[9], tau[6], det8, detFJ;
    {
      V G[9], Ji[9], H[9];
      deriv(0, J, J + 3);
      deriv(1, J + 6, G);
      det8 = adj3(J, Ji);                                        // 512 det J
      const V id = mk2(Fm<T>::rcp(lo(det8)), Fm<T>::rcp(hi(det8)));
#pragma unroll
      for (int k = 0; k < 9; ++k) Ji[k] = Ji[k] * id;
      deriv(2, G + 3, G + 6);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          H[3 * i + k] = vfma(G[3 * i], Ji[k], vfma(G[3 * i + 1], Ji[3 + k], G[3 * i + 2] * Ji[6 + k]));
          J[3 * i + k] = J[3 * i + k] + G[3 * i + k];            // 8 F J
        }
      // A = b - I = H + H^T + H H^T
      V A[6], L[6];
      const V two = mk2(T(2), T(2));
      A[0] = vfma(two, H[0], vfma(H[0], H[0], vfma(H[1], H[1], H[2] * H[2])));
      A[1] = vfma(two, H[4], vfma(H[3], H[3], vfma(H[4], H[4], H[5] * H[5])));
      A[2] = vfma(two, H[8], vfma(H[6], H[6], vfma(H[7], H[7], H[8] * H[8])));
      A[3] = H[1] + vfma(H[0], H[3], vfma(H[1], H[4], vfma(H[2], H[5], H[3])));
      A[4] = H[5] + vfma(H[3], H[6], vfma(H[4], H[7], vfma(H[5], H[8], H[7])));
      A[5] = H[2] + vfma(H[0], H[6], vfma(H[1], H[7], vfma(H[2], H[8], H[6])));
      ok &= pair_log1p<T, V>(A, L);
      const V half = mk2(T(0.5), T(0.5));
      const V theta = half * (L[0] + L[1] + L[2]);
      const V nt3 = theta * mk2(T(-1) / T(3), T(-1) / T(3));
      const V e0 = vfma(half, L[0], nt3), e1 = vfma(half, L[1], nt3), e2 = vfma(half, L[2], nt3);
      const V en2 = vfma(e0, e0, vfma(e1, e1, e2 * e2)) +
                    half * vfma(L[3], L[3], vfma(L[4], L[4], L[5] * L[5]));
      T pv[2], kp[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double xS = (double)st[h][0], F_AS = (double)st[h][1], F_SA = (double)st[h][2];
        int flag;
        ok &= law160_scalars<T>(mat, h ? hi(theta) : lo(theta), h ? hi(en2) : lo(en2), tmp, xS, F_AS, F_SA, pv[h],
                                kp[h], flag);
        if (valid) {
          sn[(tz + 4 * h) * ST_G] = (T)xS;
          sn[(tz + 4 * h) * ST_G + ST_C] = (T)F_AS;
          sn[(tz + 4 * h) * ST_G + 2 * ST_C] = (T)F_SA;
          if (tz < 3) {                                          // the next pair's state
#pragma unroll
            for (int c = 0; c < 3; ++c) st[h][c] = so[(tz + 1 + 4 * h) * ST_G + c * ST_C];
          }
        }
        active += flag == NR_CONVERGED ? 1 : 0;
      }
      // tau = pv I + kappa (L/2 - theta/3 I)
      const V kap = mk2(kp[0], kp[1]);
      const V dg = vfma(kap, nt3, mk2(pv[0], pv[1])), kh = half * kap;
#pragma unroll
      for (int k = 0; k < 3; ++k) tau[k] = vfma(kh, L[k], dg);
#pragma unroll
      for (int k = 3; k < 6; ++k) tau[k] = kh * L[k];
    }
    // Q / 8 = dV tau (F J)^-T / 8
    V q[9];
    {
      detFJ = adj3(J, B);
      const V sc = det8 * mk2(T(1.0 / 512.0) * Fm<T>::rcp(lo(detFJ)), T(1.0 / 512.0) * Fm<T>::rcp(hi(detFJ)));
#pragma unroll
      for (int k = 0; k < 6; ++k) tau[k] = tau[k] * sc;
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        q[m] = vfma(tau[0], B[3 * m], vfma(tau[3], B[3 * m + 1], tau[5] * B[3 * m + 2]));
        q[3 + m] = vfma(tau[3], B[3 * m], vfma(tau[1], B[3 * m + 1], tau[4] * B[3 * m + 2]));
        q[6 + m] = vfma(tau[5], B[3 * m], vfma(tau[4], B[3 * m + 1], tau[2] * B[3 * m + 2]));
      }
      // det F <= 0 (det F = det(8 F J) / det(8 J)): counted by the redo
      const V dd = detFJ * det8;
      ok &= lo(dd) > T(0) && hi(dd) > T(0);
    }
    // f_a = -sum_g Q_g dN_a(g), summed as the coefficients of (-1)^popc(a & k)
    T qs[3], qt[3], qz[3], ut[3], uz[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      qs[i] = lo(q[3 * i]) + hi(q[3 * i]);
      qt[i] = lo(q[3 * i + 1]) + hi(q[3 * i + 1]);
      ut[i] = hi(q[3 * i + 1]) - lo(q[3 * i + 1]);
      qz[i] = lo(q[3 * i + 2]) + hi(q[3 * i + 2]);
      uz[i] = hi(q[3 * i + 2]) - lo(q[3 * i + 2]);
    }
    {
      const V s2 = mk2(qs[0], qs[1]), t2 = mk2(qt[0], qt[1]), z2 = mk2(qz[0], qz[1]);
      const V d2z = mk2(uz[0], uz[1]), pp = mk2(p, p), tp = mk2(t * p, t * p);
      const V u = vfma(pp, mk2(ut[0], ut[1]), tt * s2);
      F2[1] = F2[1] + u;
      F2[2] = F2[2] + t2;
      F2[3] = F2[3] + s2;
      F2[4] = F2[4] + z2;
      F2[5] = vfma(zz, u, vfma(tp, d2z, F2[5]));
      F2[6] = vfma(zz, t2, vfma(tt, z2, F2[6]));
      F2[7] = vfma(zz, s2, vfma(pp, d2z, F2[7]));
    }
    {
      const T u = p * ut[2] + t * qs[2];
      F1[1] += u;
      F1[2] += qt[2];
      F1[3] += qs[2];
      F1[4] += qz[2];
      F1[5] += z * u + t * p * uz[2];
      F1[6] += z * qt[2] + t * qz[2];
      F1[7] += z * qs[2] + p * uz[2];
    }
  }

  // ---- scatter ------------------------------------------------------------
  if (valid && ok) {
    int nid[8];
    solo_nodes(a, ec, nid);                                      // from cache: not held across the loop
    // f_a = -F1 x1 + F2 x2 + F3 x3 + F4 x4 + F5 x5 - F6 x6 - F7 x7, xk = (-1)^popc(a & k):
    // solo_wht with its signs of k = 2, 3, 4 undone
    auto node_forces = [](auto* w) {
      w[1] = -w[1];
      w[6] = -w[6];
      w[7] = -w[7];
      solo_wht(w);
      w[2] = -w[2];
      w[3] = -w[3];
      w[4] = -w[4];
    };
    node_forces(F2);
    node_forces(F1);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      double* dst = a.f + nid[k];
      atomicAdd(dst, (double)lo(F2[k]));
      atomicAdd(dst + a.npad, (double)hi(F2[k]));
      atomicAdd(dst + 2 * a.npad, (double)F1[k]);
    }
  } else if (valid) {
    solo_element_any<T, MAT>(&a, ec);
  }
  const int n = __reduce_add_sync(0xffffffffu, valid && ok ? active : 0);
  if (n && (threadIdx.x & 31) == 0) atomicAdd(a.cnt + CNT_NR_ACTIVE, (unsigned long long)n);
}

}  // namespace sma
