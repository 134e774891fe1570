// Element assembly into the node-block CSR system (sm_100a).
//
// Replaces the element loops of
//   IntElmAss_NS_overset            src/assembleNavSto.f90:76-336 (+e3LHS/e3RHS)
//   IntElmAss_NSVOF_Quenching_STAB  src/solveQuenching.f90:122-573
//   IntElmAss_Tem_Quenching_STAB    src/solveQuenching.f90:579-882
// together with the element Dirichlet treatment (BCLhs_3D / BCLhs_NS_conv /
// BCLhs_tem, src/BCLhs_3D.f90) and the scatter (FillSparseMat_*,
// LocaltoGlobalNSVOF_3D).
//
// Scheme (deterministic, atomic-free):
//   * element pass: one thread per element evaluates its Gauss points once and
//     writes a compact summary, the sums every block of its matrix is formed
//     from, and its residual rows;
//   * edge pass (tets): the work of an off-diagonal entry (A, B) is the list of
//     elements holding both nodes, in ascending order, the same list for
//     (B, A); a pair of lanes takes the two entries of an edge, expands one
//     block per element from the summaries and writes its block; 8 lanes per
//     node do the same for the diagonal block and the residual (hexahedra: a
//     row pass of their own, assemble_hex.cuh);
//   * the Dirichlet treatment of the reference zeroes element rows/columns
//     and puts 1 on the element diagonal; both commute with the sum, so they
//     are applied once at the write: masked entries are 0, a constrained
//     diagonal entry equals the number of elements around A.
#include "ovs_internal.cuh"

#include <math.h>
#include <string.h>

#include <type_traits>
#include <vector>

namespace {

// ------------------------------------------------------------------ params
struct AsmArgs {
  const void* rec;        // alpha-stage node records, REC values per node
  const uint8_t* ibc;     // N
  const int* rowptr;
  const int* colidx;
  const int* n2e_ptr;
  const int* n2e;         // node's elements as places of their summaries, by ascending id: (t << 3) | local node
  const unsigned* n2s;    // slots of each entry's element nodes in the row
  const int4* row_rec;    // per row in processing order: {A, rowptr[A], n2e_ptr[A], deg | sd << 8 | ne << 16}
  const int4* edge_rec;   // edges (tets): {A, B, slot of (A, B), slot of (B, A)}, tile by tile of rows
  const unsigned* edge_ptr;   //   offsets into edge_list, one per edge and the end
  const unsigned* edge_list;  //   (t << 4) | (local node of A << 2) | local node of B
  const unsigned* tile_edge;  // first edge of every tile of OVS_TILE_ROWS rows, and the end
  void* vals;             // nnz*NV
  void* rhs;              // NF*N field-major
  const void* kbuf;       // hex tensor-core block values (E x 64 x 24), or null
  int* flags;             // [0] non-positive DetJ count, [1] non-finite residual
  int N;
  int mat, vec;
  int max_deg;
  ovs_params p;
};

// value position tables of the internal slot layout (24 values per slot):
//   0..3  K(1,1) K(1,2) K(1,3) G(1)     row u1
//   4..7  K(2,1) K(2,2) K(2,3) G(2)     row u2
//   8..11 K(3,1) K(3,2) K(3,3) G(3)     row u3
//  12..15 D(1)   D(2)   D(3)   M        row p
//  16..19 LSU(1) LSU(2) LSU(3) LS       row phi
//  20..23 ULS(1) ULS(2) ULS(3) PLS      column phi
// The NS system keeps the first 16, the temperature system one value.
// IBC bit d <=> IBC(:, d+1) == 1: bits 0-2 velocity, 3 pressure, 4 VOF, 5 T.
// rowbits: A-side constraints that zero the entry (element row zeroing),
// colbits: B-side constraints (element column zeroing), diagbit: the entry
// set to 1 on the element diagonal.  Row/column rules follow BCLhs_3D
// (src/BCLhs_3D.f90:18-120) and BCLhs_NS_conv (:295-424) with the pressure at
// IBC column 4 and VOF at column 5; note M is only row-zeroed, ULS only
// column-zeroed, and LSU(i) is also zeroed by the u_i constraint of the ROW
// node (BCLhs_NS_conv :313,:345,:377).
constexpr uint8_t U0 = 1, U1 = 2, U2 = 4, PB = 8, FB = 16, TB = 32;
__constant__ uint8_t c_rowbits[24] = {U0, U0, U0, U0, U1, U1, U1, U1, U2, U2, U2, U2,
                                      PB, PB, PB, PB, FB | U0, FB | U1, FB | U2, FB, 0, 0, 0, PB};
__constant__ uint8_t c_colbits[24] = {U0, U1, U2, PB, U0, U1, U2, PB, U0, U1, U2, PB,
                                      U0, U1, U2, 0, U0, U1, U2, FB, FB, FB, FB, FB};
__constant__ uint8_t c_diagbit[24] = {U0, 0, 0, 0, 0, U1, 0, 0, 0, 0, U2, 0,
                                      0, 0, 0, PB, 0, 0, 0, FB, 0, 0, 0, 0};

// tet 4-point rule (src/genGP_GW.f90:332-353); N = (xi, eta, zeta, 1-xi-eta-zeta)
template <typename T>
__device__ __forceinline__ void tet_shape(int g, T N[4]) {
  const T a = (T)0.5854101966249685, b = (T)0.1381966011250105;
  T xi = (g == 0) ? a : b, eta = (g == 1) ? a : b, ze = (g == 2) ? a : b;
  N[0] = xi; N[1] = eta; N[2] = ze;
  N[3] = (T)1.0 - xi - eta - ze;
}

// FP64 node records held in shared memory instead of registers (64 values
// per element, transposed so a warp's accesses hit 32 consecutive banks),
// and zero rounding remainders: the FP64 element routines otherwise need
// more registers than a thread has.
template <typename T> struct SmemRecRow {
  const volatile T* p;   // volatile: read where used, not hoisted into registers
  __device__ __forceinline__ T operator[](int k) const { return p[(size_t)k * 128]; }
};
template <typename T> struct SmemRecs {
  const T* p;   // this thread's column of a [64][128] block array
  __device__ __forceinline__ SmemRecRow<T> operator[](int n) const { return SmemRecRow<T>{p + (size_t)n * 16 * 128}; }
};
template <typename T> struct ZeroRow {
  __device__ __forceinline__ T operator[](int) const { return (T)0; }
};
template <typename T> struct ZeroRecs {
  __device__ __forceinline__ ZeroRow<T> operator[](int) const { return ZeroRow<T>{}; }
};

// VOF field at tet Gauss point g in FP64 from the record value (slot k)
// plus its rounding remainder (lo[.][3]): sum_a N_a phi_a, in node order
template <typename T, typename RA, typename LA>
__device__ __forceinline__ double gp_phi(const RA& r, const LA& lo, int k, int g) {
  const double a = 0.5854101966249685, b = 0.1381966011250105;
  const double xi = (g == 0) ? a : b, eta = (g == 1) ? a : b, ze = (g == 2) ? a : b;
  const double N[4] = {xi, eta, ze, 1.0 - xi - eta - ze};
  double s = 0.0;
#pragma unroll
  for (int n = 0; n < 4; ++n) s += ((double)r[n][k] + (double)lo[n][3]) * N[n];
  return s;
}

// the clamp of prop_interp (src/e3int.f90:4-13): phic = min(max(phi, 0), 1)
__device__ __forceinline__ double clamp01(double x) { return fmax(fmin(x, 1.0), 0.0); }

// store NV (multiple of 4) register values to 16-byte aligned shared memory
template <int NV>
__device__ __forceinline__ void store_row(float* dst, const float* v) {
#pragma unroll
  for (int k = 0; k < NV; k += 4)
    *reinterpret_cast<float4*>(dst + k) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
}
template <int NV>
__device__ __forceinline__ void store_row(double* dst, const double* v) {
#pragma unroll
  for (int k = 0; k < NV; k += 2)
    *reinterpret_cast<double2*>(dst + k) = make_double2(v[k], v[k + 1]);
}

// 4 values to global memory with the streaming cache hint (st.global.cs):
// the CSR values are written once and not read again by the pass, so they
// should not evict the element summaries the pass still reads from L2
__device__ __forceinline__ void store4_cs(float* dst, const float* v) {
  __stcs(reinterpret_cast<float4*>(dst), make_float4(v[0], v[1], v[2], v[3]));
}
__device__ __forceinline__ void store4_cs(double* dst, const double* v) {
  __stcs(reinterpret_cast<double2*>(dst), make_double2(v[0], v[1]));
  __stcs(reinterpret_cast<double2*>(dst) + 1, make_double2(v[2], v[3]));
}

template <typename T>
__device__ __forceinline__ T pick4(const T v[4], int i) {
  return i == 0 ? v[0] : (i == 1 ? v[1] : (i == 2 ? v[2] : v[3]));
}

// Node records: REC = 20 values per node.  0-2: x+d (rounded to T),
// 3-15: the fields of the pass, 16-18: the rounding remainder of x+d, 19:
// the rounding remainder of the VOF field.  With the remainders, edge
// vectors x_j - x_k keep full T accuracy on fine meshes far from the origin,
// and the VOF value that blends properties 1000:1 is exact to FP64 (in FP64
// the remainders are 0).
constexpr int REC = 20;
__device__ __forceinline__ void load_rec(const float* rec, int node, float r[16], float lo[4]) {
  const float4* p = reinterpret_cast<const float4*>(rec) + (size_t)node * 5;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float4 v = __ldg(p + k);
    r[4 * k] = v.x; r[4 * k + 1] = v.y; r[4 * k + 2] = v.z; r[4 * k + 3] = v.w;
  }
  float4 v = __ldg(p + 4);
  lo[0] = v.x; lo[1] = v.y; lo[2] = v.z; lo[3] = v.w;
}
__device__ __forceinline__ void load_rec(const double* rec, int node, double r[16], double lo[4]) {
  const double2* p = reinterpret_cast<const double2*>(rec) + (size_t)node * 10;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    double2 v = __ldg(p + k);
    r[2 * k] = v.x; r[2 * k + 1] = v.y;
  }
  // FP64 records round nothing: their remainders (slots 16-19) are exactly 0
  lo[0] = lo[1] = lo[2] = lo[3] = 0.0;
}

// Geometry of a linear tet on the current configuration x+d
// (eval_shape_fem, src/eval_shape_FEM.f90:4-61, with get_inverse_3x3,
// src/eval_shape.f90:85-112).  xd[a][i] = x+d of node a.  The Jacobian of a
// linear tet is the same at every Gauss point, so it is evaluated once.
template <typename T, typename LA>
__device__ __forceinline__ T tet_geometry(const T xd[4][3], const LA& lo, T g[4][3], T G[3][3]) {
  T A[3][3], Ai[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) A[i][j] = (xd[j][i] - xd[3][i]) + (lo[j][i] - lo[3][i]);
  Ai[0][0] = A[1][1] * A[2][2] - A[2][1] * A[1][2];
  Ai[0][1] = A[2][1] * A[0][2] - A[0][1] * A[2][2];
  Ai[0][2] = A[0][1] * A[1][2] - A[0][2] * A[1][1];
  T tmp = (T)1.0 / (Ai[0][0] * A[0][0] + Ai[0][1] * A[1][0] + Ai[0][2] * A[2][0]);
  Ai[0][0] *= tmp; Ai[0][1] *= tmp; Ai[0][2] *= tmp;
  Ai[1][0] = (A[1][2] * A[2][0] - A[1][0] * A[2][2]) * tmp;
  Ai[1][1] = (A[0][0] * A[2][2] - A[2][0] * A[0][2]) * tmp;
  Ai[1][2] = (A[1][0] * A[0][2] - A[0][0] * A[1][2]) * tmp;
  Ai[2][0] = (A[1][0] * A[2][1] - A[1][1] * A[2][0]) * tmp;
  Ai[2][1] = (A[2][0] * A[0][1] - A[0][0] * A[2][1]) * tmp;
  Ai[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * tmp;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    g[0][j] = Ai[0][j]; g[1][j] = Ai[1][j]; g[2][j] = Ai[2][j];
    g[3][j] = (-Ai[0][j] - Ai[1][j]) - Ai[2][j];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      G[i][j] = Ai[0][i] * Ai[0][j] + Ai[1][i] * Ai[1][j] + Ai[2][i] * Ai[2][j];
  return (T)1.0 / tmp;
}

template <typename T>
__device__ __forceinline__ T quad_uGu(const T u[3], const T G[3][3]) {
  T t = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) t += u[i] * G[i][j] * u[j];
  return t;
}

// e3DC_beta2's INTEGER dummy receiving a real(8) (src/e3STAB.f90:175-189):
// the callee reads the low 4 bytes of the double.
__device__ __forceinline__ int low_word(double v) {
  return (int)(unsigned)(__double_as_longlong(v) & 0xffffffffULL);
}

__device__ __forceinline__ void cfl_max(unsigned long long* bits, double v) {
  if (v >= 0.0) atomicMax(bits, (unsigned long long)__double_as_longlong(v));
}

// ----------------------------------------------------- element summaries
// Pass 1 (one thread per element) evaluates everything the element matrix
// needs from its Gauss points, once, plus the element's residual rows, and
// stores it as a compact summary of SW values.  Pass 2 (the edge pass) forms
// the blocks of each element matrix from the summaries.  Inactive
// elements (solid on the NS+VOF pass, non-target on the NS pass) store zero
// sums and zero residuals, which makes every expanded block exactly zero.
// NS / NS+VOF: the Gauss-point sums of the block formulas (see add_block),
// which pass 1 forms once per element, in groups of 4 values that a lane of
// the edge pass reads with one load each:
//   [0, ND0)    per (row node a, column node b), PW values at PW (4a + b):
//               NS+VOF {S_ab, L1_ab + E_ab, PL_ab, V_ab}, NS {S_ab}
//   [ND0, T0)   per node n: grad N_n (3) and U_n (NS: 0)
//   [T0, C0)    T_n (4), Q_n (4)
//   [C0, RHS0)  NS+VOF KA KB MM KDP dphi (3) PR; NS KA KB MM PR
//   [RHS0, SW)  the residual: (u1, u2, u3, p) of every node, then NS+VOF phi (4)
// (PR = fact2 w, the sum of fact2 w N_n over the points, the same for every
// node; U_n is both U_b and W_a of the block formulas)
//   TEM  : the element matrix itself (a scalar system: smaller than what it
//          would be expanded from) as K_ab, K_ba of the six edges a < b (12),
//          then K_aa and the residual of every node (8)
// GQ: the values pass 1 keeps per Gauss point for the sums: uadv (3) and
// rt = rho tauM; NS+VOF: uadv (3) rho rt tauLS src eps ufac plfac (the
// factors of the phase-change terms).
template <int KIND> struct Lay;
template <> struct Lay<OVS_ASM_NS> {
  static constexpr int PW = 1, ND0 = 16, T0 = 32, C0 = 40, RHS0 = 44, SW = 60, NF = 4, NV = 16, GQ = 4;
};
template <> struct Lay<OVS_ASM_NSVOF> {
  static constexpr int PW = 4, ND0 = 64, T0 = 80, C0 = 88, RHS0 = 96, SW = 116, NF = 5, NV = 24, GQ = 10;
};
template <> struct Lay<OVS_ASM_TEM> {
  static constexpr int SW = 20, RHS0 = 12, NF = 1, NV = 1;
};

// number of the edge {a, b} of a tet, a < b in the order 01 02 03 12 13 23
__device__ __forceinline__ constexpr int tet_edge(int a, int b) { return a * (5 - a) / 2 + b - 1; }

// 4 values of an element summary (global memory; 16-byte aligned in FP32,
// 32-byte aligned in FP64, where every 4-value group of a summary sits on
// a 32-byte boundary) with one vector store.  FP64 uses the 256-bit global
// store of sm_100: one instruction instead of two 128-bit stores, measured
// 5.9 against 7.1 ms for the FP64 NS+VOF element pass at 128^3 (the pass
// writes 29 such groups per tet).  The asm carries no memory clobber: the
// element pass never reads a summary it writes, and the row pass that
// reads it is a later launch
template <typename T>
__device__ __forceinline__ void put4(T* d, T a, T b, T c, T e) {
  d[0] = a; d[1] = b; d[2] = c; d[3] = e;
}
__device__ __forceinline__ void put4(float* d, float a, float b, float c, float e) {
  *reinterpret_cast<float4*>(d) = make_float4(a, b, c, e);
}
__device__ __forceinline__ void put4(double* d, double a, double b, double c, double e) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(d), "d"(a), "d"(b), "d"(c), "d"(e));
}

// The Gauss-point sums of the NS / NS+VOF block formulas (add_block)
// from the per-point values q (layout GQ above), the shape gradients g and
// the weight w, written to the summary o: with c_n = uadv . grad N_n,
//   S_ab  = sum w rho (Na + rt ca)(fact1 Nb + fact2 cb)
//   L1_ab = sum w (Na + tauLS ca)(fact1 Nb + fact2 cb + fact2 Nb src)
//   E_ab  = sum eps Na Nb      PL_ab = -sum plfac Na Nb
//   V_ab  = sum fact2 w (Na + tauLS ca) Nb
//   U_n   = sum ufac Nn        T_n = sum w rt (fact1 Nn + fact2 cn)
//   Q_n   = sum fact2 w rt cn
// (rho = rho_ns on the NS pass).  Each sum is formed once per element here
// instead of once per block in the row pass.  block_sums_row writes the
// pairs of row node a and node a's record (a may vary per lane: the
// per-node values are picked by selects, which fold for a constant a).
template <typename T, int KIND>
__device__ __forceinline__ void block_sums_row(const T (&q)[4][Lay<KIND>::GQ], const T (&g)[4][3], T w, T fact1,
                                               T fact2, T rho_ns, int a, T* o, T (&tq)[8]) {
  using L = Lay<KIND>;
  constexpr bool vof = KIND == OVS_ASM_NSVOF;
  T c[4][4];
#pragma unroll
  for (int gp = 0; gp < 4; ++gp)
#pragma unroll
    for (int n = 0; n < 4; ++n) c[gp][n] = q[gp][0] * g[n][0] + q[gp][1] * g[n][1] + q[gp][2] * g[n][2];
  T S[4], L1[4], PL[4], V[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) S[b] = L1[b] = PL[b] = V[b] = 0;
#pragma unroll
  for (int gp = 0; gp < 4; ++gp) {
    T N[4];
    tet_shape<T>(gp, N);
    const T Na = pick4<T>(N, a), ca = pick4<T>(c[gp], a);
    const T rho = vof ? q[gp][3] : rho_ns;
    const T rt = vof ? q[gp][4] : q[gp][3];
    const T alpha = w * rho * (Na + rt * ca);
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const T beta = fact1 * N[b] + fact2 * c[gp][b];
      S[b] += alpha * beta;
      if constexpr (vof) {
        const T gam = w * (Na + q[gp][5] * ca);
        L1[b] += gam * (beta + fact2 * N[b] * q[gp][6]) + q[gp][7] * Na * N[b];
        PL[b] -= q[gp][9] * Na * N[b];
        V[b] += fact2 * gam * N[b];
      }
    }
  }
  if constexpr (vof) {
#pragma unroll
    for (int b = 0; b < 4; ++b) put4(o + L::PW * (4 * a + b), S[b], L1[b], PL[b], V[b]);
  } else {
    put4(o + L::PW * 4 * a, S[0], S[1], S[2], S[3]);
  }
  T Tn = 0, U = 0, Q = 0;
#pragma unroll
  for (int gp = 0; gp < 4; ++gp) {
    T N[4];
    tet_shape<T>(gp, N);
    const T Nn = pick4<T>(N, a), cn = pick4<T>(c[gp], a);
    const T rt = vof ? q[gp][4] : q[gp][3];
    Tn += w * rt * (fact1 * Nn + fact2 * cn);
    Q += fact2 * w * rt * cn;
    if constexpr (vof) U += q[gp][8] * Nn;
  }
  T ga[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const T col[4] = {g[0][d], g[1][d], g[2][d], g[3][d]};
    ga[d] = pick4<T>(col, a);
  }
  put4(o + L::ND0 + 4 * a, ga[0], ga[1], ga[2], U);
  tq[a] = Tn;
  tq[4 + a] = Q;
}

// all four rows of the element (one thread per element)
template <typename T, int KIND>
__device__ __forceinline__ void block_sums(const T (&q)[4][Lay<KIND>::GQ], const T (&g)[4][3], T w, T fact1,
                                           T fact2, T rho_ns, T* o) {
  T tq[8];
#pragma unroll
  for (int a = 0; a < 4; ++a) block_sums_row<T, KIND>(q, g, w, fact1, fact2, rho_ns, a, o, tq);
  put4(o + Lay<KIND>::T0, tq[0], tq[1], tq[2], tq[3]);
  put4(o + Lay<KIND>::T0 + 4, tq[4], tq[5], tq[6], tq[7]);
}

// The CFL number delt sqrt(taua), largest over an element's points: the
// point routines keep the largest taua and the element kernel takes one
// square root of it (sqrt and the product are monotone and correctly
// rounded, so this is the largest point value exactly; measured FP64
// NS+VOF 4.24 -> 4.12 ms, T 1.62 -> 1.49 ms, FP32 T 0.91 -> 0.79 ms).
// The FP32 NS+VOF pass keeps the value per point: the same change made
// that kernel slower (2.79 -> 3.05 ms at its 3-block bound, 3.26 at 4,
// 3.30 at 2).
template <typename T, int KIND> struct CflPerPoint { static constexpr bool v = false; };
template <> struct CflPerPoint<float, OVS_ASM_NSVOF> { static constexpr bool v = true; };

// 1 / sqrt(x): the reciprocal square root
__device__ __forceinline__ double inv_sqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float inv_sqrt(float x) { return rsqrtf(x); }

struct SumArgs {
  const void* rec;
  const int* ien;      // in storage order, as elm_id and the summaries
  const int* elm_id;
  void* sum;
  int* flags;
  unsigned long long* cfl_bits;
  int E;
  ovs_params p;
};

template <typename T, typename RA, typename LA>
__device__ __forceinline__ void element_geometry(const RA& r, const LA& lo, T g[4][3], T G[3][3],
                                                 T& detj, T& GG, T& trG) {
  T xd[4][3];
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int i = 0; i < 3; ++i) xd[n][i] = r[n][i];
  detj = tet_geometry<T>(xd, lo, g, G);
  GG = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int i = 0; i < 3; ++i) GG += G[i][j] * G[i][j];
  trG = G[0][0] + G[1][1] + G[2][2];
}

// pass 1, NS-only: IntElmAss_NS_overset's Gauss loop with e3LHS_3D_fluid_Old /
// e3Rhs_3D_fluid (quirks: uprime = 0, kap_dc = NS_kdc_a, tauBar = 0)
template <typename T, bool MAT = true, typename RA, typename LA>
__device__ void summarize_ns(const SumArgs& a, const RA& r, const LA& lo, bool target, T* o,
                             double& tamax, T& detj_out) {
  const ovs_params& p = a.p;
  T g[4][3], G[3][3], detj, GG, trG;
  element_geometry<T>(r, lo, g, G, detj, GG, trG);
  detj_out = detj;
  const T w = detj * (T)(0.25 / 6.0);
  T du[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      du[i][j] = r[0][3 + i] * g[0][j] + r[1][3 + i] * g[1][j] + r[2][3 + i] * g[2][j] + r[3][3 + i] * g[3][j];
  const T divu = du[0][0] + du[1][1] + du[2][2];
  const T rho = (T)p.rhoa, mu = (T)p.mua, mupkdc = mu + (T)p.ns_kdc_a;
  const T fact2 = (T)(p.alfi * p.gami * p.delt);
  const T taut = (T)(4.0 / (p.delt * p.delt));
  // the element's constants as reciprocals (rho, mu and trG are fixed over
  // its points): products instead of per-point divisions
  const T irho = (T)1.0 / rho, itrG = (T)1.0 / trG;
  const T nu = mu * irho;
  T KA = 0, KB = 0, MM = 0;
  T ru[4][3], rp[4], q[4][Lay<OVS_ASM_NS>::GQ];
#pragma unroll
  for (int n = 0; n < 4; ++n) { ru[n][0] = ru[n][1] = ru[n][2] = 0; rp[n] = 0; }
#pragma unroll
  for (int gp = 0; gp < 4; ++gp) {
    T N[4];
    tet_shape<T>(gp, N);
    T ui[3], umi[3], aci[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      ui[d] = r[0][3 + d] * N[0] + r[1][3 + d] * N[1] + r[2][3 + d] * N[2] + r[3][3 + d] * N[3];
      umi[d] = r[0][6 + d] * N[0] + r[1][6 + d] * N[1] + r[2][6 + d] * N[2] + r[3][6 + d] * N[3];
      aci[d] = r[0][9 + d] * N[0] + r[1][9 + d] * N[1] + r[2][9 + d] * N[2] + r[3][9 + d] * N[3];
    }
    const T pri = r[0][12] * N[0] + r[1][12] * N[1] + r[2][12] * N[2] + r[3][12] * N[3];
    const T uadv[3] = {ui[0] - umi[0], ui[1] - umi[1], ui[2] - umi[2]};
    const T taua = quad_uGu<T>(uadv, G);
    const T taud = nu * nu * (T)12.0 * GG;
    const T tauM = irho * inv_sqrt(taut + taua + taud);
    const T tauC = rho * sqrt(taua + taud) * itrG;
    if ((double)taua > tamax) tamax = (double)taua;   // CFL number: delt sqrt(max taua), in the kernel
    q[gp][0] = uadv[0]; q[gp][1] = uadv[1]; q[gp][2] = uadv[2]; q[gp][3] = rho * tauM;
    if (target) {
      KA += fact2 * mupkdc * w;
      KB += fact2 * tauC * w;
      MM += fact2 * w * tauM;
      const T ptot = pri - tauC * divu;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const T tmp1 = rho * (aci[i] + uadv[0] * du[i][0] + uadv[1] * du[i][1] + uadv[2] * du[i][2]) - (T)p.gravvec[i] * rho;
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const T sym = mupkdc * (g[n][0] * (du[i][0] + du[0][i]) + g[n][1] * (du[i][1] + du[1][i]) +
                                  g[n][2] * (du[i][2] + du[2][i]));
          ru[n][i] -= (N[n] * tmp1 + (sym - g[n][i] * ptot)) * w;
        }
      }
#pragma unroll
      for (int n = 0; n < 4; ++n) rp[n] -= (N[n] * divu) * w;
    }
  }
  using L = Lay<OVS_ASM_NS>;
  T* orh = o + (MAT ? L::RHS0 : 0);
#pragma unroll
  for (int n = 0; n < 4; ++n) put4(orh + 4 * n, ru[n][0], ru[n][1], ru[n][2], rp[n]);
  if constexpr (MAT) put4(o + L::C0, KA, KB, MM, target ? fact2 * w : (T)0);
  if constexpr (MAT)
    block_sums<T, OVS_ASM_NS>(q, g, target ? w : (T)0, (T)p.almi, fact2, rho, o);
}

// One Gauss point of the NS+VOF quench routine (src/solveQuenching.f90:
// 295-523): the point values q (layout GQ of Lay<NSVOF>) and, on fluid
// elements, the point's terms of KA, KB, MM, KDP and of the residual rows,
// added to the accumulators.  The viscous RHS broadcast (:508-510) is kept:
// the three scalars sum_j gN_a,j (du(j,k) + du(k,j)), k = 1..3, are
// subtracted from every momentum component.  ui, umi, aci, pri, phid (FP64),
// rphii, Ti: the fields at the point; N: its shape values.
// Reciprocals taken once per element for the Gauss-point routines: of the
// launch constants ts, rhoa, rhow, tref and of the element's trG, GG and
// sqrt(GG).  The point formulas multiply by them where the reference
// divides (a quotient and the product with the reciprocal differ by
// rounding only); each FP64 division is a reciprocal sequence of its own.
// At a point, one reciprocal of rho (rho cp for the temperature) serves
// nu, tauM (kk, tauT), and 1/sqrt is the reciprocal square root
// (inv_sqrt).  Measured for the FP64 element passes at 128^3: NS+VOF 5.9
// -> 4.35 ms with the per-element reciprocals -> 4.24 ms with the point
// ones, T 2.45 -> 1.74 -> 1.62 ms (FP32: 3.83 -> 2.78 and 1.25 -> 0.91).
template <typename T> struct PointInv {
  T ts, rhoa, rhow, tref, trG, GG, sGG, taut;   // taut = 4 / delt^2 itself
};
template <typename T>
__device__ __forceinline__ PointInv<T> point_inv(const ovs_params& p, T trG, T GG) {
  PointInv<T> iv;
  iv.taut = (T)(4.0 / (p.delt * p.delt));
  iv.ts = (T)(1.0 / p.ts);
  iv.rhoa = (T)(1.0 / p.rhoa);
  iv.rhow = (T)(1.0 / p.rhow);
  iv.tref = (T)(1.0 / p.tref);
  iv.trG = (T)1.0 / trG;
  iv.GG = (T)1.0 / GG;
  iv.sGG = (T)1.0 / sqrt(GG);
  return iv;
}

template <typename T>
__device__ __forceinline__ void nsvof_point(const ovs_params& p, bool fluid, const T (&N)[4], const T (&g)[4][3],
                                            const T (&G)[3][3], T GG, T trG, T w, const T (&du)[3][3],
                                            const T (&dp)[3], const T (&dphi)[3], T divu, const T (&svis)[4],
                                            const T (&gdphi)[4], const T (&ui)[3], const T (&umi)[3],
                                            const T (&aci)[3], T pri, double phid, T rphii, T Ti,
                                            T* q, T& KA, T& KB, T& MM, T& KDP, T (&ru)[4][3], T (&rp)[4],
                                            T (&rf)[4], double& tamax, const PointInv<T>& iv) {
  const T fact2 = (T)(p.alfi * p.delt * p.gami);
  const T taut = iv.taut;
  const T rhoa = (T)p.rhoa, rhow = (T)p.rhow, ts = (T)p.ts;
  const T ira = iv.rhoa - iv.rhow;
  const bool kdc_on = fabs(p.ns_kdc_w) + fabs(p.ns_kdc_a) > 0.0;
  const bool kdcphi_on = fabs(p.lsc_kdc) > 0.0;
  const T phii = (T)phid;
  const double phicd = clamp01(phid);
  const T phic = (T)phicd;
  T mdot, dmd;
  if (Ti > ts) {
    mdot = (T)p.c_evap * (T)(1.0 - phicd) * rhow * (Ti - ts) * iv.ts;
    dmd = -(T)p.c_evap * rhow * (Ti - ts) * iv.ts * (T)p.c_dmdot;
  } else {
    mdot = (T)p.c_cond * phic * rhoa * (Ti - ts) * iv.ts;
    dmd = (T)p.c_cond * rhoa * (Ti - ts) * iv.ts * (T)p.c_dmdot;
  }
  const T vdot = mdot * iv.rhoa - mdot * iv.rhow;
  T rho, mu;
  if (fluid) {
    rho = (T)(p.rhow * (1.0 - phicd) + p.rhoa * phicd);
    mu = (T)(p.muw * (1.0 - phicd) + p.mua * phicd);
  } else {
    rho = (T)p.rhos; mu = (T)p.mus;
  }
  const T lambda = (T)(-2.0 / 3.0) * mu;
  if (phid < 0.0 || phid > 1.0) dmd = 0;
  const T uadv[3] = {ui[0] - umi[0], ui[1] - umi[1], ui[2] - umi[2]};
  T tmp1[3], rL[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T conv = du[i][0] * uadv[0] + du[i][1] * uadv[1] + du[i][2] * uadv[2];
    tmp1[i] = rho * aci[i] + rho * conv - (T)p.gravvec[i] * rho;
    rL[i] = tmp1[i] + dp[i];
  }
  const T res_phi = rphii + (uadv[0] * dphi[0] + uadv[1] * dphi[1] + uadv[2] * dphi[2]) + phii * vdot - mdot * iv.rhoa;
  const T taua = quad_uGu<T>(uadv, G);
  const T irho = (T)1.0 / rho;
  const T nu = mu * irho;
  const T taud = nu * nu * (T)12.0 * GG;
  const T tauM = irho * inv_sqrt(taut + taua + taud);
  const T tauLS = inv_sqrt(taut + taua);
  const T tauC = rho * sqrt(taua + taud) * iv.trG;
  if constexpr (CflPerPoint<T, OVS_ASM_NSVOF>::v) {
    const double cf = (double)p.delt * sqrt((double)taua);
    if (cf > tamax) tamax = cf;
  } else if ((double)taua > tamax) {
    tamax = (double)taua;   // CFL number: delt sqrt(max taua), in the kernel
  }
  T kdc = 0;
  if (kdc_on) {
    const double nk = (double)(p.ns_kdc_w * (1.0 - phicd) + p.ns_kdc_a * phicd);
    const T rr = rL[0] * rL[0] + rL[1] * rL[1] + rL[2] * rL[2];
    kdc = (T)low_word(nk) * sqrt(rr * iv.GG);
  }
  T kdphi = 0;
  if (kdcphi_on) kdphi = (T)p.lsc_kdc * fabs(res_phi) * iv.sGG;
  const T mupk = mu + kdc;
  const T dmdi = dmd * ira;
  q[0] = uadv[0]; q[1] = uadv[1]; q[2] = uadv[2];
  q[3] = rho; q[4] = rho * tauM; q[5] = tauLS;
  q[6] = vdot + phii * ira * dmd - dmd * iv.rhoa;
  const T wf = fluid ? w : (T)0;   // solid elements contribute nothing
  q[7] = fact2 * wf * tauC * dmdi * dmdi;
  q[8] = fact2 * tauC * dmdi * wf;
  q[9] = fact2 * dmdi * wf;
  if (!fluid) return;
  KA += fact2 * mupk * w;
  KB += fact2 * (tauC + lambda) * w;
  MM += fact2 * w * tauM;
  KDP += fact2 * w * kdphi;
  T c[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) c[n] = uadv[0] * g[n][0] + uadv[1] * g[n][1] + uadv[2] * g[n][2];
  const T tdiv = -pri + tauC * divu;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      ru[n][i] += w * (-N[n] * tmp1[i] - g[n][i] * tdiv + g[n][i] * tauC * vdot - g[n][i] * lambda * divu -
                       mupk * svis[n] + rho * c[n] * (-tauM * rL[i]));
    rp[n] += w * (-N[n] * (divu - vdot) + (g[n][0] * rL[0] + g[n][1] * rL[1] + g[n][2] * rL[2]) * (-tauM));
    rf[n] += w * (-(N[n] + tauLS * c[n]) * res_phi - kdphi * gdphi[n] + N[n] * dmdi * tauC * (divu - vdot));
  }
}

// svis (the viscous broadcast) and g . grad phi per node, from the
// gradients
template <typename T>
__device__ __forceinline__ void nsvof_node_terms(const T (&g)[4][3], const T (&du)[3][3], const T (&dphi)[3],
                                                 T (&svis)[4], T (&gdphi)[4]) {
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    T sv = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k)
      sv += g[n][0] * (du[0][k] + du[k][0]) + g[n][1] * (du[1][k] + du[k][1]) + g[n][2] * (du[2][k] + du[k][2]);
    svis[n] = sv;
    gdphi[n] = g[n][0] * dphi[0] + g[n][1] * dphi[1] + g[n][2] * dphi[2];
  }
}

// pass 1, NS+VOF quench (src/solveQuenching.f90:295-523), one thread per
// element: geometry and gradients, the four Gauss points (nsvof_point),
// then the residual rows, the element constants and the block sums
template <typename T, bool MAT = true, typename RA, typename LA>
__device__ void summarize_nsvof(const SumArgs& a, const RA& r, const LA& lo, bool fluid, T* o,
                                double& tamax, T& detj_out) {
  const ovs_params& p = a.p;
  T g[4][3], G[3][3], detj, GG, trG;
  element_geometry<T>(r, lo, g, G, detj, GG, trG);
  detj_out = detj;
  const T w = detj * (T)(0.25 / 6.0);
  T du[3][3], dp[3], dphi[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      du[i][j] = r[0][3 + i] * g[0][j] + r[1][3 + i] * g[1][j] + r[2][3 + i] * g[2][j] + r[3][3 + i] * g[3][j];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    dp[j] = r[0][12] * g[0][j] + r[1][12] * g[1][j] + r[2][12] * g[2][j] + r[3][12] * g[3][j];
    dphi[j] = r[0][13] * g[0][j] + r[1][13] * g[1][j] + r[2][13] * g[2][j] + r[3][13] * g[3][j];
  }
  const T divu = du[0][0] + du[1][1] + du[2][2];
  T svis[4], gdphi[4];
  nsvof_node_terms<T>(g, du, dphi, svis, gdphi);
  const PointInv<T> iv = point_inv<T>(p, trG, GG);
  T KA = 0, KB = 0, MM = 0, KDP = 0;
  T ru[4][3], rp[4], rf[4], q[4][Lay<OVS_ASM_NSVOF>::GQ];
#pragma unroll
  for (int n = 0; n < 4; ++n) { ru[n][0] = ru[n][1] = ru[n][2] = 0; rp[n] = 0; rf[n] = 0; }
#pragma unroll (std::is_same<RA, SmemRecs<T>>::value ? 1 : 4)
  for (int gp = 0; gp < 4; ++gp) {
    T N[4];
    tet_shape<T>(gp, N);
    T ui[3], umi[3], aci[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      ui[d] = r[0][3 + d] * N[0] + r[1][3 + d] * N[1] + r[2][3 + d] * N[2] + r[3][3 + d] * N[3];
      umi[d] = r[0][6 + d] * N[0] + r[1][6 + d] * N[1] + r[2][6 + d] * N[2] + r[3][6 + d] * N[3];
      aci[d] = r[0][9 + d] * N[0] + r[1][9 + d] * N[1] + r[2][9 + d] * N[2] + r[3][9 + d] * N[3];
    }
    const T pri = r[0][12] * N[0] + r[1][12] * N[1] + r[2][12] * N[2] + r[3][12] * N[3];
    const double phid = gp_phi<T>(r, lo, 13, gp);   // VOF in FP64 for the 1000:1 property blend
    const T rphii = r[0][14] * N[0] + r[1][14] * N[1] + r[2][14] * N[2] + r[3][14] * N[3];
    const T Ti = r[0][15] * N[0] + r[1][15] * N[1] + r[2][15] * N[2] + r[3][15] * N[3];
    nsvof_point<T>(p, fluid, N, g, G, GG, trG, w, du, dp, dphi, divu, svis, gdphi, ui, umi, aci, pri, phid, rphii, Ti,
                   q[gp], KA, KB, MM, KDP, ru, rp, rf, tamax, iv);
  }
  using L = Lay<OVS_ASM_NSVOF>;
  if constexpr (MAT) {
#pragma unroll
    for (int n = 0; n < 4; ++n) put4(o + L::RHS0 + 4 * n, ru[n][0], ru[n][1], ru[n][2], rp[n]);
    put4(o + L::RHS0 + 16, rf[0], rf[1], rf[2], rf[3]);
    put4(o + L::C0, KA, KB, MM, KDP);
    put4(o + L::C0 + 4, dphi[0], dphi[1], dphi[2], fluid ? (T)(p.alfi * p.delt * p.gami) * w : (T)0);
  } else {   // 5 values per node
    T rh[20];
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      rh[5 * n] = ru[n][0]; rh[5 * n + 1] = ru[n][1]; rh[5 * n + 2] = ru[n][2];
      rh[5 * n + 3] = rp[n]; rh[5 * n + 4] = rf[n];
    }
#pragma unroll
    for (int k = 0; k < 20; k += 4) put4(o + k, rh[k], rh[k + 1], rh[k + 2], rh[k + 3]);
  }
  if constexpr (MAT)
    block_sums<T, OVS_ASM_NSVOF>(q, g, fluid ? w : (T)0, (T)p.almi, (T)(p.alfi * p.delt * p.gami), (T)0, o);
}

// pass 1, temperature (src/solveQuenching.f90:712-856).  Record layout of
// this pass: xd(0:2) u(3:5) um(6:8) phi(9) T(10) rT(11).  The element matrix
// (:814-839) is formed here, per Gauss point
//   K(a,b) += w (Na + trc ca) (rcp (fact1 Nb + fact2 cb) - fact2 dSe Nb)
// with trc = tauT rho cp, c_n = uadv . grad N_n, then K(a,b) += HK gab; solid
// elements take uadv = dSe = trc = 0, which turns the fluid block formula
// into the solid one.
template <typename T, bool MAT = true, typename RA, typename LA>
__device__ void summarize_tem(const SumArgs& a, const RA& r, const LA& lo, bool fluid, T* o,
                              double& tamax, T& detj_out) {
  const ovs_params& p = a.p;
  T g[4][3], G[3][3], detj, GG, trG;
  element_geometry<T>(r, lo, g, G, detj, GG, trG);
  detj_out = detj;
  const T w = detj * (T)(0.25 / 6.0);
  const PointInv<T> iv = point_inv<T>(p, trG, GG);
  T dT[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) dT[j] = r[0][10] * g[0][j] + r[1][10] * g[1][j] + r[2][10] * g[2][j] + r[3][10] * g[3][j];
  const T fact2 = (T)(p.alfi * p.gami * p.delt);
  const T ts = (T)p.ts, cpw = (T)p.cpw, cpa = (T)p.cpa, lh = (T)p.lh;
  T gdT[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) gdT[n] = g[n][0] * dT[0] + g[n][1] * dT[1] + g[n][2] * dT[2];
  T HK = 0, rt[4] = {0, 0, 0, 0};
  const T fact1 = (T)p.almi;
  T K[4][4];
#pragma unroll
  for (int ia = 0; ia < 4; ++ia)
#pragma unroll
    for (int ib = 0; ib < 4; ++ib) K[ia][ib] = (T)0;
  const bool kdc_on = fabs(p.tem_kdc) > 0.0;
#pragma unroll
  for (int gp = 0; gp < 4; ++gp) {
    T N[4];
    tet_shape<T>(gp, N);
    const double phid = gp_phi<T>(r, lo, 9, gp);
    const T Ti = r[0][10] * N[0] + r[1][10] * N[1] + r[2][10] * N[2] + r[3][10] * N[3];
    const T rTi = r[0][11] * N[0] + r[1][11] * N[1] + r[2][11] * N[2] + r[3][11] * N[3];
    T ui[3], umi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      ui[d] = r[0][3 + d] * N[0] + r[1][3 + d] * N[1] + r[2][3 + d] * N[2] + r[3][3 + d] * N[3];
      umi[d] = r[0][6 + d] * N[0] + r[1][6 + d] * N[1] + r[2][6 + d] * N[2] + r[3][6 + d] * N[3];
    }
    const double phicd = clamp01(phid);
    const T phic = (T)phicd;
    T mdot, dmdT;
    if (Ti > ts) {
      mdot = (T)p.c_evap * (T)(1.0 - phicd) * (T)p.rhow * (Ti - ts) * iv.ts;
      dmdT = (T)p.c_evap * (T)(1.0 - phicd) * (T)p.rhow * iv.ts * (T)p.c_dmdot;
    } else {
      mdot = (T)p.c_cond * phic * (T)p.rhoa * (Ti - ts) * iv.ts;
      dmdT = (T)p.c_cond * phic * (T)p.rhoa * iv.ts * (T)p.c_dmdot;
    }
    T rho, cp, hk, rcp;
    if (fluid) {
      rho = (T)(p.rhow * (1.0 - phicd) + p.rhoa * phicd);
      cp = (T)(p.cpw * (1.0 - phicd) + p.cpa * phicd);
      hk = (T)(p.kappaw * (1.0 - phicd) + p.kappaa * phicd);
      rcp = (T)((p.rhow * p.cpw) * (1.0 - phicd) + (p.rhoa * p.cpa) * phicd);
    } else {
      rho = (T)p.rhos; cp = (T)p.cps; hk = (T)p.kappas; rcp = (T)(p.rhos * p.cps);
    }
    const T uadv[3] = {ui[0] - umi[0], ui[1] - umi[1], ui[2] - umi[2]};
    const T Se = ((cpw - cpa) * (Ti - ts) - lh) * mdot;
    const T udT = uadv[0] * dT[0] + uadv[1] * dT[1] + uadv[2] * dT[2];
    const T res = rcp * (rTi + udT) - Se;
    const T taua = quad_uGu<T>(uadv, G);
    T tt = taua + iv.taut;
    const T ircp = (T)1.0 / (rho * cp);
    const T kk = hk * ircp;
    tt = tt + kk * kk * (T)12.0 * GG;
    const T tauT = ircp * inv_sqrt(tt);
    if ((double)taua > tamax) tamax = (double)taua;   // CFL number: delt sqrt(max taua), in the kernel
    T kdcT = 0;
    if (kdc_on && fluid) kdcT = (T)p.tem_kdc * fabs(res) * iv.sGG * iv.tref;
    const T dSe = (cpw - cpa) * mdot + ((cpw - cpa) * (Ti - ts) - lh) * dmdT;
    if constexpr (MAT) {
      const T uq[3] = {fluid ? uadv[0] : (T)0, fluid ? uadv[1] : (T)0, fluid ? uadv[2] : (T)0};
      const T dSq = fluid ? dSe : (T)0, trq = fluid ? tauT * rcp : (T)0;
      T cq[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) cq[n] = g[n][0] * uq[0] + g[n][1] * uq[1] + g[n][2] * uq[2];
#pragma unroll
      for (int ia = 0; ia < 4; ++ia) {
        const T aw = w * (N[ia] + trq * cq[ia]);
#pragma unroll
        for (int ib = 0; ib < 4; ++ib) K[ia][ib] += aw * (rcp * (fact1 * N[ib] + fact2 * cq[ib]) - fact2 * dSq * N[ib]);
      }
    }
    if (fluid) {
      HK += fact2 * (hk + kdcT) * w;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const T cn = uadv[0] * g[n][0] + uadv[1] * g[n][1] + uadv[2] * g[n][2];
        rt[n] += w * (-N[n] * rcp * (rTi + udT) + N[n] * Se - rcp * tauT * cn * res - (hk + kdcT) * gdT[n]);
      }
    } else {
      HK += fact2 * hk * w;
#pragma unroll
      for (int n = 0; n < 4; ++n) rt[n] += w * (-N[n] * rcp * rTi - hk * gdT[n]);
    }
  }
#pragma unroll
  for (int ia = 0; ia < 4; ++ia) {
    if constexpr (MAT) {
      o[Lay<OVS_ASM_TEM>::RHS0 + 2 * ia + 1] = rt[ia];
#pragma unroll
      for (int ib = 0; ib < 4; ++ib)
        o[ia == ib ? Lay<OVS_ASM_TEM>::RHS0 + 2 * ia
                   : 2 * (ia < ib ? tet_edge(ia, ib) : tet_edge(ib, ia)) + (ia < ib ? 0 : 1)] =
            K[ia][ib] + HK * (g[ia][0] * g[ib][0] + g[ia][1] * g[ib][1] + g[ia][2] * g[ib][2]);
    } else {
      o[ia] = rt[ia];
    }
  }
}

// -------------------------------------------------- pass 2: block expansion
// 4 consecutive values with one read-only load (FP64: the 256-bit load of
// sm_100; summary groups are 32-byte aligned there)
__device__ __forceinline__ void ldv4(const float* p, float* d) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(p));
  d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
}
__device__ __forceinline__ void ldv4(const double* p, double* d) {
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(d[0]), "=d"(d[1]), "=d"(d[2]), "=d"(d[3]) : "l"(p));
}
// 2 consecutive values
__device__ __forceinline__ void ldv2(const float* p, float* d) {
  const float2 v = __ldg(reinterpret_cast<const float2*>(p));
  d[0] = v.x; d[1] = v.y;
}
__device__ __forceinline__ void ldv2(const double* p, double* d) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(p));
  d[0] = v.x; d[1] = v.y;
}

// the summary values an NS/NS+VOF block (row node a, column node b) is formed
// from: the nodes' gradients and U, Q of the row, T of the column, the element
// constants and the pair sums
template <typename T> struct BlockIn {
  T ga[4], gb[4], Qa, Tb, cs[8], pr[4];
};

template <typename T, int KIND>
__device__ __forceinline__ void load_block(const T* sm, int a, int b, BlockIn<T>& in) {
  using L = Lay<KIND>;
  ldv4(sm + L::ND0 + 4 * a, in.ga);
  ldv4(sm + L::ND0 + 4 * b, in.gb);
  ldv4(sm + L::C0, in.cs);
  if constexpr (KIND == OVS_ASM_NSVOF) {
    ldv4(sm + L::C0 + 4, in.cs + 4);
    ldv4(sm + L::PW * (4 * a + b), in.pr);
  } else {
    in.pr[0] = __ldg(sm + L::PW * (4 * a + b));
  }
  in.Tb = __ldg(sm + L::T0 + b);
  in.Qa = __ldg(sm + L::T0 + 4 + a);
}

// Block of row node a, column node b added to o (formulas factored from the
// reference's per Gauss point sums, with the sums of block_sums):
//   K(i,j) = KA ga_j gb_i + KB ga_i gb_j + delta_ij (KA gab + S_ab)
//   G(i) = -ga_i PR + gb_i Q_a      D(i) = gb_i PR + ga_i T_b
//   M = MM gab    LS = L1_ab + E_ab + KDP gab    ULS(i) = ga_i U_b
//   PLS = PL_ab   LSU(i) = dphi_i V_ab - gb_i U_a
template <typename T, int KIND>
__device__ __forceinline__ void add_block(const BlockIn<T>& in, T* o) {
  constexpr bool vof = KIND == OVS_ASM_NSVOF;
  const T KA = in.cs[0], KB = in.cs[1], MM = in.cs[2], PR = vof ? in.cs[7] : in.cs[3];
  const T gab = in.ga[0] * in.gb[0] + in.ga[1] * in.gb[1] + in.ga[2] * in.gb[2];
  const T dg = KA * gab + in.pr[0];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T ka = KA * in.gb[i], kb = KB * in.ga[i];
#pragma unroll
    for (int j = 0; j < 3; ++j) o[4 * i + j] += ka * in.ga[j] + kb * in.gb[j];
    o[5 * i] += dg;
    o[4 * i + 3] += in.gb[i] * in.Qa - in.ga[i] * PR;
    o[12 + i] += in.gb[i] * PR + in.ga[i] * in.Tb;
  }
  o[15] += MM * gab;
  if constexpr (vof) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      o[16 + d] += in.cs[4 + d] * in.pr[3] - in.gb[d] * in.ga[3];
      o[20 + d] += in.ga[d] * in.gb[3];
    }
    o[19] += in.pr[1] + in.cs[3] * gab;
    o[23] += in.pr[2];
  }
}

template <typename T> struct Vec4 {};
template <> struct Vec4<float> {
  __device__ static void add(float* dst, const float* src) {
    float4 a = *reinterpret_cast<float4*>(dst);
    float4 b = *reinterpret_cast<const float4*>(src);
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    *reinterpret_cast<float4*>(dst) = a;
  }
};
template <> struct Vec4<double> {
  __device__ static void add(double* dst, const double* src) {
    double2 a0 = reinterpret_cast<double2*>(dst)[0], a1 = reinterpret_cast<double2*>(dst)[1];
    double2 b0 = reinterpret_cast<const double2*>(src)[0], b1 = reinterpret_cast<const double2*>(src)[1];
    a0.x += b0.x; a0.y += b0.y; a1.x += b1.x; a1.y += b1.y;
    reinterpret_cast<double2*>(dst)[0] = a0;
    reinterpret_cast<double2*>(dst)[1] = a1;
  }
};

// ---------------------------------------------------------- pass 1 kernel
// blocks per SM the element pass is compiled for: the FP32 NS+VOF pass at 3
// (168 registers, measured faster than the unbounded 178 and than 2 or 4),
// the FP32 temperature pass at 4 (1.25 against 1.45 ms at 160 registers),
// the others as the compiler chooses (the FP64 temperature pass measured
// slower at 3)
template <typename T, int KIND> struct SumMinBlocks { static constexpr int v = 1; };
template <> struct SumMinBlocks<float, OVS_ASM_NSVOF> { static constexpr int v = 3; };
template <> struct SumMinBlocks<float, OVS_ASM_TEM> { static constexpr int v = 4; };

template <typename T, int KIND, bool SMEMREC> struct SumBlocks { static constexpr int v = SumMinBlocks<T, KIND>::v; };
// FP64 with the node records in shared memory: 2 blocks (up to 255
// registers, measured 7.1 ms for NS+VOF at 128^3 against 7.6 ms at 3
// blocks and 10.2 ms at 4)
template <int KIND> struct SumBlocks<double, KIND, true> { static constexpr int v = 2; };

// MAT false (vector-only pass): the summary is the residual rows alone, 4 NF
// values per element.
template <typename T, int KIND, bool SMEMREC, bool MAT = true>
__global__ void __launch_bounds__(128, (MAT ? SumBlocks<T, KIND, SMEMREC>::v : SMEMREC ? 3 : 1))
element_summary_kernel(const SumArgs a) {
  using L = Lay<KIND>;
  constexpr int SW = MAT ? L::SW : 4 * L::NF;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double tamax = 0.0;   // the element's largest taua over its points (CflPerPoint: largest CFL number)
  int nbad = 0;
  if (t < a.E) {
    const int4 nd = __ldg(reinterpret_cast<const int4*>(a.ien) + t);
    const int nodes[4] = {nd.x, nd.y, nd.z, nd.w};
    const T* rec = reinterpret_cast<const T*>(a.rec);
    const int eid = __ldg(a.elm_id + t);
    T detj;
    auto run = [&](const auto& r, const auto& lo, T* o) {
      if constexpr (KIND == OVS_ASM_NS) {
        const bool target = ((a.p.subdomain_flag & 1) && eid == a.p.elm_id_set[0]) ||
                            ((a.p.subdomain_flag & 2) && eid == a.p.elm_id_set[1]);
        summarize_ns<T, MAT>(a, r, lo, target, o, tamax, detj);
      } else if constexpr (KIND == OVS_ASM_NSVOF) {
        summarize_nsvof<T, MAT>(a, r, lo, eid == a.p.fluid_elm_id, o, tamax, detj);
      } else {
        summarize_tem<T, MAT>(a, r, lo, eid == a.p.fluid_elm_id, o, tamax, detj);
      }
    };
    if constexpr (SMEMREC && sizeof(T) == 8) {
      // records through shared memory; the summary written straight to
      // global memory as its values are produced
      extern __shared__ __align__(16) unsigned char sm_elem[];
      T* col = reinterpret_cast<T*>(sm_elem) + threadIdx.x;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const double2* q = reinterpret_cast<const double2*>(rec) + (size_t)nodes[n] * (REC / 2);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const double2 v = __ldg(q + k);
          col[(size_t)(n * 16 + 2 * k) * 128] = v.x;
          col[(size_t)(n * 16 + 2 * k + 1) * 128] = v.y;
        }
      }
      run(SmemRecs<T>{col}, ZeroRecs<T>{}, reinterpret_cast<T*>(a.sum) + (size_t)t * SW);
    } else {
      T r[4][16], lo[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) load_rec(rec, nodes[n], r[n], lo[n]);
      if constexpr (KIND == OVS_ASM_TEM) {
        T o[SW];
        run(r, lo, o);
        // 20 values per tet (vector-only: 4): groups of 4 (256-bit stores in FP64, the
        // summary 32-byte aligned; 2.45 against 2.52 ms at 128^3)
        T* dst = reinterpret_cast<T*>(a.sum) + (size_t)t * SW;
        if constexpr (sizeof(T) == 8) {
#pragma unroll
          for (int k = 0; k < SW; k += 4) put4(dst + k, o[k], o[k + 1], o[k + 2], o[k + 3]);
        } else {
          store_row<SW>(dst, o);
        }
      } else {
        // NS / NS+VOF write their summary with vector stores as its parts
        // are formed
        run(r, lo, reinterpret_cast<T*>(a.sum) + (size_t)t * SW);
      }
    }
    if (!(detj > (T)0)) nbad = 1;
  }
  // the CFL number of the element (CflPerPoint: already the number itself)
  double cfl = CflPerPoint<T, KIND>::v ? tamax : (double)a.p.delt * sqrt(tamax);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    cfl = fmax(cfl, __shfl_xor_sync(0xffffffffu, cfl, off));
    nbad += __shfl_xor_sync(0xffffffffu, nbad, off);
  }
  if ((threadIdx.x & 31) == 0) {
    cfl_max(a.cfl_bits, cfl);
    if (nbad) atomicAdd(a.flags, nbad);
  }
}

// ---------------------------------------------------------- pass 2 kernel
// The masks of the Dirichlet treatment, per value position v:
// bits 0-7 row (A) constraints, 8-15 column (B) constraints, 16-23 the
// diagonal entry set to 1 per element.
__device__ __forceinline__ unsigned mask_of(int v) {
  return (unsigned)c_rowbits[v] | ((unsigned)c_colbits[v] << 8) | ((unsigned)c_diagbit[v] << 16);
}

// Edge pass (tets).  A block of 4 warps takes a tile of OVS_TILE_ROWS
// consecutive rows of the row order (Morton order of the nodes, so that what
// runs at a time shares its elements and reads their summaries from L2): the
// diagonal blocks and residuals of the tile's rows, 8 lanes per row, then the
// edges the tile owns (those whose other node comes later in the order), in
// sets of 16, two lanes per edge: lane 0 the entry (A, B), lane 1 (B, A).
// Every entry adds its elements in ascending order; a diagonal block adds
// lane l's elements l, l + 8, ... and then the lanes by halving: orders fixed
// by the mesh, the same on every run.
// Bound: the summaries are read in scattered 32-byte pieces, which the L1
// data path serves at a quarter of its rate (L1 67% busy in FP64), and the loads'
// latency at 10.6 warps per SM (12.6 cycles of waiting per instruction).  So what
// counts is the bytes a block asks for, how many distinct elements a load touches
// and how many loads are in flight: 22 values per block, and the two lanes of an
// edge read the same element.  A warp per
// row with one list per entry (28 values, 24 elements a load, an exchange
// through shared memory) took 12.65 ms for the FP64 NS+VOF rows of the
// 128^3 x6 tets and 6.91 ms in FP32; this takes 5.91 and 3.35 ms (T: 1.90 ->
// 0.66 and 1.43 -> 0.48 ms).  A tile's edges are sorted by list
// length, so the rounds of a set are nearly equal.
template <typename T, int KIND>
__device__ __forceinline__ void write_entry(T* dst, T* v, const unsigned* masks, unsigned ibA, unsigned ibB) {
  constexpr int NV = Lay<KIND>::NV;
  if ((ibA | ibB) != 0u) {
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      const unsigned m = masks[u];
      if ((ibA & m & 0xffu) || ((ibB << 8) & m & 0xff00u)) v[u] = (T)0;
    }
  }
#pragma unroll
  for (int g = 0; g < NV; g += 4) store4_cs(dst + g, v + g);
}

// the diagonal block of row rr and its residual (8 lanes, l8 their index)
template <typename T, int KIND>
__device__ __forceinline__ void diag_row(const AsmArgs& a, const int4 rr, bool on, int l8, const unsigned* masks) {
  using L = Lay<KIND>;
  constexpr int NV = L::NV, NF = L::NF, NG = NV / 4;
  const int A = rr.x, deg = rr.w & 0xff, sd = (rr.w >> 8) & 0xff, ne = on ? rr.w >> 16 : 0;
  const T* sum = reinterpret_cast<const T*>(a.rec);
  T v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = (T)0;
  int pk = l8 < ne ? __ldg(a.n2e + rr.z + l8) : 0;
  for (int q = l8; q < ne; q += 8) {
    const int la = pk & 7;
    const T* se = sum + (size_t)(pk >> 3) * L::SW;
    if (q + 8 < ne) pk = __ldg(a.n2e + rr.z + q + 8);
    BlockIn<T> in;
    T r[4];
    load_block<T, KIND>(se, la, la, in);
    ldv4(se + L::RHS0 + 4 * la, r);
    add_block<T, KIND>(in, v);
#pragma unroll
    for (int f = 0; f < 4; ++f) v[NV + f] += r[f];
    if constexpr (NF == 5) v[NV + 4] += __ldg(se + L::RHS0 + 16 + la);
  }
  // lane l ends up with group l, the values 4 l .. 4 l + 3
#pragma unroll
  for (int half = 16, off = 4; off >= 1; half >>= 1, off >>= 1) {
    const bool up = l8 & off;
#pragma unroll
    for (int k = 0; k < half; ++k) {
      const T send = up ? v[k] : v[k + half], keep = up ? v[k + half] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  if (!on) return;
  const int g = l8;
  const unsigned ibA = __ldg(a.ibc + A);
  if (g < NG) {
    if (deg > 0) {
      const T cnt = (T)(rr.w >> 16);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned m = masks[4 * g + u];
        if ((ibA & m & 0xffu) || ((ibA << 8) & m & 0xff00u)) v[u] = (T)0;
        if ((ibA << 16) & m & 0xff0000u) v[u] = cnt;
      }
      store4_cs(reinterpret_cast<T*>(a.vals) + ((size_t)rr.y + sd) * NV + 4 * g, v);
    }
  } else if (a.vec) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int f = 4 * (g - NG) + u;
      if (f < NF) {
        const T x = (ibA & (1u << f)) ? (T)0 : v[u];   // IBC bits 0-4: u1 u2 u3 p phi
        if (!isfinite((double)x)) atomicOr(a.flags + 1, 1);
        __stcs(reinterpret_cast<T*>(a.rhs) + (size_t)f * a.N + A, x);
      }
    }
  }
}

template <typename T, int KIND>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 3 : 4) edge_rows_kernel(const AsmArgs a) {
  using L = Lay<KIND>;
  constexpr int NV = L::NV;
  __shared__ unsigned masks[24];
  if (threadIdx.x < 24) masks[threadIdx.x] = mask_of(threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, tile = blockIdx.x;
#pragma unroll 1
  for (int r = 4 * wid; r < OVS_TILE_ROWS; r += 16) {
    const int t = tile * OVS_TILE_ROWS + r + (lane >> 3);
    const bool on = t < a.N;
    const int4 rr = on ? __ldg(a.row_rec + t) : make_int4(0, 0, 0, 0);
    diag_row<T, KIND>(a, rr, on, lane & 7, masks);
  }
  const T* sum = reinterpret_cast<const T*>(a.rec);
  T* vals = reinterpret_cast<T*>(a.vals);
  const int p = lane & 1;
  const unsigned e1 = __ldg(a.tile_edge + tile + 1);
  unsigned i = __ldg(a.tile_edge + tile) + 16u * wid + (lane >> 1);
  // the next set's records and first list entry travel while a set runs
  int4 rec = make_int4(0, 0, 0, 0);
  unsigned c = 0, c1 = 0, ent = 0;
  if (i < e1) {
    rec = __ldg(a.edge_rec + i);
    c = __ldg(a.edge_ptr + i);
    c1 = __ldg(a.edge_ptr + i + 1);
    ent = __ldg(a.edge_list + c);
  }
  while (__any_sync(0xffffffffu, i < e1)) {
    const bool on = i < e1;
    const int4 cur = rec;
    const unsigned end = c1;
    unsigned pos = c, en = ent;
    i += 64u;
    c = c1 = 0;
    if (i < e1) {
      rec = __ldg(a.edge_rec + i);
      c = __ldg(a.edge_ptr + i);
      c1 = __ldg(a.edge_ptr + i + 1);
    }
    const unsigned ib = on ? __ldg(a.ibc + (p ? cur.y : cur.x)) : 0u;
    T acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = (T)0;
    // several elements' loads in flight (lists of 4 to 8 are the rule): FP64 four
    // at 3 blocks per SM, 6.63 -> 6.29 ms at 128^3 x6 with tiles of 32 rows (two or three 6.60 and 6.49,
    // six 6.51; 4 blocks: 7.23 with two), FP32 three at 4 blocks, 3.56 -> 3.34 (two
    // 3.37, four 3.38, 5 blocks 3.47)
    constexpr int UNR = sizeof(T) == 8 ? 4 : 3;
#pragma unroll UNR
    for (; pos < end; ++pos) {
      const unsigned now = en;
      if (pos + 1 < end) en = __ldg(a.edge_list + pos + 1);
      const int la = (now >> 2) & 3, lb = now & 3;
      BlockIn<T> in;
      load_block<T, KIND>(sum + (size_t)(now >> 4) * L::SW, p ? lb : la, p ? la : lb, in);
      add_block<T, KIND>(in, acc);
    }
    if (c < c1) ent = __ldg(a.edge_list + c);
    const unsigned other = __shfl_xor_sync(0xffffffffu, ib, 1);
    if (on) write_entry<T, KIND>(vals + (size_t)(p ? cur.w : cur.z) * NV, acc, masks, ib, other);
  }
}

// the same for the temperature system: its blocks are single values, so one
// lane takes both entries of an edge
template <typename T>
__global__ void __launch_bounds__(128) edge_rows_tem_kernel(const AsmArgs a) {
  using L = Lay<OVS_ASM_TEM>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, tile = blockIdx.x, l8 = lane & 7;
  const T* sum = reinterpret_cast<const T*>(a.rec);
  T* vals = reinterpret_cast<T*>(a.vals);
#pragma unroll 1
  for (int r = 4 * wid; r < OVS_TILE_ROWS; r += 16) {
    const int t = tile * OVS_TILE_ROWS + r + (lane >> 3);
    const bool on = t < a.N;
    const int4 rr = on ? __ldg(a.row_rec + t) : make_int4(0, 0, 0, 0);
    const int ne = rr.w >> 16;
    T k = (T)0, f = (T)0;
#pragma unroll 4
    for (int q = l8; q < ne; q += 8) {
      const int pk = __ldg(a.n2e + rr.z + q);
      T x[2];
      ldv2(sum + (size_t)(pk >> 3) * L::SW + L::RHS0 + 2 * (pk & 7), x);
      k += x[0];
      f += x[1];
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      k += __shfl_xor_sync(0xffffffffu, k, o);
      f += __shfl_xor_sync(0xffffffffu, f, o);
    }
    if (!on || l8) continue;
    const bool held = __ldg(a.ibc + rr.x) & TB;
    if (rr.w & 0xff) __stcs(vals + rr.y + ((rr.w >> 8) & 0xff), held ? (T)ne : k);
    if (a.vec) {
      const T x = held ? (T)0 : f;
      if (!isfinite((double)x)) atomicOr(a.flags + 1, 1);
      __stcs(reinterpret_cast<T*>(a.rhs) + rr.x, x);
    }
  }
  const unsigned e1 = __ldg(a.tile_edge + tile + 1);
  for (unsigned i = __ldg(a.tile_edge + tile) + threadIdx.x; i < e1; i += blockDim.x) {
    const int4 cur = __ldg(a.edge_rec + i);
    const unsigned end = __ldg(a.edge_ptr + i + 1);
    T kab = (T)0, kba = (T)0;
#pragma unroll 4
    for (unsigned q = __ldg(a.edge_ptr + i); q < end; ++q) {
      const unsigned now = __ldg(a.edge_list + q);
      const int la = (now >> 2) & 3, lb = now & 3;
      T x[2];
      ldv2(sum + (size_t)(now >> 4) * L::SW + 2 * (la < lb ? tet_edge(la, lb) : tet_edge(lb, la)), x);
      kab += la < lb ? x[0] : x[1];
      kba += la < lb ? x[1] : x[0];
    }
    const bool held = (__ldg(a.ibc + cur.x) | __ldg(a.ibc + cur.y)) & TB;
    __stcs(vals + cur.z, held ? (T)0 : kab);
    __stcs(vals + cur.w, held ? (T)0 : kba);
  }
}

// Row pass of a vector-only assembly (tets and hexahedra): 8 lanes per node
// add the element residuals of the node's elements, lane l the elements l,
// l + 8, ... of its ascending list, then the lanes' sums by halving, an order
// fixed by the mesh.  The residual evaluations of a Newton loop ask for no
// matrix; the full row pass formed every block for them (48x48x96 cells x6
// tets, FP64, both passes: 2.19 ms; this way 0.63 ms).
template <typename T, int NF>
__global__ void __launch_bounds__(256) residual_rows_kernel(const AsmArgs a, int nshl, bool tem) {
  const int lane = threadIdx.x & 31, l8 = lane & 7;
  const int A = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 3);
  const bool on = A < a.N;
  const T* sum = reinterpret_cast<const T*>(a.rec);
  T r[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) r[f] = (T)0;
  if (on) {
    const int ep = __ldg(a.n2e_ptr + A), ee = __ldg(a.n2e_ptr + A + 1);
    for (int q = ep + l8; q < ee; q += 8) {
      const int pk = __ldg(a.n2e + q);
      const T* p = sum + ((size_t)(pk >> 3) * nshl + (pk & 7)) * NF;
#pragma unroll
      for (int f = 0; f < NF; ++f) r[f] += __ldg(p + f);
    }
  }
#pragma unroll
  for (int f = 0; f < NF; ++f)
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) r[f] += __shfl_xor_sync(0xffffffffu, r[f], o);
  if (!on || l8 >= NF) return;
  T v = r[0];
#pragma unroll
  for (int f = 1; f < NF; ++f) v = l8 == f ? r[f] : v;
  const unsigned bit = tem ? TB : (l8 < 3 ? 1u << l8 : (l8 == 3 ? PB : FB));
  if (__ldg(a.ibc + A) & bit) v = (T)0;
  if (!isfinite((double)v)) atomicOr(a.flags + 1, 1);
  reinterpret_cast<T*>(a.rhs)[(size_t)l8 * a.N + A] = v;
}

// ---------------------------------------------------- alpha-stage records
// assembleQuenching / assembleNavSto alpha stage (src/solveQuenching.f90:26-37,
// src/assembleNavSto.f90:25-30) fused with the packing of the values the
// element kernels gather, 16 per node.
struct AlphaArgs {
  const double* f[OVS_F_COUNT];
  const double* xg;
  void* rec;
  int N;
  int tem;   // record layout of the temperature pass
  double almi, alfi;
};

template <typename T>
__global__ void alpha_records_kernel(const AlphaArgs a) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.N) return;
  const size_t N = a.N;
  const double am = a.almi, af = a.alfi;
  T r[REC];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const size_t k = i + N * d;
    const double dga = a.f[OVS_F_DGOLD][k] + af * (a.f[OVS_F_DG][k] - a.f[OVS_F_DGOLD][k]);
    const double xd = a.xg[k] + dga;   // xl + dl of eval_shape_fem (:34)
    r[d] = (T)xd;
    r[16 + d] = (T)(xd - (double)r[d]);
    r[3 + d] = (T)(a.f[OVS_F_UGOLD][k] + af * (a.f[OVS_F_UG][k] - a.f[OVS_F_UGOLD][k]));
    r[6 + d] = (T)(a.f[OVS_F_UGMOLD][k] + af * (a.f[OVS_F_UGM][k] - a.f[OVS_F_UGMOLD][k]));
    if (!a.tem) r[9 + d] = (T)(a.f[OVS_F_ACGOLD][k] + am * (a.f[OVS_F_ACG][k] - a.f[OVS_F_ACGOLD][k]));
  }
  const double phia = a.f[OVS_F_PHIGOLD][i] + af * (a.f[OVS_F_PHIG][i] - a.f[OVS_F_PHIGOLD][i]);
  const double ta = a.f[OVS_F_TGOLD][i] + af * (a.f[OVS_F_TG][i] - a.f[OVS_F_TGOLD][i]);
  r[19] = (T)(phia - (double)(T)phia);
  if (!a.tem) {
    r[12] = (T)a.f[OVS_F_PG][i];
    r[13] = (T)phia;
    r[14] = (T)(a.f[OVS_F_RPHIGOLD][i] + am * (a.f[OVS_F_RPHIG][i] - a.f[OVS_F_RPHIGOLD][i]));
    r[15] = (T)ta;
  } else {
    r[9] = (T)phia;
    r[10] = (T)ta;
    r[11] = (T)(a.f[OVS_F_RTGOLD][i] + am * (a.f[OVS_F_RTG][i] - a.f[OVS_F_RTGOLD][i]));
    r[12] = r[13] = r[14] = r[15] = (T)0;
  }
  T* o = reinterpret_cast<T*>(a.rec) + (size_t)i * REC;
#pragma unroll
  for (int k = 0; k < REC; ++k) o[k] = r[k];
}

template <typename T, int KIND>
int launch_edges(ovs_ctx* c, const AsmArgs& a) {
  const int tiles = (c->N + OVS_TILE_ROWS - 1) / OVS_TILE_ROWS;
  if constexpr (KIND == OVS_ASM_TEM) edge_rows_tem_kernel<T><<<tiles, 128, 0, c->stream>>>(a);
  else edge_rows_kernel<T, KIND><<<tiles, 128, 0, c->stream>>>(a);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

template <typename T, int NF>
int launch_residual_rows(ovs_ctx* c, const AsmArgs& a, bool tem) {
  residual_rows_kernel<T, NF><<<ovs_grid((size_t)c->N * 8, 256, 1 << 30), 256, 0, c->stream>>>(a, c->nshl, tem);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

// vector-only pass: the element residuals, then their sums per node.  The
// node records stay in registers unless the option asks for shared memory:
// without the matrix values that is the faster one in FP64 too (NS+VOF, both
// kernels and the alpha stage: 3.33 against 3.69 ms at 128^3, 0.41 against
// 0.45 ms at 48x48x96).
template <typename T, int KIND>
int launch_residual(ovs_ctx* c, const AsmArgs& a, const SumArgs& sa) {
  if (sizeof(T) == 8 && c->elem_smem > 0) {
    const size_t esm = sizeof(T) * 64 * 128;
    OVS_CUDA_TRY(cudaFuncSetAttribute(element_summary_kernel<T, KIND, true, false>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)esm));
    element_summary_kernel<T, KIND, true, false><<<(sa.E + 127) / 128, 128, esm, c->stream>>>(sa);
  } else {
    element_summary_kernel<T, KIND, false, false><<<(sa.E + 127) / 128, 128, 0, c->stream>>>(sa);
  }
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  return launch_residual_rows<T, Lay<KIND>::NF>(c, a, KIND == OVS_ASM_TEM);
}

// parts: bit 0 the element pass, bit 1 the row pass
template <typename T, int KIND>
int launch_assemble(ovs_ctx* c, const AsmArgs& a, const SumArgs& sa, int parts = 3) {
  if (!a.mat) return launch_residual<T, KIND>(c, a, sa);
  // pass 1: element summaries
  if (parts & 1) {
    if (sizeof(T) == 8 && (c->elem_smem > 0 || (c->elem_smem < 0 && KIND == OVS_ASM_NSVOF))) {
      // the node records of the block's 128 elements in shared memory
      const size_t esm = sizeof(T) * 64 * 128;
      OVS_CUDA_TRY(cudaFuncSetAttribute(element_summary_kernel<T, KIND, true>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)esm));
      element_summary_kernel<T, KIND, true><<<(sa.E + 127) / 128, 128, esm, c->stream>>>(sa);
    } else {
      element_summary_kernel<T, KIND, false><<<(sa.E + 127) / 128, 128, 0, c->stream>>>(sa);
    }
    ++c->launches;
    OVS_CUDA_TRY(cudaGetLastError());
  }
  if (!(parts & 2)) return OVS_OK;
  return launch_edges<T, KIND>(c, a);   // pass 2
}


// ------------------------------------------------ adjoint of the residual
// VJP of the assembled residual (the RHS the row pass writes, FP64) with
// respect to the nodal state, in reverse mode.  One thread per element
// contracts the element's residual rows with the cotangent (zero on Dirichlet
// rows, where the row pass writes 0), which leaves one scalar per Gauss point,
// and walks that point's formulas backwards: the adjoint of every
// intermediate, then of the fields at the point (spread to the nodes by the
// shape values), of the gradients and of the geometry.  Nothing is stored
// between assembly and adjoint.  A node pass sums the element terms in
// ascending element id (deterministic) and applies the alpha-stage chain
// factors: x+d_a = xg + ..., u_a = .. + alfi ug, p, phi_a = .. + alfi phig,
// T_a = .. + alfi Tg, a_a = .. + almi acg, phidot_a = .. + almi rphig,
// Tdot_a = .. + almi rTg (src/solveQuenching.f90:26-37).
// The cost is a few residual evaluations per element (196,608 tets: NS+VOF
// 0.21 ms, T 0.07 ms); the forward-mode form evaluated the residual on dual
// numbers once per nodal input, 52 times for NS+VOF (24 ms for both).
struct VjpArgs {
  const double* rec;      // FP64 alpha-stage records of the kernel's layout
  const int* ien;
  const int* elm_id;
  const uint8_t* ibc;
  const double* cot;      // NF*N field-major
  double* ge;             // E*4*NC element terms
  int E, N;
  ovs_params p;
};

// element terms per node, in the order of the output fields below
template <int KIND> struct VjpMap;
template <> struct VjpMap<OVS_ASM_NSVOF> { static constexpr int NC = 13; };   // x(3) u(3) p phi T a(3) phidot
template <> struct VjpMap<OVS_ASM_TEM> { static constexpr int NC = 9; };      // x(3) u(3) phi T Tdot
// output field (OVS_VJP_* order) and chain factor kind (0: 1, 1: alfi, 2: almi)
static const int h_vjp_out_nsvof[13] = {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12};
static const int h_vjp_fac_nsvof[13] = {0, 0, 0, 1, 1, 1, 0, 1, 1, 2, 2, 2, 2};
static const int h_vjp_out_tem[9] = {0, 1, 2, 3, 4, 5, 7, 8, 13};
static const int h_vjp_fac_tem[9] = {0, 0, 0, 1, 1, 1, 1, 1, 2};

// phase change at a point: mdot and its factor, as the residual routines take
// them; the adjoint of mdot goes to phic and T
struct PhasePoint {
  double phic, mdot, dm_dphi, dm_dT;
};
__device__ __forceinline__ PhasePoint phase_point(const ovs_params& p, double phid, double Ti) {
  PhasePoint q;
  q.phic = clamp01(phid);
  const double d = (Ti - p.ts) / p.ts;
  const bool hot = Ti > p.ts;
  const double c = hot ? p.c_evap * p.rhow : p.c_cond * p.rhoa;
  const double share = hot ? 1.0 - q.phic : q.phic;
  q.mdot = c * share * d;
  q.dm_dphi = (hot ? -c : c) * d;
  q.dm_dT = c * share / p.ts;
  return q;
}

// adjoint of the geometry: from gb (of the gradients), Gb (of G) and db (of
// DetJ) to the node coordinates, in the first three terms of each node
template <int NC>
__device__ __forceinline__ void vjp_geometry(const double (&g)[4][3], double detj, const double (&gb)[4][3],
                                             const double (&Gb)[3][3], double db, double* out) {
  double Bb[3][3], X[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      double t = gb[k][i] - gb[3][i];
#pragma unroll
      for (int j = 0; j < 3; ++j) t += (Gb[i][j] + Gb[j][i]) * g[k][j];
      Bb[k][i] = t;
    }
  // B = A^-1 (rows g_0..g_2): dB = -B dA B, d DetJ = DetJ tr(B dA)
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int l = 0; l < 3; ++l) X[k][l] = Bb[k][0] * g[l][0] + Bb[k][1] * g[l][1] + Bb[k][2] * g[l][2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double s3 = 0.0;
#pragma unroll
    for (int l = 0; l < 3; ++l) {
      const double ab = db * detj * g[l][i] - (g[0][i] * X[0][l] + g[1][i] * X[1][l] + g[2][i] * X[2][l]);
      out[l * NC + i] = ab;
      s3 -= ab;
    }
    out[3 * NC + i] = s3;
  }
}

__device__ void vjp_nsvof(const ovs_params& p, const double (&r)[4][16], const double (&vv)[4][5], double* out) {
  constexpr int NC = VjpMap<OVS_ASM_NSVOF>::NC;
  const ZeroRecs<double> lo;
  double g[4][3], G[3][3], detj, GG, trG;
  element_geometry<double>(r, lo, g, G, detj, GG, trG);
  const double w = detj * (0.25 / 6.0);
  double du[3][3], dp[3], dphi[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      du[i][j] = r[0][3 + i] * g[0][j] + r[1][3 + i] * g[1][j] + r[2][3 + i] * g[2][j] + r[3][3 + i] * g[3][j];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    dp[j] = r[0][12] * g[0][j] + r[1][12] * g[1][j] + r[2][12] * g[2][j] + r[3][12] * g[3][j];
    dphi[j] = r[0][13] * g[0][j] + r[1][13] * g[1][j] + r[2][13] * g[2][j] + r[3][13] * g[3][j];
  }
  const double divu = du[0][0] + du[1][1] + du[2][2];
  // cotangent contractions with the gradients
  double D[3][3], Q[3], R[3], hs[3], sn[4];
#pragma unroll
  for (int n = 0; n < 4; ++n) sn[n] = vv[n][0] + vv[n][1] + vv[n][2];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      D[i][j] = vv[0][i] * g[0][j] + vv[1][i] * g[1][j] + vv[2][i] * g[2][j] + vv[3][i] * g[3][j];
    Q[j] = vv[0][3] * g[0][j] + vv[1][3] * g[1][j] + vv[2][3] * g[2][j] + vv[3][3] * g[3][j];
    R[j] = vv[0][4] * g[0][j] + vv[1][4] * g[1][j] + vv[2][4] * g[2][j] + vv[3][4] * g[3][j];
    hs[j] = sn[0] * g[0][j] + sn[1] * g[1][j] + sn[2] * g[2][j] + sn[3] * g[3][j];
  }
  const double B = D[0][0] + D[1][1] + D[2][2];
  double SV = 0.0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) SV += hs[j] * (du[j][k] + du[k][j]);
  const double RdP = R[0] * dphi[0] + R[1] * dphi[1] + R[2] * dphi[2];
  const double irhoa = 1.0 / p.rhoa, ira = irhoa - 1.0 / p.rhow, itrG = 1.0 / trG, iGG = 1.0 / GG;
  const double isGG = sqrt(iGG), taut = 4.0 / (p.delt * p.delt);
  const bool kdc_on = fabs(p.ns_kdc_w) + fabs(p.ns_kdc_a) > 0.0, kdcphi_on = fabs(p.lsc_kdc) > 0.0;
  // adjoints gathered over the points
  double wb = 0.0, SVb = 0.0, GGb = 0.0, itrGb = 0.0, divb = 0.0;
  double dub[3][3], dpb[3], dfb[3], Db[3][3], Qb[3], Rb[3], Gb[3][3], nb[4][10];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    dpb[i] = dfb[i] = Qb[i] = Rb[i] = 0.0;
#pragma unroll
    for (int j = 0; j < 3; ++j) dub[i][j] = Db[i][j] = Gb[i][j] = 0.0;
  }
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int k = 0; k < 10; ++k) nb[n][k] = 0.0;
#pragma unroll 1
  for (int gp = 0; gp < 4; ++gp) {
    double N[4];
    tet_shape<double>(gp, N);
    auto at = [&](int k) { return r[0][k] * N[0] + r[1][k] * N[1] + r[2][k] * N[2] + r[3][k] * N[3]; };
    double uadv[3], a[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      uadv[d] = at(3 + d) - at(6 + d);
      a[d] = at(9 + d) - p.gravvec[d];
    }
    const double pri = at(12), phid = at(13), rphii = at(14), Ti = at(15);
    // the point's formulas, as nsvof_point
    const PhasePoint ph = phase_point(p, phid, Ti);
    const bool inside = !(phid < 0.0 || phid > 1.0), hot = Ti > p.ts;
    const double dmd_dT = !inside ? 0.0 : (hot ? -p.c_evap * p.rhow : p.c_cond * p.rhoa) / p.ts * p.c_dmdot;
    const double dmdi = dmd_dT * (Ti - p.ts) * ira;
    const double vdot = ph.mdot * ira;
    const double rho = p.rhow * (1.0 - ph.phic) + p.rhoa * ph.phic, mu = p.muw * (1.0 - ph.phic) + p.mua * ph.phic;
    const double lam = -2.0 / 3.0 * mu;
    double acc[3], rL[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      acc[i] = a[i] + du[i][0] * uadv[0] + du[i][1] * uadv[1] + du[i][2] * uadv[2];
      rL[i] = rho * acc[i] + dp[i];
    }
    const double res = rphii + (uadv[0] * dphi[0] + uadv[1] * dphi[1] + uadv[2] * dphi[2]) + phid * vdot - ph.mdot * irhoa;
    const double taua = quad_uGu<double>(uadv, G), irho = 1.0 / rho, nu = mu * irho;
    const double taud = nu * nu * 12.0 * GG, is = rsqrt(taut + taua + taud), tauM = irho * is;
    const double tauLS = rsqrt(taut + taua), sq = sqrt(taua + taud), tauC = rho * sq * itrG;
    double lw = 0.0, srr = 0.0;
    const double rr = rL[0] * rL[0] + rL[1] * rL[1] + rL[2] * rL[2];
    if (kdc_on) {
      lw = (double)low_word(p.ns_kdc_w * (1.0 - ph.phic) + p.ns_kdc_a * ph.phic);
      srr = sqrt(rr * iGG);
    }
    const double mupk = mu + lw * srr, kdphi = kdcphi_on ? p.lsc_kdc * fabs(res) * isGG : 0.0;
    const double Z = divu - vdot, F = pri - tauC * Z - lam * divu;
    double A[3], C[3], P = 0.0, V = 0.0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      A[i] = vv[0][i] * N[0] + vv[1][i] * N[1] + vv[2][i] * N[2] + vv[3][i] * N[3];
      C[i] = D[i][0] * uadv[0] + D[i][1] * uadv[1] + D[i][2] * uadv[2];
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) { P += vv[n][3] * N[n]; V += vv[n][4] * N[n]; }
    const double uR = uadv[0] * R[0] + uadv[1] * R[1] + uadv[2] * R[2];
    const double CrL = C[0] * rL[0] + C[1] * rL[1] + C[2] * rL[2], QrL = Q[0] * rL[0] + Q[1] * rL[1] + Q[2] * rL[2];
    wb += -rho * (A[0] * acc[0] + A[1] * acc[1] + A[2] * acc[2]) + B * F - mupk * SV - rho * tauM * CrL - P * Z -
          tauM * QrL - (V + tauLS * uR) * res - kdphi * RdP + V * dmdi * tauC * Z;
    // ---- backwards
    const double Fb = w * B;
    double rhob = -w * tauM * CrL, mub = -w * SV + 2.0 / 3.0 * Fb * divu, ub[3];
    SVb -= w * mupk;
    const double tMb = -w * (rho * CrL + QrL), Zb = w * (V * dmdi * tauC - P) - Fb * tauC;
    const double tCb = (w * V * dmdi - Fb) * Z;
    double resb = -w * (V + tauLS * uR);
    const double kdpb = -w * RdP;
    if (kdcphi_on) {
      resb += res > 0.0 ? kdpb * p.lsc_kdc * isGG : (res < 0.0 ? -kdpb * p.lsc_kdc * isGG : 0.0);
      GGb -= 0.5 * kdpb * kdphi * iGG;
    }
    const double kdcb = srr > 0.0 ? -w * SV * lw * 0.5 / srr : 0.0;   // of rr / GG
    GGb -= kdcb * rr * iGG * iGG;
    double tab = -0.5 * tauLS * tauLS * tauLS * (-w * uR * res);
    const double isb = tMb * irho, sumb = -0.5 * is * is * is * isb;
    double irhob = tMb * is;
    const double sqb = sq > 0.0 ? tCb * rho * itrG / (2.0 * sq) : 0.0;
    rhob += tCb * sq * itrG;
    itrGb += tCb * rho * sq;
    tab += sumb + sqb;
    const double tdb = sumb + sqb, nub = tdb * 24.0 * nu * GG;
    GGb += tdb * 12.0 * nu * nu;
    mub += nub * irho;
    irhob += nub * mu;
    rhob -= irhob * irho * irho;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Db[i][i] += w * F;
      const double Cb = -w * rho * tauM * rL[i];
      const double rLb = -w * tauM * (rho * C[i] + Q[i]) + 2.0 * rL[i] * kdcb * iGG;
      const double t1b = rLb - w * A[i];
      Qb[i] -= w * tauM * rL[i];
      dpb[i] += rLb;
      rhob += t1b * acc[i];
      const double ab = t1b * rho;   // of acceleration + convection
#pragma unroll
      for (int n = 0; n < 4; ++n) nb[n][6 + i] += N[n] * ab;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        Db[i][j] += Cb * uadv[j];
        dub[i][j] += ab * uadv[j];
        Gb[i][j] += tab * uadv[i] * uadv[j];
      }
      ub[i] = resb * dphi[i] - w * tauLS * res * R[i] + 2.0 * tab * (G[i][0] * uadv[0] + G[i][1] * uadv[1] + G[i][2] * uadv[2]);
      Rb[i] -= w * (tauLS * res * uadv[i] + kdphi * dphi[i]);
      dfb[i] += resb * uadv[i] - w * kdphi * R[i];
    }
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double Cb = -w * rho * tauM * rL[i];
        const double rLb = -w * tauM * (rho * C[i] + Q[i]) + 2.0 * rL[i] * kdcb * iGG;
        ub[j] += Cb * D[i][j] + (rLb - w * A[i]) * rho * du[i][j];
      }
    divb += Zb - Fb * lam;
    const double vb = -Zb + resb * phid, mb = vb * ira - resb * irhoa;
    double phicb = rhob * (p.rhoa - p.rhow) + mub * (p.mua - p.muw) + mb * ph.dm_dphi;
    const double Tb = mb * ph.dm_dT + w * V * tauC * Z * ira * dmd_dT;
    const double phib = resb * vdot + (inside ? phicb : 0.0);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
#pragma unroll
      for (int d = 0; d < 3; ++d) nb[n][d] += N[n] * ub[d];
      nb[n][3] += N[n] * Fb;
      nb[n][4] += N[n] * phib;
      nb[n][5] += N[n] * Tb;
      nb[n][9] += N[n] * resb;
    }
  }
  // ---- gradients and geometry
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    dub[i][i] += divb;
#pragma unroll
    for (int j = 0; j < 3; ++j) dub[i][j] += SVb * (hs[i] + hs[j]);
  }
  GGb *= 2.0;
  const double trb = -itrGb * itrG * itrG;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Gb[i][i] += trb;
#pragma unroll
    for (int j = 0; j < 3; ++j) Gb[i][j] += GGb * G[i][j];
  }
  double gb[4][3];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      double t = vv[n][3] * Qb[j] + vv[n][4] * Rb[j] + r[n][12] * dpb[j] + r[n][13] * dfb[j];
      double hb = 0.0;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        t += vv[n][i] * Db[i][j] + r[n][3 + i] * dub[i][j];
        hb += du[j][i] + du[i][j];
      }
      gb[n][j] = t + sn[n] * SVb * hb;
    }
    double* o = out + n * NC;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      o[3 + i] = nb[n][i] + dub[i][0] * g[n][0] + dub[i][1] * g[n][1] + dub[i][2] * g[n][2];
      o[9 + i] = nb[n][6 + i];
    }
    o[6] = nb[n][3] + dpb[0] * g[n][0] + dpb[1] * g[n][1] + dpb[2] * g[n][2];
    o[7] = nb[n][4] + dfb[0] * g[n][0] + dfb[1] * g[n][1] + dfb[2] * g[n][2];
    o[8] = nb[n][5];
    o[12] = nb[n][9];
  }
  vjp_geometry<NC>(g, detj, gb, Gb, wb * (0.25 / 6.0), out);
}

// record layout of the temperature pass: xd(0:2) u(3:5) um(6:8) phi(9) T(10) rT(11)
__device__ void vjp_tem(const ovs_params& p, const double (&r)[4][16], const double (&vv)[4][1], bool fluid,
                        double* out) {
  constexpr int NC = VjpMap<OVS_ASM_TEM>::NC;
  const ZeroRecs<double> lo;
  double g[4][3], G[3][3], detj, GG, trG;
  element_geometry<double>(r, lo, g, G, detj, GG, trG);
  const double w = detj * (0.25 / 6.0);
  double dT[3], R[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    dT[j] = r[0][10] * g[0][j] + r[1][10] * g[1][j] + r[2][10] * g[2][j] + r[3][10] * g[3][j];
    R[j] = vv[0][0] * g[0][j] + vv[1][0] * g[1][j] + vv[2][0] * g[2][j] + vv[3][0] * g[3][j];
  }
  const double RdT = R[0] * dT[0] + R[1] * dT[1] + R[2] * dT[2];
  const double iGG = 1.0 / GG, isGG = sqrt(iGG), taut = 4.0 / (p.delt * p.delt), dcp = p.cpw - p.cpa;
  const double tk = fabs(p.tem_kdc) > 0.0 ? p.tem_kdc / p.tref : 0.0;
  double wb = 0.0, GGb = 0.0, dTb[3] = {0, 0, 0}, Rb[3] = {0, 0, 0}, Gb[3][3], nb[4][6];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Gb[i][j] = 0.0;
#pragma unroll
  for (int n = 0; n < 4; ++n)
#pragma unroll
    for (int k = 0; k < 6; ++k) nb[n][k] = 0.0;
#pragma unroll 1
  for (int gp = 0; gp < 4; ++gp) {
    double N[4];
    tet_shape<double>(gp, N);
    auto at = [&](int k) { return r[0][k] * N[0] + r[1][k] * N[1] + r[2][k] * N[2] + r[3][k] * N[3]; };
    const double phid = at(9), Ti = at(10), rTi = at(11);
    double V = 0.0;
#pragma unroll
    for (int n = 0; n < 4; ++n) V += vv[n][0] * N[n];
    double ub[3] = {0, 0, 0}, phib = 0.0, Tb = 0.0, rTb;
    if (fluid) {
      const double uadv[3] = {at(3) - at(6), at(4) - at(7), at(5) - at(8)};
      const PhasePoint ph = phase_point(p, phid, Ti);
      const double rho = p.rhow * (1.0 - ph.phic) + p.rhoa * ph.phic, cp = p.cpw * (1.0 - ph.phic) + p.cpa * ph.phic;
      const double hk = p.kappaw * (1.0 - ph.phic) + p.kappaa * ph.phic;
      const double rcp = (p.rhow * p.cpw) * (1.0 - ph.phic) + (p.rhoa * p.cpa) * ph.phic;
      const double lat = dcp * (Ti - p.ts) - p.lh, udT = uadv[0] * dT[0] + uadv[1] * dT[1] + uadv[2] * dT[2];
      const double res = rcp * (rTi + udT) - lat * ph.mdot, taua = quad_uGu<double>(uadv, G);
      const double ircp = 1.0 / (rho * cp), kk = hk * ircp, is = rsqrt(taua + taut + kk * kk * 12.0 * GG), tauT = ircp * is;
      const double hkd = hk + tk * fabs(res) * isGG;
      const double uR = uadv[0] * R[0] + uadv[1] * R[1] + uadv[2] * R[2];
      wb += -(V + rcp * tauT * uR) * res - hkd * RdT;
      // ---- backwards
      const double hkb = -w * RdT;
      double resb = -w * (V + rcp * tauT * uR);
      resb += res > 0.0 ? hkb * tk * isGG : (res < 0.0 ? -hkb * tk * isGG : 0.0);
      GGb -= 0.5 * hkb * tk * fabs(res) * isGG * iGG;
      const double rcpb = -w * tauT * uR * res + resb * (rTi + udT);
      const double tTb = -w * rcp * uR * res, sumb = -0.5 * is * is * is * tTb * ircp;
      const double kkb = sumb * 24.0 * kk * GG, ircpb = tTb * is + kkb * hk;
      GGb += sumb * 12.0 * kk * kk;
      const double pb = -ircpb * ircp * ircp;   // of rho cp
      const double mb = -resb * lat;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        ub[i] = -w * rcp * tauT * res * R[i] + resb * rcp * dT[i] +
                2.0 * sumb * (G[i][0] * uadv[0] + G[i][1] * uadv[1] + G[i][2] * uadv[2]);
        Rb[i] -= w * (rcp * tauT * res * uadv[i] + hkd * dT[i]);
        dTb[i] += resb * rcp * uadv[i] - w * hkd * R[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) Gb[i][j] += sumb * uadv[i] * uadv[j];
      }
      const double phicb = pb * (cp * (p.rhoa - p.rhow) + rho * (p.cpa - p.cpw)) + (hkb + kkb * ircp) * (p.kappaa - p.kappaw) +
                           rcpb * (p.rhoa * p.cpa - p.rhow * p.cpw) + mb * ph.dm_dphi;
      phib = phid < 0.0 || phid > 1.0 ? 0.0 : phicb;
      Tb = -resb * dcp * ph.mdot + mb * ph.dm_dT;
      rTb = resb * rcp;
    } else {
      const double rcp = p.rhos * p.cps;
      wb += -V * rcp * rTi - p.kappas * RdT;
      rTb = -w * V * rcp;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        Rb[i] -= w * p.kappas * dT[i];
        dTb[i] -= w * p.kappas * R[i];
      }
    }
#pragma unroll
    for (int n = 0; n < 4; ++n) {
#pragma unroll
      for (int d = 0; d < 3; ++d) nb[n][d] += N[n] * ub[d];
      nb[n][3] += N[n] * phib;
      nb[n][4] += N[n] * Tb;
      nb[n][5] += N[n] * rTb;
    }
  }
  double gb[4][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) Gb[i][j] += 2.0 * GGb * G[i][j];
#pragma unroll
  for (int n = 0; n < 4; ++n) {
#pragma unroll
    for (int j = 0; j < 3; ++j) gb[n][j] = vv[n][0] * Rb[j] + r[n][10] * dTb[j];
    double* o = out + n * NC;
#pragma unroll
    for (int i = 0; i < 3; ++i) o[3 + i] = nb[n][i];
    o[6] = nb[n][3];
    o[7] = nb[n][4] + dTb[0] * g[n][0] + dTb[1] * g[n][1] + dTb[2] * g[n][2];
    o[8] = nb[n][5];
  }
  vjp_geometry<NC>(g, detj, gb, Gb, wb * (0.25 / 6.0), out);
}

template <int KIND>
__global__ void __launch_bounds__(128) residual_vjp_kernel(const VjpArgs a) {
  constexpr int NF = Lay<KIND>::NF, NC = VjpMap<KIND>::NC;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.E) return;
  const int4 nd = __ldg(reinterpret_cast<const int4*>(a.ien) + e);
  const int nodes[4] = {nd.x, nd.y, nd.z, nd.w};
  const bool fluid = __ldg(a.elm_id + e) == a.p.fluid_elm_id;
  double* out = a.ge + (size_t)e * 4 * NC;
  if (KIND == OVS_ASM_NSVOF && !fluid) {   // solid elements contribute nothing
    for (int q = 0; q < 4 * NC; ++q) out[q] = 0.0;
    return;
  }
  double r[4][16], lo[4][4], vv[4][NF];
#pragma unroll
  for (int n = 0; n < 4; ++n) load_rec(a.rec, nodes[n], r[n], lo[n]);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const unsigned ib = __ldg(a.ibc + nodes[m]);
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      const unsigned bit = KIND == OVS_ASM_TEM ? TB : (f < 3 ? (1u << f) : (f == 3 ? PB : FB));
      vv[m][f] = (ib & bit) ? 0.0 : a.cot[(size_t)f * a.N + nodes[m]];
    }
  }
  if constexpr (KIND == OVS_ASM_NSVOF) vjp_nsvof(a.p, r, vv, out);
  else vjp_tem(a.p, r, vv, fluid, out);
}

struct VjpGatherArgs {
  const int* n2e_ptr;
  const int* n2e;
  const double* ge;
  double* grad;           // OVS_VJP_COUNT*N field-major
  int N, NC;
  int q[OVS_VJP_COUNT];   // the element term of an output field, -1: zero
  double fac[OVS_VJP_COUNT];
};

// 16 lanes per node, lane q adds term q of the node's elements in ascending
// order; the block's 16 nodes leave field by field (128 contiguous bytes)
__global__ void __launch_bounds__(256) vjp_gather_kernel(const VjpGatherArgs a) {
  __shared__ double sm[16][17];
  const int q = threadIdx.x & 15, nl = threadIdx.x >> 4, A = blockIdx.x * 16 + nl;
  double s = 0.0;
  if (A < a.N && q < a.NC) {
    const int k1 = __ldg(a.n2e_ptr + A + 1);
#pragma unroll 4
    for (int k = __ldg(a.n2e_ptr + A); k < k1; ++k) {
      const int packed = __ldg(a.n2e + k);
      s += __ldg(a.ge + ((size_t)(packed >> 3) * 4 + (packed & 7)) * a.NC + q);
    }
  }
  sm[q][nl] = s;
  __syncthreads();
  const int f = nl, B = blockIdx.x * 16 + q;   // field, node
  if (f < OVS_VJP_COUNT && B < a.N)
    a.grad[(size_t)f * a.N + B] = a.q[f] < 0 ? 0.0 : a.fac[f] * sm[a.q[f]][q];
}
static_assert(OVS_VJP_COUNT <= 16, "one lane group per output field");

#include "assemble_hex.cuh"

}  // namespace

// W = f_g (x) f_g of the hex tensor-core pass, split into TF32 hi + lo, in
// the canonical K-major no-swizzle layout: row n = 8 a + b, k = 16 g + 4 r + s,
// byte offset (k / 4) * 1024 + (n / 8) * 128 + (n % 8) * 16 + (k % 4) * 4.
static float host_tf32(double x) {   // round to the nearest TF32, ties away (cvt.rna)
  float f = (float)x;
  uint32_t b;
  memcpy(&b, &f, 4);
  b = (b + 0x1000u) & 0xFFFFE000u;
  memcpy(&f, &b, 4);
  return f;
}

int hex_tc_prepare(ovs_ctx* c) {
  int st;
  if ((st = ovs_ensure(&c->hex_kbuf, sizeof(float) * (size_t)c->E * 64 * 24))) return st;
  if (c->hex_w) return OVS_OK;
  static const int sgn[8][3] = {{-1, 1, -1}, {1, 1, -1}, {1, 1, 1}, {-1, 1, 1},
                                {-1, -1, -1}, {1, -1, -1}, {1, -1, 1}, {-1, -1, 1}};
  const double q = 0.57735026918963;   // the 2x2x2 points of hex_gp
  double f[8][4][8];
  for (int g = 0; g < 8; ++g) {
    const double xi = (g & 1) ? q : -q, eta = (g & 2) ? q : -q, ze = (g & 4) ? q : -q;
    for (int a = 0; a < 8; ++a) {
      const double sx = sgn[a][0], sy = sgn[a][1], sz = sgn[a][2];
      f[g][0][a] = (1.0 + sx * xi) * (1.0 + sy * eta) * (1.0 + sz * ze) * 0.125;
      f[g][1][a] = sx * (1.0 + sy * eta) * (1.0 + sz * ze) * 0.125;
      f[g][2][a] = sy * (1.0 + sx * xi) * (1.0 + sz * ze) * 0.125;
      f[g][3][a] = sz * (1.0 + sx * xi) * (1.0 + sy * eta) * 0.125;
    }
  }
  std::vector<float> hw(2 * 8192, 0.f);
  for (int n = 0; n < 64; ++n)
    for (int k = 0; k < 128; ++k) {
      const int a = n >> 3, b = n & 7, g = k >> 4, r = (k >> 2) & 3, s = k & 3;
      const double v = f[g][r][a] * f[g][s][b];
      const float hi = host_tf32(v), lo = host_tf32(v - (double)hi);
      const size_t off = ((size_t)(k >> 2) * 1024 + (n >> 3) * 128 + (n & 7) * 16 + (k & 3) * 4) / 4;
      hw[off] = hi;
      hw[8192 + off] = lo;
    }
  if ((st = ovs_ensure((void**)&c->hex_w, sizeof(float) * 2 * 8192))) return st;
  OVS_CUDA_TRY(cudaMemcpyAsync(c->hex_w, hw.data(), sizeof(float) * 2 * 8192, cudaMemcpyHostToDevice, c->stream));
  OVS_CUDA_TRY(cudaStreamSynchronize(c->stream));
  return OVS_OK;
}

static int dispatch_assemble(ovs_ctx* c, int kernel, int prec, const AsmArgs& a, const SumArgs& sa,
                             int parts = 3) {
  if (c->nshl == 8) {   // trilinear hexahedra: NS+VOF and temperature passes
    if (kernel == OVS_ASM_NS) return OVS_ERR_ARG;
    if (prec == OVS_FP64)
      return kernel == OVS_ASM_NSVOF ? launch_assemble_hex<double, OVS_ASM_NSVOF>(c, a, sa, parts)
                                     : launch_assemble_hex<double, OVS_ASM_TEM>(c, a, sa, parts);
    return kernel == OVS_ASM_NSVOF ? launch_assemble_hex<float, OVS_ASM_NSVOF>(c, a, sa, parts)
                                   : launch_assemble_hex<float, OVS_ASM_TEM>(c, a, sa, parts);
  }
  if (prec == OVS_FP64) {
    if (kernel == OVS_ASM_NS) return launch_assemble<double, OVS_ASM_NS>(c, a, sa, parts);
    if (kernel == OVS_ASM_NSVOF) return launch_assemble<double, OVS_ASM_NSVOF>(c, a, sa, parts);
    return launch_assemble<double, OVS_ASM_TEM>(c, a, sa, parts);
  }
  if (kernel == OVS_ASM_NS) return launch_assemble<float, OVS_ASM_NS>(c, a, sa, parts);
  if (kernel == OVS_ASM_NSVOF) return launch_assemble<float, OVS_ASM_NSVOF>(c, a, sa, parts);
  return launch_assemble<float, OVS_ASM_TEM>(c, a, sa, parts);
}

static void fill_args(ovs_ctx* c, int prec, SysStore& S, int tensor_flag, AsmArgs& a, SumArgs& sa) {
  sa.rec = c->rec[prec];
  sa.ien = c->ien_t;
  sa.elm_id = c->elm_t;
  sa.sum = c->esum[prec];
  sa.flags = c->flags;
  sa.cfl_bits = c->cfl_bits;
  sa.E = c->E;
  sa.p = c->params;
  a.rec = c->esum[prec];     // pass 2 reads the summaries
  a.ibc = c->ibc;
  a.rowptr = c->rowptr;
  a.colidx = c->colidx;
  a.n2e_ptr = c->n2e_ptr;
  a.n2e = c->n2e_t;
  a.vals = S.vals;
  a.rhs = S.rhs;
  a.flags = c->flags;
  a.N = c->N;
  a.mat = (tensor_flag & OVS_TENSOR_MAT) != 0;
  a.vec = (tensor_flag & OVS_TENSOR_VEC) != 0;
  a.n2s = c->n2s;
  a.row_rec = c->row_rec;
  a.edge_rec = c->edge_rec;
  a.edge_ptr = c->edge_ptr;
  a.edge_list = c->edge_list;
  a.tile_edge = c->tile_edge;
  a.max_deg = c->max_deg;
  a.p = c->params;
  a.kbuf = nullptr;
}

// parts: 3 both passes, 1 the element pass, 2 the row pass (on the summaries
// of the warm-up run)
int ovs_profile_assemble(ovs_ctx* c, int kernel, int prec, int reps, double* ms, int parts) {
  if (kernel != OVS_ASM_NS && kernel != OVS_ASM_NSVOF && kernel != OVS_ASM_TEM) return OVS_ERR_ARG;
  const int sys = kernel == OVS_ASM_NS ? OVS_SYS_NS : (kernel == OVS_ASM_NSVOF ? OVS_SYS_NSVOF : OVS_SYS_TEM);
  SysStore& S = c->sys[sys][prec];
  if (!S.vals || !S.rhs || !c->rec[prec] || !c->esum[prec]) return OVS_ERR_STATE;
  AsmArgs a;
  SumArgs sa;
  fill_args(c, prec, S, OVS_TENSOR_MAT | OVS_TENSOR_VEC, a, sa);
  int st;
  if ((st = dispatch_assemble(c, kernel, prec, a, sa))) return st;  // warm
  OVS_CUDA_TRY(cudaEventRecord(c->ev0, c->stream));
  for (int r = 0; r < reps; ++r)
    if ((st = dispatch_assemble(c, kernel, prec, a, sa, parts))) return st;
  OVS_CUDA_TRY(cudaEventRecord(c->ev1, c->stream));
  OVS_CUDA_TRY(cudaEventSynchronize(c->ev1));
  float t = 0.f;
  OVS_CUDA_TRY(cudaEventElapsedTime(&t, c->ev0, c->ev1));
  *ms = (double)t / reps;
  return OVS_OK;
}

// the assembly status of the pass (flags and CFL number) to the host, or to
// the page-locked slots of ovs_assemble_async
static int finish_status(ovs_ctx* c, double* cfl) {
  cudaStream_t s = c->stream;
  if (c->defer_status) {   // ovs_assemble_async: the status travels to a page-locked slot, read at the wait
    const int k = c->async_n++;
    OVS_CUDA_TRY(cudaMemcpyAsync(c->h_async_flags + 4 * k, c->flags, sizeof(int) * 4, cudaMemcpyDeviceToHost, s));
    OVS_CUDA_TRY(cudaMemcpyAsync(c->h_async_cfl + k, c->cfl_bits, sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                 s));
    return OVS_OK;
  }
  int hflags[4];
  unsigned long long hcfl = 0;
  OVS_CUDA_TRY(cudaMemcpyAsync(hflags, c->flags, sizeof(hflags), cudaMemcpyDeviceToHost, s));
  OVS_CUDA_TRY(cudaMemcpyAsync(&hcfl, c->cfl_bits, sizeof(hcfl), cudaMemcpyDeviceToHost, s));
  OVS_CUDA_TRY(cudaStreamSynchronize(s));
  if (cfl) {
    double v;
    memcpy(&v, &hcfl, sizeof(v));
    *cfl = v;
  }
  if (hflags[3]) return OVS_ERR_PATTERN;
  if (hflags[2]) return OVS_ERR_TIMEOUT;
  if (hflags[1]) return OVS_ERR_NONFINITE;
  if (hflags[0]) return OVS_WARN_NEG_DETJ;
  return OVS_OK;
}

// alpha-stage records of a pass (the record layout of the NS+VOF or the
// temperature routine)
static int alpha_stage(ovs_ctx* c, int prec, bool tem) {
  AlphaArgs aa;
  for (int f = 0; f < OVS_F_COUNT; ++f) aa.f[f] = c->field[f];
  aa.xg = c->field[OVS_F_XG];
  aa.rec = c->rec[prec];
  aa.N = c->N;
  aa.tem = tem;
  aa.almi = c->params.almi;
  aa.alfi = c->params.alfi;
  if (prec == OVS_FP64) alpha_records_kernel<double><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, c->stream>>>(aa);
  else alpha_records_kernel<float><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, c->stream>>>(aa);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  return OVS_OK;
}

// one pass of `kernel` (alpha stage, element pass, row pass, faces) with its
// flags and CFL number accumulated on the device (cleared by the caller)
static int assemble_pass(ovs_ctx* c, int kernel, int tensor_flag, int prec) {
  const int sys = kernel == OVS_ASM_NS ? OVS_SYS_NS : (kernel == OVS_ASM_NSVOF ? OVS_SYS_NSVOF : OVS_SYS_TEM);
  const size_t ts = prec == OVS_FP64 ? 8 : 4;
  SysStore& S = c->sys[sys][prec];
  int st;
  if ((st = ovs_ensure(&S.vals, ts * (size_t)c->nnz * ovs_sys_nv(sys)))) return st;
  if ((st = ovs_ensure(&S.rhs, ts * (size_t)c->N * ovs_sys_nf(sys)))) return st;
  if ((st = ovs_ensure(&c->rec[prec], ts * (size_t)c->N * REC))) return st;
  const size_t sw = c->nshl == 8 ? (size_t)HexLay<OVS_ASM_NSVOF>::SW : (size_t)Lay<OVS_ASM_NSVOF>::SW;
  if ((st = ovs_ensure(&c->esum[prec], ts * (size_t)c->E * sw))) return st;
  if ((st = alpha_stage(c, prec, kernel == OVS_ASM_TEM))) return st;
  AsmArgs a;
  SumArgs sa;
  fill_args(c, prec, S, tensor_flag, a, sa);
  if ((st = dispatch_assemble(c, kernel, prec, a, sa))) return st;
  if ((st = ovs_faces_assemble(c, kernel, prec, a.mat, a.vec))) return st;
  if (a.mat) S.have_mat = true;
  if (a.vec) S.have_rhs = true;
  return OVS_OK;
}

int ovs_assemble_impl(ovs_ctx* c, int kernel, int tensor_flag, int prec, double* cfl) {
  if (!c->have_pattern || !c->have_params) return OVS_ERR_STATE;
  if (c->nshl != 4 && c->nshl != 8) return OVS_ERR_ARG;
  if (kernel == OVS_ASM_QUENCH) {   // the NS+VOF pass, then the temperature pass; one status
    if (prec != OVS_FP64 && prec != OVS_FP32) return OVS_ERR_ARG;
    int st;
    OVS_CUDA_TRY(cudaMemsetAsync(c->flags, 0, sizeof(int) * 4, c->stream));
    OVS_CUDA_TRY(cudaMemsetAsync(c->cfl_bits, 0, sizeof(unsigned long long), c->stream));
    if ((st = assemble_pass(c, OVS_ASM_NSVOF, tensor_flag, prec))) return st;
    if ((st = assemble_pass(c, OVS_ASM_TEM, tensor_flag, prec))) return st;
    return finish_status(c, cfl);
  }
  if (c->nshl == 8 && kernel == OVS_ASM_NS) return OVS_ERR_ARG;
  if (kernel != OVS_ASM_NS && kernel != OVS_ASM_NSVOF && kernel != OVS_ASM_TEM) return OVS_ERR_ARG;
  if (prec != OVS_FP64 && prec != OVS_FP32) return OVS_ERR_ARG;
  int st;
  OVS_CUDA_TRY(cudaMemsetAsync(c->flags, 0, sizeof(int) * 4, c->stream));
  OVS_CUDA_TRY(cudaMemsetAsync(c->cfl_bits, 0, sizeof(unsigned long long), c->stream));
  if ((st = assemble_pass(c, kernel, tensor_flag, prec))) return st;
  return finish_status(c, cfl);
}

int ovs_residual_vjp_impl(ovs_ctx* c, int kernel, const double* cot_host, double* grad_host) {
  if (!c->have_pattern || !c->have_params) return OVS_ERR_STATE;
  if (c->nshl != 4) return OVS_ERR_ARG;   // the adjoint covers the tet routines
  if (c->face_flags_all) return OVS_ERR_STATE;   // face terms are not differentiated
  if (kernel != OVS_ASM_NSVOF && kernel != OVS_ASM_TEM) return OVS_ERR_ARG;
  if (!cot_host || !grad_host) return OVS_ERR_ARG;
  const int tem = kernel == OVS_ASM_TEM;
  const int nf = tem ? 1 : 5, NC = tem ? VjpMap<OVS_ASM_TEM>::NC : VjpMap<OVS_ASM_NSVOF>::NC;
  const size_t N = c->N, E = c->E;
  int st;
  if ((st = ovs_ensure(&c->rec[OVS_FP64], sizeof(double) * N * REC))) return st;
  if ((st = ovs_ensure((void**)&c->vjp_cot, sizeof(double) * N * 5))) return st;
  if ((st = ovs_ensure((void**)&c->vjp_ge, sizeof(double) * E * 4 * 13))) return st;
  if ((st = ovs_ensure((void**)&c->vjp_grad, sizeof(double) * N * OVS_VJP_COUNT))) return st;
  cudaStream_t s = c->stream;
  AlphaArgs aa;
  for (int f = 0; f < OVS_F_COUNT; ++f) aa.f[f] = c->field[f];
  aa.xg = c->field[OVS_F_XG];
  aa.rec = c->rec[OVS_FP64];
  aa.N = c->N;
  aa.tem = tem;
  aa.almi = c->params.almi;
  aa.alfi = c->params.alfi;
  alpha_records_kernel<double><<<ovs_grid(c->N, 256, 1 << 30), 256, 0, s>>>(aa);
  ++c->launches;
  OVS_CUDA_TRY(cudaMemcpyAsync(c->vjp_cot, cot_host, sizeof(double) * N * nf, cudaMemcpyHostToDevice, s));
  VjpArgs va;
  va.rec = reinterpret_cast<const double*>(c->rec[OVS_FP64]);
  va.ien = c->ien;
  va.elm_id = c->elm_id;
  va.ibc = c->ibc;
  va.cot = c->vjp_cot;
  va.ge = c->vjp_ge;
  va.E = c->E;
  va.N = c->N;
  va.p = c->params;
  const int eb = (int)((E + 127) / 128);
  if (tem) residual_vjp_kernel<OVS_ASM_TEM><<<eb, 128, 0, s>>>(va);
  else residual_vjp_kernel<OVS_ASM_NSVOF><<<eb, 128, 0, s>>>(va);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  VjpGatherArgs ga;
  ga.n2e_ptr = c->n2e_ptr;
  ga.n2e = c->n2e;
  ga.ge = c->vjp_ge;
  ga.grad = c->vjp_grad;
  ga.N = c->N;
  ga.NC = NC;
  for (int f = 0; f < OVS_VJP_COUNT; ++f) { ga.q[f] = -1; ga.fac[f] = 0.0; }
  for (int q = 0; q < NC; ++q) {
    const int f = tem ? h_vjp_out_tem[q] : h_vjp_out_nsvof[q], fk = tem ? h_vjp_fac_tem[q] : h_vjp_fac_nsvof[q];
    ga.q[f] = q;
    ga.fac[f] = fk == 0 ? 1.0 : (fk == 1 ? c->params.alfi : c->params.almi);
  }
  vjp_gather_kernel<<<(c->N + 15) / 16, 256, 0, s>>>(ga);
  ++c->launches;
  OVS_CUDA_TRY(cudaGetLastError());
  OVS_CUDA_TRY(cudaMemcpyAsync(grad_host, c->vjp_grad, sizeof(double) * N * OVS_VJP_COUNT, cudaMemcpyDeviceToHost, s));
  OVS_CUDA_TRY(cudaStreamSynchronize(s));
  return OVS_OK;
}
