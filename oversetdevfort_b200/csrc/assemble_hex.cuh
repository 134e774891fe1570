// Trilinear hexahedra (nshl = 8): the NS+VOF quench and temperature
// element routines (src/solveQuenching.f90:122-882) with the 2x2x2 rule
// (src/genGP_GW.f90:355-389) and linhexshl (src/eval_shape_FEM.f90:148-196),
// assembled like the tets: an element pass writes per-Gauss-point records (T:
// the element matrix) and the element's residual rows, a row pass (one warp per
// CSR row) forms the blocks of A's row and adds them in ascending element id.
// Unlike a linear tet, a hex has different gradients at every Gauss point, so
// the row pass sums each block over the 8 points.  Included into assemble.cu's
// anonymous namespace (it uses its helpers).

// Node signs of linhexshl, N_a = (1 + sx xi)(1 + sy eta)(1 + sz zeta) / 8: bit
// set where the node sits at +1 along axis d.  The points are at +-q, so every
// shape value and derivative is one of a few constants, picked by how many of
// the node's signs match the point's.
__host__ __device__ constexpr int hex_bit(int a, int d) {
  return d == 0 ? ((a ^ (a >> 1)) & 1) : (d == 1 ? (a < 4) : ((a >> 1) & 1));
}
constexpr double HEX_P = 1.0 + 0.57735026918963, HEX_M = 1.0 - 0.57735026918963;   // 2x2x2 points (genGPandGW, weights 1)
template <typename T> __device__ __forceinline__ T hex_n3(int m) {   // N by matching signs
  constexpr double c0 = HEX_M * HEX_M * HEX_M * 0.125, c1 = HEX_P * HEX_M * HEX_M * 0.125,
                   c2 = HEX_P * HEX_P * HEX_M * 0.125, c3 = HEX_P * HEX_P * HEX_P * 0.125;
  return m == 0 ? (T)c0 : (m == 1 ? (T)c1 : (m == 2 ? (T)c2 : (T)c3));
}
template <typename T> __device__ __forceinline__ T hex_n2(int m) {   // |dN/dxi| by matching signs of the other two axes
  constexpr double c0 = HEX_M * HEX_M * 0.125, c1 = HEX_P * HEX_M * 0.125, c2 = HEX_P * HEX_P * 0.125;
  return m == 0 ? (T)c0 : (m == 1 ? (T)c1 : (T)c2);
}
template <typename T>
__device__ __forceinline__ T hex_N(int g, int a) {
  return hex_n3<T>((hex_bit(a, 0) == (g & 1)) + (hex_bit(a, 1) == ((g >> 1) & 1)) + (hex_bit(a, 2) == ((g >> 2) & 1)));
}

template <int KIND> struct HexLay;
//   NS+VOF record per point, with c_n = uadv . grad N_n: (grad N_n, c_n) of the
//   8 nodes, then the factors of the block formulas (hex_point): w rho, rt, w,
//   w tauLS | fact2 w, fact2 w rt, w rt, fact2 src | KA KB MM KDP |
//   dphi(3) ufac | eps plfac pad(2); then the residual rows 8x5
template <> struct HexLay<OVS_ASM_NSVOF> {
  static constexpr int GPW = 52, RHS0 = 8 * 52, NF = 5, SW = 8 * 52 + 40, NV = 24;
};
//   T: the 8x8 element matrix itself, row-major (a scalar system: smaller than
//   the records it would be summed from), then 8 residuals
template <> struct HexLay<OVS_ASM_TEM> {
  static constexpr int RHS0 = 64, NF = 1, SW = 72, NV = 1;
};

//   NS+VOF record per point for the tensor-core path: dxi/dx (3x3, row k =
//   xi_k) w KA KB MM KDP dphi(3) v(3) = dxi/dx uadv, rho rt tauLS src eps
//   ufac plfac pad; then the residual rows 8x5
struct HexTcLay {
  static constexpr int GPW = 28, RHS0 = 8 * 28, SW = 8 * 28 + 40;
};

__device__ __forceinline__ void lds4(const float* p, float* d) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
}
__device__ __forceinline__ void lds4(const double* p, double* d) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
}

// Element pass: 8 lanes per element, lane g evaluates Gauss point g.  A lane
// walks the element's 8 node records once (the 8 lanes read the same address)
// and keeps the sums it needs: values at the point and derivatives along the
// reference axes, which the inverse Jacobian then turns into gradients.  The
// residual rows are added over the lanes by halving, which leaves lane n with
// node n's.  NS+VOF: every lane writes its point's record (MAT) or the compact
// one of the tensor-core pass (TC).  T: the points meet in shared memory and
// lane a sums row a of the element matrix.  MAT false (vector-only pass): the
// residual rows alone.
// One thread per element held 8 records and 40 residual sums (255 registers,
// 1.4 KB of spills in FP64): 96^3 hexahedra, NS+VOF 1.78 -> 1.20 ms in FP64 and
// 0.82 -> 0.80 in FP32, T, which wrote point records for the row pass to sum,
// 1.47 -> 1.09 and 1.12 -> 0.55 ms (T rows 3.08 -> 0.59 and 2.39 -> 0.54 ms).
// Blocks per SM: 3 in FP64 (2: 1.48 ms, no spills), 6 in FP32 (4: 0.97, 5: 0.84).
template <typename T> struct HexTemStage {
  static constexpr int GPW = 44;                                       // per point: (grad, B) of 8 nodes, A of 8, HK
  static constexpr int ES = 8 * GPW + (sizeof(T) == 8 ? 2 : 4);        // element stride: elements of a warp spread over the banks
  static constexpr int bytes = 16 * ES * (int)sizeof(T);
};

// values summed over the 8 lanes of an element by halving: v holds NV values
// per node, lane n ends up with node n's in v[0..NV)
template <typename T, int NV>
__device__ __forceinline__ void hex_sum_nodes(T (&v)[8 * NV], int lane) {
#pragma unroll
  for (int half = 4, off = 4; off >= 1; half >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int k = 0; k < half * NV; ++k) {
      const T send = up ? v[k] : v[k + half * NV], keep = up ? v[k + half * NV] : v[k];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
}

template <typename T, int KIND, bool TC = false, bool MAT = true>
__global__ void __launch_bounds__(128, (sizeof(T) == 8 ? 3 : 6)) hex_element_kernel(const SumArgs a) {
  constexpr bool vof = KIND == OVS_ASM_NSVOF;
  using L = HexLay<KIND>;
  constexpr int NF = L::NF;
  constexpr int SW = !MAT ? 8 * NF : TC ? HexTcLay::SW : L::SW;
  constexpr int RHS0 = !MAT ? 0 : TC ? HexTcLay::RHS0 : L::RHS0;
  const ovs_params& p = a.p;
  const int lane = threadIdx.x & 31, gp = lane & 7;
  const int tt = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 3);
  const bool on = tt < a.E;
  const int t = on ? tt : a.E - 1;
  const T* rec = reinterpret_cast<const T*>(a.rec);
  const int mynode = __ldg(a.ien + 8 * (size_t)t + gp);
  const bool fluid = __ldg(a.elm_id + t) == p.fluid_elm_id;
  const int g0 = gp & 1, g1 = (gp >> 1) & 1, g2 = (gp >> 2) & 1;
  // shape values and reference derivatives of node n at this lane's point
  auto shape = [&](int n, T& N, T (&dN)[3]) {
    const int m0 = hex_bit(n, 0) == g0, m1 = hex_bit(n, 1) == g1, m2 = hex_bit(n, 2) == g2;
    N = hex_n3<T>(m0 + m1 + m2);
    const T d0 = hex_n2<T>(m1 + m2), d1 = hex_n2<T>(m0 + m2), d2 = hex_n2<T>(m0 + m1);
    dN[0] = hex_bit(n, 0) ? d0 : -d0;
    dN[1] = hex_bit(n, 1) ? d1 : -d1;
    dN[2] = hex_bit(n, 2) ? d2 : -d2;
  };
  T J[3][3], ur[3][3], pr[3], fr[3];   // T pass: fr holds the temperature's derivatives, ur and pr are unused
  T ui[3], umi[3], aci[3], pri = 0, rphii = 0, Ti = 0, rTi = 0;
  double phid = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    ui[i] = umi[i] = aci[i] = pr[i] = fr[i] = 0;
#pragma unroll
    for (int j = 0; j < 3; ++j) J[i][j] = ur[i][j] = 0;
  }
  T x0[3], l0[3];
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    T r[16], lo[4], N, dN[3];
    load_rec(rec, __shfl_sync(0xffffffffu, mynode, (lane & 24) + n), r, lo);
    shape(n, N, dN);
    if (n == 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) { x0[i] = r[i]; l0[i] = lo[i]; }
    } else {
      // dx/dxi from coordinates relative to node 0 (sum_a dN_a = 0), so the
      // FP32 path keeps the edge lengths to full precision
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const T d = (r[i] - x0[i]) + (lo[i] - l0[i]);
#pragma unroll
        for (int j = 0; j < 3; ++j) J[i][j] += d * dN[j];
      }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      ui[i] += r[3 + i] * N;
      umi[i] += r[6 + i] * N;
      if constexpr (vof) {
        aci[i] += r[9 + i] * N;
        pr[i] += r[12] * dN[i];
        fr[i] += r[13] * dN[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) ur[i][j] += r[3 + i] * dN[j];
      } else {
        fr[i] += r[10] * dN[i];
      }
    }
    phid += ((double)r[vof ? 13 : 9] + (double)lo[3]) * hex_n3<double>((hex_bit(n, 0) == g0) + (hex_bit(n, 1) == g1) +
                                                                      (hex_bit(n, 2) == g2));
    if constexpr (vof) {
      pri += r[12] * N;
      rphii += r[14] * N;
      Ti += r[15] * N;
    } else {
      Ti += r[10] * N;
      rTi += r[11] * N;
    }
  }
  // inverse Jacobian, DetJ (eval_shape_fem), G
  T Ai[3][3], G[3][3];
  Ai[0][0] = J[1][1] * J[2][2] - J[2][1] * J[1][2];
  Ai[0][1] = J[2][1] * J[0][2] - J[0][1] * J[2][2];
  Ai[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
  const T tmp = (T)1.0 / (Ai[0][0] * J[0][0] + Ai[0][1] * J[1][0] + Ai[0][2] * J[2][0]);
  Ai[0][0] *= tmp; Ai[0][1] *= tmp; Ai[0][2] *= tmp;
  Ai[1][0] = (J[1][2] * J[2][0] - J[1][0] * J[2][2]) * tmp;
  Ai[1][1] = (J[0][0] * J[2][2] - J[2][0] * J[0][2]) * tmp;
  Ai[1][2] = (J[1][0] * J[0][2] - J[0][0] * J[1][2]) * tmp;
  Ai[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) * tmp;
  Ai[2][1] = (J[2][0] * J[0][1] - J[0][0] * J[2][1]) * tmp;
  Ai[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * tmp;
  const T w = (T)1.0 / tmp;   // hex weights are 1
  T GG = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      G[i][j] = Ai[0][i] * Ai[0][j] + Ai[1][i] * Ai[1][j] + Ai[2][i] * Ai[2][j];
      GG += G[i][j] * G[i][j];
    }
  auto grad = [&](const T (&d)[3], T (&g)[3]) {
#pragma unroll
    for (int j = 0; j < 3; ++j) g[j] = d[0] * Ai[0][j] + d[1] * Ai[1][j] + d[2] * Ai[2][j];
  };
  const T fact2 = (T)(p.alfi * p.delt * p.gami), taut = (T)(4.0 / (p.delt * p.delt)), ts = (T)p.ts;
  const double phicd = clamp01(phid);
  const T phic = (T)phicd;
  const T uadv[3] = {ui[0] - umi[0], ui[1] - umi[1], ui[2] - umi[2]};
  const T taua = quad_uGu<T>(uadv, G);
  T* out = reinterpret_cast<T*>(a.sum) + (size_t)t * SW;
  T rr[8 * NF];
  if constexpr (vof) {   // src/solveQuenching.f90:295-523
    const T trG = G[0][0] + G[1][1] + G[2][2];
    T du[3][3], dp[3], dphi[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) grad(ur[i], du[i]);
    grad(pr, dp);
    grad(fr, dphi);
    const T rhoa = (T)p.rhoa, rhow = (T)p.rhow;
    // reciprocals of the launch constants: the point formulas multiply by
    // them where the reference divides (as the tet routines)
    const T its = (T)(1.0 / p.ts), irhoa = (T)(1.0 / p.rhoa), irhow = (T)(1.0 / p.rhow), ira = irhoa - irhow;
    const T divu = du[0][0] + du[1][1] + du[2][2], phii = (T)phid;
    T mdot, dmd;
    if (Ti > ts) {
      mdot = (T)p.c_evap * (T)(1.0 - phicd) * rhow * (Ti - ts) * its;
      dmd = -(T)p.c_evap * rhow * (Ti - ts) * its * (T)p.c_dmdot;
    } else {
      mdot = (T)p.c_cond * phic * rhoa * (Ti - ts) * its;
      dmd = (T)p.c_cond * rhoa * (Ti - ts) * its * (T)p.c_dmdot;
    }
    const T vdot = mdot * irhoa - mdot * irhow;
    T rho, mu;
    if (fluid) {
      rho = (T)(p.rhow * (1.0 - phicd) + p.rhoa * phicd);
      mu = (T)(p.muw * (1.0 - phicd) + p.mua * phicd);
    } else {
      rho = (T)p.rhos; mu = (T)p.mus;
    }
    const T lambda = (T)(-2.0 / 3.0) * mu;
    if (phid < 0.0 || phid > 1.0) dmd = 0;
    T tmp1[3], rL[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const T conv = du[i][0] * uadv[0] + du[i][1] * uadv[1] + du[i][2] * uadv[2];
      tmp1[i] = rho * aci[i] + rho * conv - (T)p.gravvec[i] * rho;
      rL[i] = tmp1[i] + dp[i];
    }
    const T res_phi = rphii + (uadv[0] * dphi[0] + uadv[1] * dphi[1] + uadv[2] * dphi[2]) + phii * vdot - mdot * irhoa;
    const T irho = (T)1.0 / rho;
    const T nu = mu * irho;
    const T taud = nu * nu * (T)12.0 * GG;
    const T tauM = irho * inv_sqrt(taut + taua + taud);
    const T tauLS = inv_sqrt(taut + taua);
    const T tauC = rho * sqrt(taua + taud) / trG;
    T kdc = 0;
    if (fabs(p.ns_kdc_w) + fabs(p.ns_kdc_a) > 0.0) {
      const double nk = (double)(p.ns_kdc_w * (1.0 - phicd) + p.ns_kdc_a * phicd);
      kdc = (T)low_word(nk) * sqrt((rL[0] * rL[0] + rL[1] * rL[1] + rL[2] * rL[2]) / GG);
    }
    T kdphi = 0;
    if (fabs(p.lsc_kdc) > 0.0) kdphi = (T)p.lsc_kdc * fabs(res_phi) / sqrt(GG);
    const T mupk = mu + kdc, dmdi = dmd * ira;
    const T wf = fluid ? w : (T)0;   // solid elements contribute nothing
    const T src = vdot + phii * ira * dmd - dmd * irhoa, fw = fact2 * wf;
    T* prec = out + gp * (TC ? HexTcLay::GPW : L::GPW);
    if constexpr (MAT && TC) {
      if (on) {
        put4(prec, Ai[0][0], Ai[0][1], Ai[0][2], Ai[1][0]);
        put4(prec + 4, Ai[1][1], Ai[1][2], Ai[2][0], Ai[2][1]);
        put4(prec + 8, Ai[2][2], wf, fw * mupk, fw * (tauC + lambda));
        put4(prec + 12, fw * tauM, fw * kdphi, dphi[0], dphi[1]);
        put4(prec + 16, dphi[2], Ai[0][0] * uadv[0] + Ai[0][1] * uadv[1] + Ai[0][2] * uadv[2],
             Ai[1][0] * uadv[0] + Ai[1][1] * uadv[1] + Ai[1][2] * uadv[2],
             Ai[2][0] * uadv[0] + Ai[2][1] * uadv[1] + Ai[2][2] * uadv[2]);
        put4(prec + 20, rho, rho * tauM, tauLS, src);
        put4(prec + 24, fw * tauC * dmdi * dmdi, fw * tauC * dmdi, fw * dmdi, (T)0);
      }
    } else if constexpr (MAT) {
      const T rt = rho * tauM;
      if (on) {
        put4(prec + 32, wf * rho, rt, wf, wf * tauLS);
        put4(prec + 36, fw, fw * rt, wf * rt, fact2 * src);
        put4(prec + 40, fw * mupk, fw * (tauC + lambda), fw * tauM, fw * kdphi);
        put4(prec + 44, dphi[0], dphi[1], dphi[2], fw * tauC * dmdi);
        put4(prec + 48, fw * tauC * dmdi * dmdi, fw * dmdi, (T)0, (T)0);
      }
    }
    T h[3];   // the viscous broadcast (:508-510) as one vector: svis_n = grad N_n . h
#pragma unroll
    for (int j = 0; j < 3; ++j) h[j] = (du[j][0] + du[0][j]) + (du[j][1] + du[1][j]) + (du[j][2] + du[2][j]);
    const T tdiv = -pri + tauC * divu;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      T N, dN[3], g[3];
      shape(n, N, dN);
      grad(dN, g);
      const T c = uadv[0] * g[0] + uadv[1] * g[1] + uadv[2] * g[2];
      if constexpr (MAT && !TC)
        if (on) put4(prec + 4 * n, g[0], g[1], g[2], c);
      const T sv = g[0] * h[0] + g[1] * h[1] + g[2] * h[2];
#pragma unroll
      for (int i = 0; i < 3; ++i)
        rr[5 * n + i] = wf * (-N * tmp1[i] - g[i] * tdiv + g[i] * tauC * vdot - g[i] * lambda * divu - mupk * sv +
                              rho * c * (-tauM * rL[i]));
      rr[5 * n + 3] = wf * (-N * (divu - vdot) + (g[0] * rL[0] + g[1] * rL[1] + g[2] * rL[2]) * (-tauM));
      rr[5 * n + 4] = wf * (-(N + tauLS * c) * res_phi - kdphi * (g[0] * dphi[0] + g[1] * dphi[1] + g[2] * dphi[2]) +
                            N * dmdi * tauC * (divu - vdot));
    }
  } else {   // src/solveQuenching.f90:712-856
    const T cpw = (T)p.cpw, cpa = (T)p.cpa, lh = (T)p.lh, its = (T)(1.0 / p.ts), itref = (T)(1.0 / p.tref);
    T dT[3];
    grad(fr, dT);
    T mdot, dmdT;
    if (Ti > ts) {
      mdot = (T)p.c_evap * (T)(1.0 - phicd) * (T)p.rhow * (Ti - ts) * its;
      dmdT = (T)p.c_evap * (T)(1.0 - phicd) * (T)p.rhow * its * (T)p.c_dmdot;
    } else {
      mdot = (T)p.c_cond * phic * (T)p.rhoa * (Ti - ts) * its;
      dmdT = (T)p.c_cond * phic * (T)p.rhoa * its * (T)p.c_dmdot;
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
    const T Se = ((cpw - cpa) * (Ti - ts) - lh) * mdot;
    const T udT = uadv[0] * dT[0] + uadv[1] * dT[1] + uadv[2] * dT[2];
    const T res = rcp * (rTi + udT) - Se;
    const T ircp = (T)1.0 / (rho * cp), kk = hk * ircp;
    const T tauT = ircp * inv_sqrt(taua + taut + kk * kk * (T)12.0 * GG);
    T kdcT = 0;
    if (fabs(p.tem_kdc) > 0.0 && fluid) kdcT = (T)p.tem_kdc * fabs(res) * inv_sqrt(GG) * itref;
    const T dSe = (cpw - cpa) * mdot + ((cpw - cpa) * (Ti - ts) - lh) * dmdT;
    // solid: no advection, no source
    const T fl = fluid ? (T)1 : (T)0, trq = fl * tauT * rcp, dSq = fl * dSe, HK = hk + kdcT;
    const T rmass = fluid ? res : rcp * rTi;
    extern __shared__ __align__(16) unsigned char hex_sm[];
    using HT = HexTemStage<T>;
    T* eb = reinterpret_cast<T*>(hex_sm) + (threadIdx.x >> 3) * HT::ES;   // this element's points
    T* q = eb + gp * HT::GPW;
    const T fact1 = (T)p.almi;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      T N, dN[3], g[3];
      shape(n, N, dN);
      grad(dN, g);
      const T c = fl * (uadv[0] * g[0] + uadv[1] * g[1] + uadv[2] * g[2]);
      rr[n] = w * (-N * rmass - trq * c * res - HK * (g[0] * dT[0] + g[1] * dT[1] + g[2] * dT[2]));
      if constexpr (MAT) {
        const T v[4] = {g[0], g[1], g[2], rcp * (fact1 * N + fact2 * c) - fact2 * dSq * N};
        store_row<4>(q + 4 * n, v);
        q[32 + n] = w * (N + trq * c);
      }
    }
    if constexpr (MAT) {
      q[40] = fact2 * HK * w;
      __syncwarp();
      T K[8];
#pragma unroll
      for (int b = 0; b < 8; ++b) K[b] = (T)0;
#pragma unroll 1
      for (int k = 0; k < 8; ++k) {   // row gp of the matrix, point k
        const T* z = eb + k * HT::GPW;
        T ga[4];
        lds4(z + 4 * gp, ga);
        const T A = z[32 + gp], hk2 = z[40];
        ga[0] *= hk2; ga[1] *= hk2; ga[2] *= hk2;
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          T gb[4];
          lds4(z + 4 * b, gb);
          K[b] += A * gb[3] + (ga[0] * gb[0] + ga[1] * gb[1] + ga[2] * gb[2]);
        }
      }
      if (on) {
        put4(out + 8 * gp, K[0], K[1], K[2], K[3]);
        put4(out + 8 * gp + 4, K[4], K[5], K[6], K[7]);
      }
    }
  }
  hex_sum_nodes<T, NF>(rr, lane);
  if (on)
#pragma unroll
    for (int f = 0; f < NF; ++f) out[RHS0 + NF * gp + f] = rr[f];
  double cfl = (double)p.delt * sqrt((double)taua);   // the largest over the warp's points
  int nbad = 0;
  const unsigned bad = __ballot_sync(0xffffffffu, on && !(w > (T)0));
  // an element counts once
  for (int e = 0; e < 4; ++e) nbad += ((bad >> (8 * e)) & 0xffu) != 0u;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) cfl = fmax(cfl, __shfl_xor_sync(0xffffffffu, cfl, off));
  if (lane == 0) {
    cfl_max(a.cfl_bits, cfl);
    if (nbad) atomicAdd(a.flags, nbad);
  }
}

// The block (row node a, column node b) of one Gauss point added to o, the
// per-point forms of the tet block sums (add_block): ga, gb the nodes' gradients
// and c, Na, Nb their shape values, s the point's factors (HexLay).
template <typename T>
__device__ __forceinline__ void hex_point(const T (&ga)[4], const T (&gb)[4], T Na, T Nb, T f1, T f2,
                                          const T (&s)[20], T (&o)[24]) {
  const T gab = ga[0] * gb[0] + ga[1] * gb[1] + ga[2] * gb[2];
  const T beta = f1 * Nb + f2 * gb[3];
  const T P = s[4] * Nb, Q = s[5] * ga[3], R = s[4] * Na, Tt = s[6] * beta;
  const T dg = s[8] * gab + s[0] * (Na + s[1] * ga[3]) * beta;
  const T gam = s[2] * Na + s[3] * ga[3], V = f2 * Nb * gam, uNa = s[15] * Na, uNb = s[15] * Nb, NN = Na * Nb;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T ka = s[8] * gb[i], kb = s[9] * ga[i];
#pragma unroll
    for (int j = 0; j < 3; ++j) o[4 * i + j] += ka * ga[j] + kb * gb[j];
    o[5 * i] += dg;
    o[4 * i + 3] += gb[i] * Q - ga[i] * P;
    o[12 + i] += gb[i] * R + ga[i] * Tt;
    o[16 + i] += s[12 + i] * V - gb[i] * uNa;
    o[20 + i] += ga[i] * uNb;
  }
  o[15] += s[10] * gab;
  o[19] += gam * (beta + s[7] * Nb) + s[11] * gab + s[16] * NN;
  o[23] -= s[17] * NN;
}

// ------------------------------------------------------------------------
// Tensor-core element matrices (FP32 NS+VOF hexahedra).
//
// Every block value t of the quench matrix is, per Gauss point g, a bilinear
// form in the features (N, grad N) of the row node a and the column node b.
// Written with the reference-element features f_g = (N, dN/dxi) (the same
// for every element), the element's block is
//     K_t[a][b] = sum_g sum_{r,s} C'_{t,g}[r][s] f_g[r][a] f_g[s][b],
// with C' = T^T C T, T = diag(1, dxi/dx^T) mapping reference to physical
// gradients.  So all element matrices of a tile are ONE dense product
//     D[(t, e), (a, b)] = A[(t, e), (g, r, s)] * W[(g, r, s), (a, b)],
// M = 8 types x 16 elements = 128, K = 8 points x 16 = 128, N = 64, with
// the constant W = f_g (x) f_g shared by all elements, on tcgen05 (kind::tf32,
// A and W K-major in shared memory without swizzle, D in TMEM).  FP32
// accuracy comes from the 3xTF32 split A_hi W_hi + A_hi W_lo + A_lo W_hi
// (W's split precomputed on the host).  One CTA of 256 threads per SM loops
// over tiles of 16 elements; thread (element el, point g)
// of each half builds its point's 4x4 C' for 4 of a group's 8 slot values
// (three groups of 8 cover the 24; the value is a template parameter),
// thread 0 issues the 48 MMAs of a group into its 64 TMEM columns and
// commits them to an mbarrier; the epilogue reads the 192 columns back and
// writes each element's 64 x 24 block values (slot order) through shared
// memory with coalesced stores.

constexpr int TC_EB = 16;                                 // elements per tile
constexpr int TC_KST = 64 * 24 + 4;                       // staging floats per element (padded)
constexpr int TC_A_BYTES = 128 * 128 * 4;                 // one A operand (hi or lo)
constexpr int TC_W_BYTES = 64 * 128 * 4;                  // one W operand (hi or lo)
constexpr int TC_SMEM = 2 * TC_A_BYTES + 2 * TC_W_BYTES;  // 192 KB
constexpr int TC_TMEM_COLS = 256;                         // 3 groups x 64 columns
constexpr long TC_WAIT_LIMIT = 1L << 26;                  // bounded mbarrier wait (iterations)

struct HexTcArgs {
  const float* rec;    // element records, HexTcLay
  const float* w;      // W hi then W lo, canonical K-major no-swizzle layout (2 x 8192 floats)
  float* kbuf;         // E x 64 x 24 block values
  int* flags;          // [2] set when an mbarrier wait gave up
  int E;
  float fact1, fact2;
};

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float tc_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return __uint_as_float(r);
}
// shared-memory matrix descriptor: SWIZZLE_NONE, K-major, version 1
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void tc_mma(uint32_t dcol, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
               ::"r"(dcol), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
  uint32_t done = 0;
  for (long it = 0; it < TC_WAIT_LIMIT && !done; ++it)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
__device__ __forceinline__ void tc_ld16(uint32_t addr, float* v) {
  uint32_t r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// C' (reference features, row-major 4x4: [r][s], r on the row node a) of slot
// value t at one point, from the point record q (HexTcLay): the per-point
// forms of hex_point with u.grad N = v . dN/dxi (v = dxi/dx uadv),
// grad N_a . grad N_b = dN_a/dxi Gh dN_b/dxi (Gh = dxi/dx dxi/dx^T) and the
// physical derivative j = dN/dxi . a_j (a_j column j of dxi/dx).
template <int t>
__device__ __forceinline__ void tc_coeffs(const float* q, const float Gh[3][3], float f1, float f2, float C[16]) {
#pragma unroll
  for (int k = 0; k < 16; ++k) C[k] = 0.f;
  const float w = q[9], KA = q[10], KB = q[11], MM = q[12], KDP = q[13];
  const float v[3] = {q[17], q[18], q[19]};
  const float rho = q[20], rt = q[21], tls = q[22], src = q[23], eps = q[24], ufac = q[25], plfac = q[26];
  auto A = [&](int k, int j) { return q[3 * k + j]; };   // dxi_k/dx_j
  if constexpr (t < 12 && (t & 3) != 3) {  // K(i, j)
    constexpr int i = t >> 2, j = t & 3;
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) C[4 * (1 + k) + 1 + l] = KA * A(k, j) * A(l, i) + KB * A(k, i) * A(l, j);
    if constexpr (i == j) {
      const float al[4] = {1.f, rt * v[0], rt * v[1], rt * v[2]};
      const float be[4] = {f1, f2 * v[0], f2 * v[1], f2 * v[2]};
      const float wr = w * rho;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) C[4 * r + c] += wr * al[r] * be[c];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) C[4 * (1 + k) + 1 + l] += KA * Gh[k][l];
    }
  } else if constexpr (t < 12) {           // G(i)
    constexpr int i = t >> 2;
    const float fw = f2 * w;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      C[4 * (1 + k)] = -fw * A(k, i);
#pragma unroll
      for (int l = 0; l < 3; ++l) C[4 * (1 + k) + 1 + l] = fw * rt * v[k] * A(l, i);
    }
  } else if constexpr (t < 15) {           // D(d)
    constexpr int d = t - 12;
    const float wrt = w * rt;
#pragma unroll
    for (int l = 0; l < 3; ++l) C[1 + l] = f2 * w * A(l, d);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      C[4 * (1 + k)] = wrt * A(k, d) * f1;
#pragma unroll
      for (int l = 0; l < 3; ++l) C[4 * (1 + k) + 1 + l] = wrt * A(k, d) * f2 * v[l];
    }
  } else if constexpr (t == 15) {          // M
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) C[4 * (1 + k) + 1 + l] = MM * Gh[k][l];
  } else if constexpr (t < 19) {           // LSU(d)
    constexpr int d = t - 16;
    const float c0 = q[14 + d] * f2 * w;
    C[0] = c0;
#pragma unroll
    for (int k = 0; k < 3; ++k) C[4 * (1 + k)] = c0 * tls * v[k];
#pragma unroll
    for (int l = 0; l < 3; ++l) C[1 + l] = -ufac * A(l, d);
  } else if constexpr (t == 19) {          // LS
    const float al[4] = {1.f, tls * v[0], tls * v[1], tls * v[2]};
    const float ga[4] = {f1 + f2 * src, f2 * v[0], f2 * v[1], f2 * v[2]};
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) C[4 * r + c] = w * al[r] * ga[c];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) C[4 * (1 + k) + 1 + l] += KDP * Gh[k][l];
    C[0] += eps;
  } else if constexpr (t < 23) {           // ULS(d)
    constexpr int d = t - 20;
#pragma unroll
    for (int k = 0; k < 3; ++k) C[4 * (1 + k)] = ufac * A(k, d);
  } else {                                 // PLS
    C[0] = -plfac;
  }
}

// A rows m = 16 t8 + el, 16-byte chunk kc = 4 g + r (hi and lo operands)
template <int t>
__device__ __forceinline__ void tc_store_type(const float* q, const float Gh[3][3], float f1, float f2,
                                              unsigned char* sAh, unsigned char* sAl, int el, int g) {
  float C[16];
  tc_coeffs<t>(q, Gh, f1, f2, C);
  const int m = 16 * (t & 7) + el;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int off = (4 * g + r) * 2048 + (m >> 3) * 128 + (m & 7) * 16;
    float4 h, l;
    h.x = tc_tf32(C[4 * r]); h.y = tc_tf32(C[4 * r + 1]); h.z = tc_tf32(C[4 * r + 2]); h.w = tc_tf32(C[4 * r + 3]);
    l.x = tc_tf32(C[4 * r] - h.x); l.y = tc_tf32(C[4 * r + 1] - h.y);
    l.z = tc_tf32(C[4 * r + 2] - h.z); l.w = tc_tf32(C[4 * r + 3] - h.w);
    *reinterpret_cast<float4*>(sAh + off) = h;
    *reinterpret_cast<float4*>(sAl + off) = l;
  }
}

// the 8 slot values of group GRP: the warp-uniform half hf of the CTA builds 4 of them
template <int GRP>
__device__ __forceinline__ void tc_store_group(int hf, const float* q, const float Gh[3][3], float f1, float f2,
                                               unsigned char* sAh, unsigned char* sAl, int el, int g) {
  if (hf == 0) {
    tc_store_type<8 * GRP + 0>(q, Gh, f1, f2, sAh, sAl, el, g);
    tc_store_type<8 * GRP + 1>(q, Gh, f1, f2, sAh, sAl, el, g);
    tc_store_type<8 * GRP + 2>(q, Gh, f1, f2, sAh, sAl, el, g);
    tc_store_type<8 * GRP + 3>(q, Gh, f1, f2, sAh, sAl, el, g);
  } else {
    tc_store_type<8 * GRP + 4>(q, Gh, f1, f2, sAh, sAl, el, g);
    tc_store_type<8 * GRP + 5>(q, Gh, f1, f2, sAh, sAl, el, g);
    tc_store_type<8 * GRP + 6>(q, Gh, f1, f2, sAh, sAl, el, g);
    tc_store_type<8 * GRP + 7>(q, Gh, f1, f2, sAh, sAl, el, g);
  }
}

constexpr int TC_THREADS = 256;

// builds group GRP's operands, issues its MMAs and waits for them; false when the wait gave up
template <int GRP>
__device__ __forceinline__ bool tc_group(int hf, const float* q, const float Gh[3][3], float f1, float f2,
                                         unsigned char* sAh, unsigned char* sAl, unsigned char* sWh,
                                         unsigned char* sWl, int el, int g, uint32_t tm, uint32_t barp,
                                         uint32_t idesc, uint32_t& phase) {
  tc_store_group<GRP>(hf, q, Gh, f1, f2, sAh, sAl, el, g);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (threadIdx.x == 0) {
    const uint32_t dcol = tm + 64 * GRP;
    const uint32_t ah = tc_smem(sAh), al = tc_smem(sAl), wh = tc_smem(sWh), wl = tc_smem(sWl);
    for (int ks = 0; ks < 16; ++ks)
      tc_mma(dcol, tc_desc(ah + ks * 4096, 2048, 128), tc_desc(wh + ks * 2048, 1024, 128), idesc, ks > 0);
    for (int ks = 0; ks < 16; ++ks)
      tc_mma(dcol, tc_desc(ah + ks * 4096, 2048, 128), tc_desc(wl + ks * 2048, 1024, 128), idesc, 1u);
    for (int ks = 0; ks < 16; ++ks)
      tc_mma(dcol, tc_desc(al + ks * 4096, 2048, 128), tc_desc(wh + ks * 2048, 1024, 128), idesc, 1u);
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(barp)
                 : "memory");
  }
  // the operands are free again (and, after the last group, D is complete)
  const bool done = tc_wait(barp, phase);
  const bool ok = __syncthreads_and(done) != 0;
  if (ok) phase ^= 1u;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  return ok;
}

__global__ void __launch_bounds__(TC_THREADS, 1) hex_tc_matrix_kernel(const HexTcArgs a) {
  extern __shared__ __align__(1024) unsigned char tc_sm[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tbase;
  unsigned char* sAh = tc_sm;
  unsigned char* sAl = tc_sm + TC_A_BYTES;
  unsigned char* sWh = tc_sm + 2 * TC_A_BYTES;
  unsigned char* sWl = sWh + TC_W_BYTES;
  float* kst = reinterpret_cast<float*>(tc_sm);             // epilogue staging over the A operands
  const int t = threadIdx.x, wid = t >> 5, lane = t & 31;
  const int hf = t >> 7, tt = t & 127;                      // half of the CTA (4 of each group's 8 values)
  const int el = tt & 15, g = tt >> 4;                      // this thread's element and point
  {  // W hi / lo into shared memory (already in the canonical layout)
    const float4* src = reinterpret_cast<const float4*>(a.w);
    float4* dst = reinterpret_cast<float4*>(sWh);
    for (int i = t; i < 2 * TC_W_BYTES / 16; i += TC_THREADS) dst[i] = src[i];
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (wid == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&tbase)),
                 "r"(TC_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tm = tbase, barp = tc_smem(&bar);
  // kind::tf32, F32 accumulate, A and B K-major, N = 64, M = 128
  const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
  const float f1 = a.fact1, f2 = a.fact2;
  uint32_t phase = 0;
  bool ok = true;
  const int ntiles = (a.E + TC_EB - 1) / TC_EB;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int e0 = tile * TC_EB, e = e0 + el;
    float q[HexTcLay::GPW];
    if (e < a.E) {
      const float4* r4 = reinterpret_cast<const float4*>(a.rec + (size_t)e * HexTcLay::SW + g * HexTcLay::GPW);
#pragma unroll
      for (int k = 0; k < HexTcLay::GPW / 4; ++k) {
        const float4 x = __ldg(r4 + k);
        q[4 * k] = x.x; q[4 * k + 1] = x.y; q[4 * k + 2] = x.z; q[4 * k + 3] = x.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < HexTcLay::GPW; ++k) q[k] = 0.f;
    }
    float Gh[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int l = 0; l < 3; ++l) Gh[k][l] = q[3 * k] * q[3 * l] + q[3 * k + 1] * q[3 * l + 1] + q[3 * k + 2] * q[3 * l + 2];
    ok = tc_group<0>(hf, q, Gh, f1, f2, sAh, sAl, sWh, sWl, el, g, tm, barp, idesc, phase) &&
         tc_group<1>(hf, q, Gh, f1, f2, sAh, sAl, sWh, sWl, el, g, tm, barp, idesc, phase) &&
         tc_group<2>(hf, q, Gh, f1, f2, sAh, sAl, sWh, sWl, el, g, tm, barp, idesc, phase);
    if (!ok) break;
    // epilogue: warp quartet hf reads columns [32 hf, 32 hf + 32) of each group's 64, lanes 32 (wid % 4) + lane
    {
      const int w4 = wid & 3, m = 32 * w4 + lane, t8 = m >> 4, eli = m & 15;
      float* dst = kst + eli * TC_KST;
#pragma unroll
      for (int grp = 0; grp < 3; ++grp)
#pragma unroll
        for (int c = 0; c < 32; c += 16) {
          const int c0 = 32 * hf + c;
          float v[16];
          tc_ld16(tm + ((uint32_t)(32 * w4) << 16) + 64 * grp + c0, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) dst[(c0 + j) * 24 + 8 * grp + t8] = v[j];
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    {
      const int nel = min(TC_EB, a.E - e0);
      float4* out = reinterpret_cast<float4*>(a.kbuf + (size_t)e0 * 1536);
      for (int i = t; i < nel * 384; i += TC_THREADS) {
        const int ee = i / 384, j4 = i - ee * 384;
        out[i] = *reinterpret_cast<const float4*>(kst + ee * TC_KST + 4 * j4);
      }
    }
    __syncthreads();   // staging (the A operands) free for the next tile
  }
  if (!ok) {   // give the MMAs in flight one more bounded wait before TMEM is released
    tc_wait(barp, phase);
    if (t == 0) atomicOr(a.flags + 2, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (wid == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(TC_TMEM_COLS));
}

// shared memory per warp: blocks [4 elements][8 columns][BSTR], RHS rows
// [4][RSTR], row accumulator [max_deg][NVP]; ints: slots [4][8], columns
template <typename T, int KIND> struct HexSmem {
  static constexpr int NV = HexLay<KIND>::NV, NF = HexLay<KIND>::NF;
  static constexpr int CH = 4;
  static constexpr int NVP = (NV < 4) ? 1 : NV;
  static constexpr int BSTR = (NV < 4) ? 1 : NV + 16 / (int)sizeof(T);
  static constexpr int RSTR = NF + 1;
  __host__ __device__ static size_t bytes(int max_deg) {
    size_t b = sizeof(T) * ((size_t)8 * CH * BSTR + (size_t)CH * RSTR + (size_t)max_deg * NVP);
    b = (b + 15) & ~(size_t)15;
    b += sizeof(int) * ((size_t)8 * CH + max_deg);
    return (b + 15) & ~(size_t)15;
  }
};

template <typename T, int KIND, bool TC = false>
__global__ void __launch_bounds__(128) hex_rows_kernel(const AsmArgs a) {
  using S = HexSmem<T, KIND>;
  using L = HexLay<KIND>;
  constexpr int NV = S::NV, NF = S::NF, NVP = S::NVP, BSTR = S::BSTR, RSTR = S::RSTR, CH = S::CH;
  constexpr int WARPS = 4;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned masks[24];
  if (threadIdx.x < 24) masks[threadIdx.x] = (KIND == OVS_ASM_TEM) ? (TB | (TB << 8) | (TB << 16)) : mask_of(threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned char* base = smem_raw + (size_t)wid * S::bytes(a.max_deg);
  T* blk = reinterpret_cast<T*>(base);                 // [CH][8][BSTR]
  T* rvs = blk + 8 * CH * BSTR;                        // [CH][RSTR]
  T* acc = rvs + CH * RSTR;                            // [max_deg][NVP]
  size_t off = sizeof(T) * ((size_t)8 * CH * BSTR + (size_t)CH * RSTR + (size_t)a.max_deg * NVP);
  off = (off + 15) & ~(size_t)15;
  int* slot = reinterpret_cast<int*>(base + off);      // [CH][8]
  int* cols = slot + 8 * CH;                           // [max_deg]
  const T* sum = reinterpret_cast<const T*>(a.rec);
  const uint2* n2s8 = reinterpret_cast<const uint2*>(a.n2s);
  const int jl = lane >> 3, bl = lane & 7;
  for (int A = blockIdx.x * WARPS + wid; A < a.N; A += gridDim.x * WARPS) {
    const int rp = a.rowptr[A], deg = a.rowptr[A + 1] - rp;
    const int ep = a.n2e_ptr[A], ne = a.n2e_ptr[A + 1] - ep;
    for (int s = lane; s < deg; s += 32) cols[s] = a.colidx[rp + s];
    for (int q = lane; q < deg * NVP; q += 32) acc[q] = (T)0;
    T racc = (T)0;
    __syncwarp();
    for (int c0 = 0; c0 < ne; c0 += CH) {
      const int nc = min(CH, ne - c0);
      if (jl < nc) {
        const int packed = __ldg(a.n2e + ep + c0 + jl);
        const uint2 sl = __ldg(n2s8 + ep + c0 + jl);
        const int e = packed >> 3, la = packed & 7;
        T o[NVP], rv[NF];
        if constexpr (TC) {   // block values of the tensor-core pass, slot order
          const float4* kb = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.kbuf) +
                                                             ((size_t)e * 64 + la * 8 + bl) * 24);
#pragma unroll
          for (int v = 0; v < 6; ++v) {
            const float4 x = __ldg(kb + v);
            o[4 * v] = x.x; o[4 * v + 1] = x.y; o[4 * v + 2] = x.z; o[4 * v + 3] = x.w;
          }
#pragma unroll
          for (int f = 0; f < NF; ++f) rv[f] = sum[(size_t)e * HexTcLay::SW + HexTcLay::RHS0 + 5 * la + f];
        } else {
          o[0] = __ldg(sum + (size_t)e * L::SW + 8 * la + bl);
          rv[0] = sum[(size_t)e * L::SW + L::RHS0 + la];
        }
        T* dst = blk + (jl * 8 + bl) * BSTR;
        if constexpr (NV >= 4) {
#pragma unroll
          for (int v = 0; v < NV; v += 4) store_row<4>(dst + v, o + v);
        } else {
          dst[0] = o[0];
        }
        const unsigned word = bl < 4 ? sl.x : sl.y;
        slot[jl * 8 + bl] = (int)((word >> (8 * (bl & 3))) & 0xffu);
        if (bl == 0) {
#pragma unroll
          for (int f = 0; f < NF; ++f) rvs[jl * RSTR + f] = rv[f];
        }
      }
      __syncwarp();
      // ordered reduction: the 8 blocks of one element go to distinct slots
      if constexpr (NV >= 4) {
        constexpr int NG = NV / 4;
        for (int j = 0; j < nc; ++j) {
          for (int q = lane; q < 8 * NG; q += 32) {
            const int b = q / NG, gidx = q - b * NG;
            Vec4<T>::add(acc + slot[j * 8 + b] * NVP + gidx * 4, blk + (j * 8 + b) * BSTR + gidx * 4);
          }
          __syncwarp();
        }
      } else {
        for (int j = 0; j < nc; ++j) {
          if (lane < 8) acc[slot[j * 8 + lane]] += blk[j * 8 + lane];
          __syncwarp();
        }
      }
      if (lane < NF)
        for (int j = 0; j < nc; ++j) racc += rvs[j * RSTR + lane];
      __syncwarp();
    }
    // row write with the Dirichlet treatment (as for the tets)
    const unsigned ibA = a.ibc[A];
    {
      T* outp = reinterpret_cast<T*>(a.vals) + (size_t)rp * NV;
      const T cnt = (T)ne;
      if constexpr (NV >= 4) {
        constexpr int NG = NV / 4;
        for (int q = lane; q < deg * NG; q += 32) {
          const int s = q / NG, gidx = q - s * NG;
          const int B = cols[s];
          const unsigned ibB = __ldg(a.ibc + B);
          const bool dg = B == A;
          T v4[4];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const unsigned m = masks[4 * gidx + t];
            T val = acc[s * NVP + 4 * gidx + t];
            if ((ibA & m & 0xffu) || ((ibB << 8) & m & 0xff00u)) val = (T)0;
            if (dg && ((ibA << 16) & m & 0xff0000u)) val = cnt;
            v4[t] = val;
          }
          store_row<4>(outp + (size_t)s * NV + 4 * gidx, v4);
        }
      } else {
        for (int q = lane; q < deg; q += 32) {
          const int B = cols[q];
          const unsigned ibB = __ldg(a.ibc + B);
          T val = acc[q];
          if ((ibA & TB) || (ibB & TB)) val = (T)0;
          if (B == A && (ibA & TB)) val = cnt;
          outp[q] = val;
        }
      }
    }
    if (a.vec && lane < NF) {
      unsigned bit;
      if (KIND == OVS_ASM_TEM) bit = TB;
      else bit = (lane < 3) ? (1u << lane) : (lane == 3 ? PB : FB);
      T v = (ibA & bit) ? (T)0 : racc;
      if (!isfinite((double)v)) atomicOr(a.flags + 1, 1);
      reinterpret_cast<T*>(a.rhs)[(size_t)lane * a.N + A] = v;
    }
    __syncwarp();
  }
}

// Row pass of the NS+VOF hexahedra: one warp per CSR row, in the order of the
// row records.  A chunk is 4 of the row's elements, 8 lanes per element, a
// column per lane.  The elements' point records pass through shared memory two
// points at a time, copied asynchronously ahead of the points being summed, and
// a lane sums its block over the 8 points in registers.  Then the chunk's 32
// blocks meet in the same shared memory, and each output task (slot, 4-value
// group) adds the blocks of its slot in ascending element order (`has` and
// `colof` name them; `acc` carries the sums between chunks) and in the last
// chunk writes the group, consecutive lanes writing consecutive groups.
// Bound: latency at 16 (FP64) and 20 (FP32) warps per SM; the FP64 pipe is a
// third busy (74 operations per block and point), the shared-memory reads that
// feed it another third.  96^3 hexahedra: FP64 11.03 -> 6.62 ms, FP32 5.42 ->
// 4.01 ms against records read from global memory at every point, one point
// after the other, with the shape values recomputed; two columns per lane and 8
// elements per chunk took 7.31 and 4.23 ms (254 and 166 registers).
template <typename T> struct HexRows {
  static constexpr int GPS = 2;                                        // points per stage
  static constexpr int EPC = 4, LPE = 8;                               // elements per chunk, lanes per element
  static constexpr int GPW = HexLay<OVS_ASM_NSVOF>::GPW;
  static constexpr int ES = GPS * GPW + (sizeof(T) == 8 ? 2 : 8);      // element stride: quarter warps spread over the banks
  static constexpr int BST = sizeof(T) == 8 ? 26 : 28;                 // block stride
  static constexpr int UNITS = GPS * GPW * (int)sizeof(T) / 16;        // 16-byte copies per element and stage
  static constexpr size_t stage = sizeof(T) * (size_t)(2 * EPC * ES > 8 * EPC * BST ? 2 * EPC * ES : 8 * EPC * BST);
  static_assert(GPS * GPW * sizeof(T) % 16 == 0 && ES * sizeof(T) % 16 == 0 && BST * sizeof(T) % 16 == 0, "16-byte units");
  // per warp: stages (then blocks), per slot the columns of the chunk's
  // elements, which of them hold the slot, the Dirichlet mask; carried sums
  __host__ __device__ static size_t slots(int max_deg) { return ((size_t)max_deg + 3) & ~(size_t)3; }
  __host__ __device__ static size_t bytes(int max_deg, bool carry) {
    return stage + (EPC + 8) * slots(max_deg) + (carry ? sizeof(T) * 24 * (size_t)max_deg : 0);
  }
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(128, (sizeof(T) == 8 ? 4 : 5)) hex_block_rows_kernel(const AsmArgs a, int carry) {
  using L = HexLay<OVS_ASM_NSVOF>;
  using H = HexRows<T>;
  constexpr int EPC = H::EPC, LPE = H::LPE;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned masks[24];
  __shared__ T Nt[8][8];
  if (threadIdx.x < 24) masks[threadIdx.x] = mask_of(threadIdx.x);
  if (threadIdx.x < 64) Nt[threadIdx.x >> 3][threadIdx.x & 7] = hex_N<T>(threadIdx.x >> 3, threadIdx.x & 7);
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, el = lane / LPE, cp = lane % LPE;
  unsigned char* base = smem_raw + (size_t)wid * H::bytes(a.max_deg, carry);
  T* st = reinterpret_cast<T*>(base);
  const int ns = (int)H::slots(a.max_deg);
  uint8_t* colof = base + H::stage;                            // [ns][EPC]: column of element j in slot s
  unsigned* has = reinterpret_cast<unsigned*>(colof + EPC * ns);   // [ns]: bit j, element j holds slot s
  unsigned* cib = has + ns;                                    // [ns]
  T* acc = reinterpret_cast<T*>(cib + ns);
  const T* sum = reinterpret_cast<const T*>(a.rec);
  const uint2* n2s8 = reinterpret_cast<const uint2*>(a.n2s);
  const T f1 = (T)a.p.almi, f2 = (T)(a.p.alfi * a.p.delt * a.p.gami);
  // a row's record, and element ids and slots of its first chunk, travel while
  // the row before it is summed
  int t = blockIdx.x * 4 + wid;
  const int step = gridDim.x * 4;
  int4 rn = t < a.N ? __ldg(a.row_rec + t) : make_int4(0, 0, 0, 0);
  int pkn = 0;
  uint2 wn = make_uint2(0u, 0u);
  if (el < rn.w >> 16) {
    pkn = __ldg(a.n2e + rn.z + el);
    wn = __ldg(n2s8 + rn.z + el);
  }
  for (; t < a.N; t += step) {
    const int4 rr = rn;
    const int A = rr.x, deg = rr.w & 0xff, sd = (rr.w >> 8) & 0xff, ne = rr.w >> 16;
    T* out = reinterpret_cast<T*>(a.vals) + (size_t)rr.y * 24;
    T res[2] = {(T)0, (T)0};   // residual fields cp and (lane 0 of an element) 4
    unsigned ibA = 0;
    for (int c0 = 0; c0 == 0 || c0 < ne; c0 += EPC) {
      const int nc = min(EPC, ne - c0);
      const bool on = el < nc;
      int pk = pkn;
      uint2 w = wn;
      if (c0 > 0 && on) {
        pk = __ldg(a.n2e + rr.z + c0 + el);
        w = __ldg(n2s8 + rr.z + c0 + el);
      }
      const int la = pk & 7;
      const T* mine = sum + (size_t)(pk >> 3) * L::SW;
      auto fetch = [&](int k) {   // stage k: points 2 k, 2 k + 1 of the chunk's elements, an element by its 8 lanes
        if (on) {
          unsigned char* dst = reinterpret_cast<unsigned char*>(st + ((k & 1) * EPC + el) * H::ES) + 16 * cp;
          const unsigned char* src = reinterpret_cast<const unsigned char*>(mine + k * H::GPS * H::GPW) + 16 * cp;
#pragma unroll
          for (int u = 0; u < H::UNITS; u += LPE)
            if (u + LPE <= H::UNITS || cp < H::UNITS - u) cp_async16(dst + 16 * u, src + 16 * u);
        }
        cp_async_commit();
      };
      fetch(0);
      fetch(1);
      int col = 0;
      unsigned ibB = 0;
      T r0 = (T)0, r1 = (T)0;
      if (c0 == 0) {
        if (lane < deg) col = __ldg(a.colidx + rr.y + lane);
        ibA = __ldg(a.ibc + A);
        rn = t + step < a.N ? __ldg(a.row_rec + t + step) : make_int4(0, 0, 0, 0);
      }
      for (int s = lane; s < deg; s += 32) has[s] = 0u;
      __syncwarp();
      if (on) {   // the lane's column
        const unsigned s = ((cp < 4 ? w.x : w.y) >> (8 * (cp & 3))) & 0xffu;
        colof[EPC * s + el] = (uint8_t)cp;
        atomicOr(has + s, 1u << el);
        if (cp < 4) r0 = __ldg(mine + L::RHS0 + 5 * la + cp);
        if (cp == 0) r1 = __ldg(mine + L::RHS0 + 5 * la + 4);
      }
      T o[24];
#pragma unroll
      for (int v = 0; v < 24; ++v) o[v] = (T)0;
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {
        if (k < 3) cp_async_wait<1>(); else cp_async_wait<0>();
        __syncwarp();
        if (k == 1 && c0 == 0) {
          if (lane < deg) ibB = __ldg(a.ibc + col);
          pkn = 0;
          if (el < rn.w >> 16) {
            pkn = __ldg(a.n2e + rn.z + el);
            wn = __ldg(n2s8 + rn.z + el);
          }
        }
        if (on) {
#pragma unroll 1
          for (int h = 0; h < H::GPS; ++h) {
            const T* q = st + ((k & 1) * EPC + el) * H::ES + h * H::GPW;
            const T* N = Nt[H::GPS * k + h];
            T s[20], ga[4], gb[4];
#pragma unroll
            for (int v = 0; v < 20; v += 4) lds4(q + 32 + v, s + v);
            lds4(q + 4 * la, ga);
            lds4(q + 4 * cp, gb);
            hex_point<T>(ga, gb, N[la], N[cp], f1, f2, s, o);
          }
        }
        __syncwarp();
        if (k < 2) fetch(k + 2);
      }
      if (c0 == 0) {
        if (lane < deg) cib[lane] = ibB;
        for (int s = lane + 32; s < deg; s += 32) cib[s] = __ldg(a.ibc + __ldg(a.colidx + rr.y + s));
      }
      res[0] += r0;
      res[1] += r1;
      // the chunk's blocks, in the stages' place
      if (on) {
#pragma unroll
        for (int v = 0; v < 24; v += 4) store_row<4>(st + lane * H::BST + v, o + v);
      }
      __syncwarp();
      const bool last = c0 + EPC >= ne;
      for (int q = lane; q < deg * 6; q += 32) {
        const int s = q / 6, g = q - 6 * s;
        if (!last && c0 > 0 && has[s] == 0u) continue;   // nothing of this chunk
        T v[4] = {(T)0, (T)0, (T)0, (T)0};
        if (c0 > 0) lds4(acc + 24 * s + 4 * g, v);
        const T* blk = st + 4 * g;
        for (unsigned m = has[s]; m; m &= m - 1) {   // ascending elements; an element's 8 columns have distinct slots
          const int j = __ffs(m) - 1;
          T x[4];
          lds4(blk + (j * 8 + colof[EPC * s + j]) * H::BST, x);
          v[0] += x[0]; v[1] += x[1]; v[2] += x[2]; v[3] += x[3];
        }
        if (!last) {
          store_row<4>(acc + 24 * s + 4 * g, v);
          continue;
        }
        const unsigned ib = cib[s];
        if ((ibA | ib) != 0u) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const unsigned m = masks[4 * g + u];
            if ((ibA & m & 0xffu) || ((ib << 8) & m & 0xff00u)) v[u] = (T)0;
            if (s == sd && ((ibA << 16) & m & 0xff0000u)) v[u] = (T)ne;
          }
        }
        store4_cs(out + 24 * (size_t)s + 4 * g, v);
      }
      __syncwarp();
    }
    // residual: the elements' lanes added by halving (fields 0-3 and 4)
#pragma unroll
    for (int o = 16; o >= LPE; o >>= 1) {
      res[0] += __shfl_xor_sync(0xffffffffu, res[0], o);
      res[1] += __shfl_xor_sync(0xffffffffu, res[1], o);
    }
    if (a.vec && lane < 4) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int f = u ? 4 : lane;
        if (u && lane) break;
        const T v = (ibA & (1u << f)) ? (T)0 : res[u];   // IBC bits 0-4: u1 u2 u3 p phi
        if (!isfinite((double)v)) atomicOr(a.flags + 1, 1);
        reinterpret_cast<T*>(a.rhs)[(size_t)f * a.N + A] = v;
      }
    }
  }
}

template <typename T, int KIND>
int launch_assemble_hex(ovs_ctx* c, const AsmArgs& a0, const SumArgs& sa, int parts) {
  if (!a0.mat) {   // vector-only pass, as for the tets
    hex_element_kernel<T, KIND, false, false><<<(sa.E + 15) / 16, 128, 0, c->stream>>>(sa);
    ++c->launches;
    OVS_CUDA_TRY(cudaGetLastError());
    return launch_residual_rows<T, HexLay<KIND>::NF>(c, a0, KIND == OVS_ASM_TEM);
  }
  constexpr bool can_tc = std::is_same<T, float>::value && KIND == OVS_ASM_NSVOF;
  const bool tc = can_tc && c->hex_tc;
  AsmArgs a = a0;
  if (tc) {
    int st;
    if ((st = hex_tc_prepare(c))) return st;
    a.kbuf = c->hex_kbuf;
  }
  if (parts & 1) {
    if (tc) {
      if constexpr (can_tc) {
        hex_element_kernel<T, KIND, true><<<(sa.E + 15) / 16, 128, 0, c->stream>>>(sa);
        ++c->launches;
        OVS_CUDA_TRY(cudaGetLastError());
        HexTcArgs ta;
        ta.rec = reinterpret_cast<const float*>(sa.sum);
        ta.w = c->hex_w;
        ta.kbuf = reinterpret_cast<float*>(c->hex_kbuf);
        ta.flags = c->flags;
        ta.E = sa.E;
        ta.fact1 = (float)sa.p.almi;
        ta.fact2 = (float)(sa.p.alfi * sa.p.delt * sa.p.gami);
        OVS_CUDA_TRY(cudaFuncSetAttribute(hex_tc_matrix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM));
        const int ntiles = (sa.E + TC_EB - 1) / TC_EB;
        const int grid = ntiles < c->num_sms ? ntiles : c->num_sms;
        if (grid > 0) {
          hex_tc_matrix_kernel<<<grid, TC_THREADS, TC_SMEM, c->stream>>>(ta);
          ++c->launches;
          OVS_CUDA_TRY(cudaGetLastError());
        }
      }
    } else {
      hex_element_kernel<T, KIND><<<(sa.E + 15) / 16, 128, KIND == OVS_ASM_TEM ? HexTemStage<T>::bytes : 0, c->stream>>>(sa);
      ++c->launches;
      OVS_CUDA_TRY(cudaGetLastError());
    }
  }
  if (!(parts & 2)) return OVS_OK;
  // most: the bytes for the longest row there is.  The limit belongs to the kernel,
  // whatever the context, so it is always that: no call lowers it under another
  // thread's launch
  auto launch = [&](auto kern, size_t smem, size_t most, auto... more) -> int {
    OVS_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    int per_sm = 0;
    OVS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, smem));
    if (per_sm < 1) return OVS_ERR_ARG;
    long need = ((long)c->N + 3) / 4;
    long grid = (long)per_sm * c->num_sms * 4;
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    kern<<<(int)grid, 128, smem, c->stream>>>(a, more...);
    ++c->launches;
    OVS_CUDA_TRY(cudaGetLastError());
    return OVS_OK;
  };
  if constexpr (KIND == OVS_ASM_NSVOF) {
    if (!tc) {
      const int carry = c->max_elem > HexRows<T>::EPC;
      return launch(hex_block_rows_kernel<T>, HexRows<T>::bytes(a.max_deg, carry) * 4,
                    HexRows<T>::bytes(OVS_MAX_DEG, true) * 4, carry);
    }
    if constexpr (can_tc)
      return launch(hex_rows_kernel<T, KIND, true>, HexSmem<T, KIND>::bytes(a.max_deg) * 4,
                    HexSmem<T, KIND>::bytes(OVS_MAX_DEG) * 4);
    return OVS_ERR_ARG;
  } else {
    return launch(hex_rows_kernel<T, KIND, false>, HexSmem<T, KIND>::bytes(a.max_deg) * 4,
                  HexSmem<T, KIND>::bytes(OVS_MAX_DEG) * 4);
  }
}
