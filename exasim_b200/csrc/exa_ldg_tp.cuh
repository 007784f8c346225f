// LDG residual of tensor-product elements (quadrilaterals and hexahedra whose shape tables are
// Kronecker products of the 1D ones) in two launches: the interior faces, then the elements.
// Included by exa_model.cu beside exa_ldg.cuh, whose kernels serve all other elements.
//
// Interpolation to the Gauss points and the weighted sums back run one dimension at a time: an
// element of N1^ND nodes costs O(ND N1^(ND + 1)) per field each way instead of O(N1^(2 ND)) (p = 3
// hexahedron: 768 against 4096 products to the points, 2304 against 16384 back with derivatives).
// The 1D tables are kernel parameters, so with every index fixed at compile time they come as
// constant operands of the FMAs.  What is left is HBM traffic: states, stage source, geometry and
// residual once each.  The Jacobian products by differences fold their linear combinations in.
// Measured (B200, 3D Euler, p = 3; before: dense products with the element tables, 7 launches):
// residual and norm on 20^3 359 -> 118 us; 150 GMRES steps on 12^3 23.5 -> 13.5 ms.
#pragma once
#include "exa_ldg.cuh"

template <int N1>
struct Tensor1D {
  double S[N1 * N1];   // S[g + N1 a]: nodal function a at Gauss point g
  double D[N1 * N1];   // its derivative
  double Sw[N1 * N1];  // S and D times the Gauss weight of g
  double Dw[N1 * N1];
};

template <int N1>
Tensor1D<N1> tensor_1d(const ExaTensor& T) {
  Tensor1D<N1> t;
  for (int a = 0; a < N1; ++a)
    for (int g = 0; g < N1; ++g) {
      t.S[g + N1 * a] = T.S[g + N1 * a];
      t.D[g + N1 * a] = T.D[g + N1 * a];
      t.Sw[g + N1 * a] = T.w[g] * T.S[g + N1 * a];
      t.Dw[g + N1 * a] = T.w[g] * T.D[g + N1 * a];
    }
  return t;
}

// what the residual is of and what becomes of it: u + eps v (v may be null), and
// out = cr R + c0 R0 (R0 may be null)
struct LdgState {
  const double *u, *v, *R0;
  double eps, cr, c0;
  __device__ double at(long long i) const { return v ? 1.0 * u[i] + eps * v[i] : u[i]; }
};

// index of point (i0, i1, i2) with rows padded to an odd length: pencils along every dimension
// then start in different banks (p = 3: none of the three passes conflicts)
template <int ND, int N1>
struct TpIdx {
  static constexpr int SY = N1 | 1, SZ = N1 * SY;
  static constexpr int NP = ND == 3 ? N1 * N1 * N1 : N1 * N1;
  static constexpr int NPAD = ND == 3 ? N1 * SZ : N1 * SY;
  static constexpr int NPEN = NP / N1;  // pencils per field
  __device__ static int point(int i) {
    if constexpr (ND == 3) return i % N1 + SY * ((i / N1) % N1) + SZ * (i / (N1 * N1));
    else return i % N1 + SY * (i / N1);
  }
  // first point of pencil q along dimension d
  __device__ static int pencil(int d, int q) {
    if constexpr (ND == 3) {
      const int x = q % N1, y = q / N1;
      return d == 0 ? SY * x + SZ * y : (d == 1 ? x + SZ * y : x + SY * y);
    } else {
      return d == 0 ? SY * q : q;
    }
  }
  __device__ static constexpr int stride(int d) { return d == 0 ? 1 : (d == 1 ? SY : SZ); }
};

// out[g] = sum_a T[g + N1 a] in[a]  (to the points), and the transpose (back to the nodes)
template <int N1>
__device__ __forceinline__ void tp_to_points(const double (&T)[N1 * N1], const double (&in)[N1], double (&out)[N1]) {
#pragma unroll
  for (int g = 0; g < N1; ++g) {
    double s = T[g] * in[0];
#pragma unroll
    for (int a = 1; a < N1; ++a) s = fma(T[g + N1 * a], in[a], s);
    out[g] = s;
  }
}
template <int N1>
__device__ __forceinline__ void tp_to_nodes(const double (&T)[N1 * N1], const double (&in)[N1], double (&out)[N1]) {
#pragma unroll
  for (int a = 0; a < N1; ++a) {
    double s = T[N1 * a] * in[0];
#pragma unroll
    for (int g = 1; g < N1; ++g) s = fma(T[g + N1 * a], in[g], s);
    out[a] = s;
  }
}

// Interior faces, FB per block: the states of both sides at the face nodes, to the Gauss points
// one dimension at a time, one thread per point for both fluxes and jac fhat, and back.  The
// arithmetic per point is that of ldg_face_inner_kernel.
constexpr int LTP_FT = 128;
template <int ND, int NCU, int N1>
constexpr int ltp_faces() {
  return ND == 3 ? (N1 >= 5 ? 8 : 16) : 32;
}
template <class Mdl, int ND, int NCU, int N1>
__global__ void __launch_bounds__(LTP_FT, 4)
    ldg_face_tp_kernel(LdgArgs A, LdgState U, int nfaces, const __grid_constant__ Tensor1D<N1> T) {
  constexpr int FD = ND - 1, NPF = FD == 2 ? N1 * N1 : N1, NPE = TpIdx<ND, N1>::NP;
  constexpr int SY = N1 | 1, PAD = FD == 2 ? N1 * SY : SY, NPEN = NPF / N1;
  constexpr int FB = ltp_faces<ND, NCU, N1>();
  __shared__ double s[FB][2][NCU][PAD];
  const ExaDims& P = A.P;
  const int f0 = blockIdx.x * FB, nf = min(FB, nfaces - f0), tid = threadIdx.x;
  auto pos = [](int a) { return FD == 2 ? a % N1 + SY * (a / N1) : a; };
  for (int t = tid; t < nf * 2 * NPF; t += LTP_FT) {
    const int a = t % NPF, sd = (t / NPF) % 2, j = t / (2 * NPF);
    const int k = A.fcon[2LL * (NPF * (long long)(f0 + j) + a) + sd];
    const long long o = (k % NPE) + (long long)NPE * NCU * (k / NPE);
#pragma unroll
    for (int c = 0; c < NCU; ++c) s[j][sd][c][pos(a)] = U.at(o + NPE * c);
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < FD; ++d) {
    for (int t = tid; t < nf * 2 * NCU * NPEN; t += LTP_FT) {
      const int q = t % NPEN;
      double* b = &s[0][0][0][0] + (t / NPEN) * PAD + (FD == 2 ? (d == 0 ? SY * q : q) : 0);
      const int st = d == 0 ? 1 : SY;
      double in[N1], out[N1];
#pragma unroll
      for (int a = 0; a < N1; ++a) in[a] = b[a * st];
      tp_to_points<N1>(T.S, in, out);
#pragma unroll
      for (int g = 0; g < N1; ++g) b[g * st] = out[g];
    }
    __syncthreads();
  }
  for (int t = tid; t < nf * NPF; t += LTP_FT) {
    const int g = t % NPF, j = t / NPF, f = f0 + j, p = pos(g);
    const int e1 = A.f2e[4 * f], l1 = A.f2e[4 * f + 1];
    const double* fg = A.faceg + ((long long)e1 * P.nfe + l1) * P.faceg_stride() + g;
    double x[ND], n[ND], u1[NCU], u2[NCU], f1[NCU * ND], f2[NCU * ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      x[d] = fg[NPF * d];
      n[d] = fg[NPF * (ND + d)];
    }
    const double jac = fg[NPF * 2 * ND];
#pragma unroll
    for (int c = 0; c < NCU; ++c) {
      u1[c] = s[j][0][c][p];
      u2[c] = s[j][1][c][p];
    }
#pragma unroll
    for (int q = 0; q < NCU * ND; ++q) f1[q] = f2[q] = 0.0;
    Mdl::flux_only(0, f1, x, u1, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NCU, NCU, ND, ND, P.nco,
                   P.ncw);
    Mdl::flux_only(0, f2, x, u2, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NCU, NCU, ND, ND, P.nco,
                   P.ncw);
#pragma unroll
    for (int k = 0; k < NCU; ++k) {
      double v = (0.5 * (f1[k] + f2[k])) * n[0];
#pragma unroll
      for (int d = 1; d < ND; ++d) v += (0.5 * (f1[k + NCU * d] + f2[k + NCU * d])) * n[d];
      if (A.ntau <= 1) {
        v += A.tau[0] * (u1[k] - u2[k]);
      } else if (A.ntau == NCU) {
        v += A.tau[k] * (u1[k] - u2[k]);
      } else {
#pragma unroll
        for (int i = 0; i < NCU; ++i) v += A.tau[i * NCU + k] * (u1[i] - u2[i]);
      }
      s[j][0][k][p] = v * jac;  // this thread alone reads and writes the point
    }
  }
  __syncthreads();
#pragma unroll
  for (int d = FD - 1; d >= 0; --d) {
    for (int t = tid; t < nf * NCU * NPEN; t += LTP_FT) {
      const int q = t % NPEN, k = (t / NPEN) % NCU, j = t / (NPEN * NCU);
      double* b = &s[j][0][k][FD == 2 ? (d == 0 ? SY * q : q) : 0];
      const int st = d == 0 ? 1 : SY;
      double in[N1], out[N1];
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = b[g * st];
      tp_to_nodes<N1>(T.Sw, in, out);
#pragma unroll
      for (int a = 0; a < N1; ++a) b[a * st] = out[a];
    }
    __syncthreads();
  }
  for (int t = tid; t < nf * NCU * NPF; t += LTP_FT) {
    const int a = t % NPF, k = (t / NPF) % NCU, j = t / (NPF * NCU);
    A.Rh[(long long)f0 * NPF * NCU + t] = s[j][0][k][pos(a)];
  }
}

// Elements, EB per block: states (and stage source) to the Gauss points, flux and source there,
// the weighted sums back, then minus or plus the face residuals of the element's faces and the
// sign and scaling of Residual.  Four arrays per element: the fields' values become, point by
// point, the source and the three flux components times the geometry.
template <int ND, int NCU, int N1>
constexpr int ltp_elems() {
  constexpr int tasks = TpIdx<ND, N1>::NPEN * NCU;
  return tasks >= 96 ? 1 : (tasks >= 64 ? 2 : 128 / tasks);
}
template <int ND, int NCU, int N1>
constexpr int ltp_threads() {
  return (TpIdx<ND, N1>::NPEN * NCU * ltp_elems<ND, NCU, N1>() + 31) / 32 * 32;
}
template <class Mdl, int ND, int NCU, int N1>
__global__ void __launch_bounds__(ltp_threads<ND, NCU, N1>())
    ldg_elem_tp_kernel(AsmArgs A, LdgState U, const int* nslot, const int* fslot, const double* Rh, double* out, int ne,
                       const __grid_constant__ Tensor1D<N1> T) {
  using X = TpIdx<ND, N1>;
  constexpr int NP = X::NP, PAD = X::NPAD, NPEN = X::NPEN, EB = ltp_elems<ND, NCU, N1>();
  constexpr int NT = ltp_threads<ND, NCU, N1>(), NA = ND + 1;
  extern __shared__ double lsm[];  // [EB][NA][NCU][PAD]
  const ExaDims& P = A.P;
  const int e0 = blockIdx.x * EB, nb = min(EB, ne - e0), tid = threadIdx.x;
  auto arr = [&](int j, int q, int k) { return lsm + ((j * NA + q) * NCU + k) * PAD; };
  for (int t = tid; t < nb * NCU * NP; t += NT) {
    const int i = t % NP, k = (t / NP) % NCU, j = t / (NP * NCU), p = X::point(i);
    const long long o = (long long)e0 * NP * NCU + t;
    arr(j, 0, k)[p] = U.at(o);
    if (A.tdep) arr(j, 1, k)[p] = A.sdg[o];
  }
  __syncthreads();
  const int nin = A.tdep ? 2 : 1;
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    for (int t = tid; t < nb * NCU * NPEN; t += NT) {
      const int q = t % NPEN, k = (t / NPEN) % NCU, j = t / (NPEN * NCU);
      for (int f = 0; f < nin; ++f) {
        double* b = arr(j, f, k) + X::pencil(d, q);
        double in[N1], o[N1];
#pragma unroll
        for (int a = 0; a < N1; ++a) in[a] = b[a * X::stride(d)];
        tp_to_points<N1>(T.S, in, o);
#pragma unroll
        for (int g = 0; g < N1; ++g) b[g * X::stride(d)] = o[g];
      }
    }
    __syncthreads();
  }
  for (int t = tid; t < nb * NP; t += NT) {
    const int g = t % NP, j = t / NP, p = X::point(g);
    const double* eg = A.elemg + (long long)(e0 + j) * P.elemg_stride() + g;
    const double* Xx = eg + NP * ND;
    double x[ND], u[NCU], s[NCU], f[NCU * ND], td[NCU];
#pragma unroll
    for (int c = 0; c < ND; ++c) x[c] = eg[NP * c];
#pragma unroll
    for (int k = 0; k < NCU; ++k) {
      u[k] = arr(j, 0, k)[p];
      s[k] = 0.0;
      td[k] = 1.0;
    }
#pragma unroll
    for (int q = 0; q < NCU * ND; ++q) f[q] = 0.0;
    if (!A.tdep || A.sourcefunc == 1)
      Mdl::source_only(0, s, x, u, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NCU, NCU, ND, ND, P.nco,
                       P.ncw);
    Mdl::flux_only(0, f, x, u, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NCU, NCU, ND, ND, P.nco,
                   P.ncw);
    if (A.tdep && A.tdfunc == 1)
      Mdl::tdfunc(0, td, x, u, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NCU, NCU, ND, ND, P.nco,
                  P.ncw);
    const double J = Xx[NP * ND * ND];
#pragma unroll
    for (int k = 0; k < NCU; ++k) {
      double sg = s[k];
      if (A.tdep) {
        double fv = 1.0 * arr(j, 1, k)[p] + (-A.dtfactor) * u[k];
        if (A.tdfunc == 1) fv = 1.0 * fv * td[k];
        sg = 1.0 * sg + 1.0 * fv;
      }
      arr(j, 0, k)[p] = sg * J;
    }
#pragma unroll
    for (int m = 0; m < ND; ++m) {
      double xr[ND];
#pragma unroll
      for (int c = 0; c < ND; ++c) xr[c] = Xx[NP * (c + ND * m)];
#pragma unroll
      for (int k = 0; k < NCU; ++k) {
        double v = f[k] * xr[0];
#pragma unroll
        for (int c = 1; c < ND; ++c) v += f[k + NCU * c] * xr[c];
        arr(j, 1 + m, k)[p] = v;
      }
    }
  }
  __syncthreads();
  // back: the pass along dimension d turns the source and the remaining flux components (0 .. d),
  // and adds component d through the derivative to the source
#pragma unroll
  for (int d = ND - 1; d >= 0; --d) {
    for (int t = tid; t < nb * NCU * NPEN; t += NT) {
      const int q = t % NPEN, k = (t / NPEN) % NCU, j = t / (NPEN * NCU);
      const int at = X::pencil(d, q);
      double in[N1], o[N1], der[N1];
      const double* bd = arr(j, 1 + d, k) + at;
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = bd[g * X::stride(d)];
      tp_to_nodes<N1>(T.Dw, in, der);
#pragma unroll
      for (int a = 0; a <= d; ++a) {  // array 0, then components 0 .. d - 1
        double* b = arr(j, a, k) + at;
#pragma unroll
        for (int g = 0; g < N1; ++g) in[g] = b[g * X::stride(d)];
        tp_to_nodes<N1>(T.Sw, in, o);
#pragma unroll
        for (int g = 0; g < N1; ++g) b[g * X::stride(d)] = a == 0 ? o[g] + der[g] : o[g];
      }
    }
    __syncthreads();
  }
  const double sc = 1.0 / A.dtfactor;
  for (int t = tid; t < nb * NCU * NP; t += NT) {
    const int i = t % NP, k = (t / NP) % NCU, j = t / (NP * NCU);
    double v = arr(j, 0, k)[X::point(i)];
    // the faces the node lies on, in the order of the element's faces; bit 31: second element
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      const int sl = nslot[ND * i + c];
      if (sl >= 0) {
        const unsigned w = (unsigned)fslot[(long long)(e0 + j) * P.ndf + sl];
        const double r = Rh[(long long)(w & 0x7fffffffu) + (long long)P.npf * k];
        v = (w >> 31) ? v + r : v - r;
      }
    }
    v = -1.0 * v;
    if (A.tdep) v = sc * v;
    const long long o = (long long)e0 * NP * NCU + t;
    out[o] = U.R0 ? U.cr * v + U.c0 * U.R0[o] : v;
  }
}

// Launches both for the model's (nd, ncu) and the elements' order; false when there is no instance.
// rc: EXA_OK or the error of a launch.
template <class Mdl>
bool launch_ldg_tp(const LdgArgs& F, const AsmArgs& A, const LdgState& U, const ExaTensor& T, const int* nslot,
                   const int* fslot, double* out, cudaStream_t st, int (*boundary)(void*), void* bctx, int* rc) {
  const ExaDims& P = A.P;
  *rc = EXA_OK;
  if (T.n1 == 0 || P.nc != P.ncu || P.ncx != P.nd) return false;
#define EXA_LTP(ND, NCU, N1)                                                                                     \
  if (P.nd == ND && P.ncu == NCU && T.n1 == N1) {                                                                \
    *rc = [&]() -> int {                                                                                         \
      const Tensor1D<N1> t1 = tensor_1d<N1>(T);                                                                  \
      constexpr int FB = ltp_faces<ND, NCU, N1>(), EB = ltp_elems<ND, NCU, N1>();                                \
      if (P.nf0 > 0) {                                                                                           \
        ldg_face_tp_kernel<Mdl, ND, NCU, N1><<<(P.nf0 + FB - 1) / FB, LTP_FT, 0, st>>>(F, U, P.nf0, t1);          \
        EXA_LAUNCH_CHECK();                                                                                      \
      }                                                                                                          \
      EXA_TRY(boundary(bctx));                                                                                   \
      const size_t sm = sizeof(double) * EB * (ND + 1) * NCU * TpIdx<ND, N1>::NPAD;                              \
      auto kern = ldg_elem_tp_kernel<Mdl, ND, NCU, N1>;                                                          \
      EXA_TRY(exa_allow_smem((const void*)kern, sm));                                                            \
      kern<<<(P.ne + EB - 1) / EB, ltp_threads<ND, NCU, N1>(), sm, st>>>(A, U, nslot, fslot, F.Rh, out, P.ne, t1); \
      EXA_LAUNCH_CHECK();                                                                                        \
      return EXA_OK;                                                                                             \
    }();                                                                                                         \
    return true;                                                                                                 \
  }
  // the pairs that a model of the package without q has; p = 2 and 3 (contexts refuse element blocks
  // above 320 x 320)
  EXA_LTP(3, 5, 3) EXA_LTP(3, 5, 4)
#undef EXA_LTP
  return false;
}
