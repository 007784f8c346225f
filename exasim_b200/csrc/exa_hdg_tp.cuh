// HDG residual and q recovery of tensor-product elements, one launch each (besides the trace
// scatter): volume and face integrals one dimension at a time (exa_ldg_tp.cuh), everything of an
// element in shared memory between its states and its results.
//
// q = M^-1 (C u - E uhat): with as many Gauss points as nodes per dimension the quadrature mass
// matrix is M = Phi^T diag(w jac) Phi with a square Phi = S x S (x S), so M^-1 is applied by the 1D
// inverse of S and a division at the Gauss points; no element matrix is read (p = 4 hexahedra read
// 125 KB of M^-1 per element through getq_mf_kernel, 20 KB in all here).
//
// Bound: launches and latency on small meshes, shared-memory passes and the states and geometry from
// HBM on large ones.  Measured (B200, q recovery, residual and norm; before: 5 GEMMs and 6 kernels):
// 2D Navier-Stokes, 33 x 33, p = 3: 140 -> 72 us; 3D convection-diffusion, 5^3 to 15^3, p = 2 to 4:
// 2.0 to 2.9 times; a 16^3 stage solve of the mixed form (three of each) 14.8 -> 13.5 ms.
#pragma once
#include "exa_ldg_tp.cuh"

template <int N1>
struct TensorInv {
  double Si[N1 * N1];  // Si[a + N1 g]: the inverse of S[g + N1 a]
  double w[N1];
};
template <int N1>
TensorInv<N1> tensor_inv(const ExaTensor& T) {
  TensorInv<N1> t;
  long double A[N1][2 * N1];
  for (int g = 0; g < N1; ++g)
    for (int a = 0; a < N1; ++a) {
      A[g][a] = T.S[g + N1 * a];
      A[g][N1 + a] = g == a ? 1.0L : 0.0L;
    }
  for (int k = 0; k < N1; ++k) {  // Gauss-Jordan with row pivoting
    int p = k;
    for (int r = k + 1; r < N1; ++r)
      if (fabsl(A[r][k]) > fabsl(A[p][k])) p = r;
    for (int c = 0; c < 2 * N1; ++c) std::swap(A[k][c], A[p][c]);
    const long double d = 1.0L / A[k][k];
    for (int c = 0; c < 2 * N1; ++c) A[k][c] *= d;
    for (int r = 0; r < N1; ++r) {
      if (r == k) continue;
      const long double f = A[r][k];
      for (int c = 0; c < 2 * N1; ++c) A[r][c] -= f * A[k][c];
    }
  }
  for (int a = 0; a < N1; ++a)
    for (int g = 0; g < N1; ++g) t.Si[a + N1 * g] = (double)A[a][N1 + g];
  for (int g = 0; g < N1; ++g) t.w[g] = T.w[g];
  return t;
}

// sizes of the element kernels: NF fields per element, elements per block, threads
template <int ND, int N1>
struct HtpSize {
  using X = TpIdx<ND, N1>;
  static constexpr int FD = ND - 1, NPF = X::NP / N1, NFE = 2 * ND;
  static constexpr int FY = N1 | 1, FPAD = FD == 2 ? N1 * FY : FY, FPEN = NPF / N1;
  __device__ static int fpos(int a) { return FD == 2 ? a % N1 + FY * (a / N1) : a; }
  // pencil q along dimension d of a face
  __device__ static int fpencil(int d, int q) { return FD == 2 ? (d == 0 ? FY * q : q) : 0; }
  __device__ static int fstride(int d) { return d == 0 ? 1 : FY; }
  static constexpr int eb(int fields) {
    const int tasks = X::NPEN * fields;
    return tasks >= 96 ? 1 : (tasks >= 64 ? 2 : (128 / tasks > 8 ? 8 : 128 / tasks));
  }
  static constexpr int threads(int fields) {
    const int t = (X::NPEN * fields * eb(fields) + 31) / 32 * 32;
    return t > 256 ? 256 : t;
  }
};

// one pass of a set of arrays: dst_pencil[out] = T in, arrays [count] PAD apart from base
template <int N1, bool BACK>
__device__ __forceinline__ void tp_line(double* b, int st, const double (&T)[N1 * N1]) {
  double in[N1], out[N1];
#pragma unroll
  for (int a = 0; a < N1; ++a) in[a] = b[a * st];
  if (BACK) tp_to_nodes<N1>(T, in, out);
  else tp_to_points<N1>(T, in, out);
#pragma unroll
  for (int a = 0; a < N1; ++a) b[a * st] = out[a];
}

// Ru (volume minus face terms) and Rh of each element (RuEquationElemBlock / ElemFaceBlock without
// Jacobians, uequation.cpp:790-1077); the arithmetic per point is vol_pointwise_kernel's and
// face_kernel<Mdl, false>'s.
template <int ND, int NCU, int NC, int N1>
struct HdgTp {
  using Z = HtpSize<ND, N1>;
  static constexpr int NV = NC + NCU > (ND + 1) * NCU ? NC + NCU : (ND + 1) * NCU;  // volume arrays
  static constexpr int EB = Z::eb(NC), NT = Z::threads(NC);
  static constexpr int vol = NV * Z::X::NPAD, face = Z::NFE * (NC + NCU) * Z::FPAD;
  static constexpr size_t smem = sizeof(double) * EB * (vol + face);
};
template <class Mdl, int ND, int NCU, int NC, int N1>
__global__ void __launch_bounds__((HdgTp<ND, NCU, NC, N1>::NT))
    hdg_resid_tp_kernel(AsmArgs A, const int* nslot, double* Ru, double* Rh, int ne,
                        const __grid_constant__ Tensor1D<N1> T) {
  using H = HdgTp<ND, NCU, NC, N1>;
  using Z = HtpSize<ND, N1>;
  using X = TpIdx<ND, N1>;
  constexpr int NP = X::NP, PAD = X::NPAD, NPEN = X::NPEN, EB = H::EB, NT = H::NT, NPF = Z::NPF, NFE = Z::NFE;
  constexpr int NFA = NC + NCU;  // arrays per face: u, q, then uhat
  extern __shared__ double hsm[];
  const ExaDims& P = A.P;
  const int e0 = blockIdx.x * EB, nb = min(EB, ne - e0), tid = threadIdx.x;
  auto arr = [&](int j, int q) { return hsm + (j * H::NV + q) * PAD; };
  double* fsm = hsm + EB * H::vol;
  auto farr = [&](int j, int l, int q) { return fsm + ((j * NFE + l) * NFA + q) * Z::FPAD; };
  // states, stage source, face traces
  for (int t = tid; t < nb * NC * NP; t += NT) {
    const int i = t % NP, c = (t / NP) % NC, j = t / (NP * NC);
    arr(j, c)[X::point(i)] = A.udg[(long long)e0 * NP * NC + t];
  }
  if (A.tdep)
    for (int t = tid; t < nb * NCU * NP; t += NT) {
      const int i = t % NP, k = (t / NP) % NCU, j = t / (NP * NCU);
      arr(j, NC + k)[X::point(i)] = A.sdg[(long long)e0 * NP * NCU + t];
    }
  for (int t = tid; t < nb * NFE * NPF; t += NT) {
    const int a = t % NPF, l = (t / NPF) % NFE, j = t / (NPF * NFE), e = e0 + j;
    const int node = A.perm[a + NPF * l], pos = Z::fpos(a);
    const double* U = A.udg + (long long)e * NP * NC + node;
#pragma unroll
    for (int c = 0; c < NC; ++c) farr(j, l, c)[pos] = U[NP * c];
    const double* uh = A.uh + NCU * (long long)A.elemcon[a + NPF * l + P.ndf * e];
#pragma unroll
    for (int k = 0; k < NCU; ++k) farr(j, l, NC + k)[pos] = uh[k];
  }
  __syncthreads();
  // to the Gauss points of the element and of its faces
  const int nin = NC + (A.tdep ? NCU : 0);
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    for (int t = tid; t < nb * nin * NPEN; t += NT) {
      const int q = t % NPEN, c = (t / NPEN) % nin, j = t / (NPEN * nin);
      tp_line<N1, false>(arr(j, c) + X::pencil(d, q), X::stride(d), T.S);
    }
    if (d < ND - 1)
      for (int t = tid; t < nb * NFE * NFA * Z::FPEN; t += NT) {
        const int q = t % Z::FPEN;
        tp_line<N1, false>(fsm + (t / Z::FPEN) * Z::FPAD + Z::fpencil(d, q), Z::fstride(d), T.S);
      }
    __syncthreads();
  }
  // volume points: source and flux times the geometry, in place
  for (int t = tid; t < nb * NP; t += NT) {
    const int g = t % NP, j = t / NP, p = X::point(g);
    const double* eg = A.elemg + (long long)(e0 + j) * P.elemg_stride() + g;
    const double* Xx = eg + NP * ND;
    double x[ND], u[NC], s[NCU], f[NCU * ND], td[NCU], sd[NCU];
#pragma unroll
    for (int c = 0; c < ND; ++c) x[c] = eg[NP * c];
#pragma unroll
    for (int c = 0; c < NC; ++c) u[c] = arr(j, c)[p];
#pragma unroll
    for (int k = 0; k < NCU; ++k) {
      s[k] = 0.0;
      td[k] = 1.0;
      sd[k] = A.tdep ? arr(j, NC + k)[p] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < NCU * ND; ++q) f[q] = 0.0;
    if (!A.tdep || A.sourcefunc == 1)
      Mdl::source_only(0, s, x, u, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NC, NCU, ND, ND, P.nco,
                       P.ncw);
    Mdl::flux_only(0, f, x, u, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NC, NCU, ND, ND, P.nco,
                   P.ncw);
    if (A.tdep && A.tdfunc == 1)
      Mdl::tdfunc(0, td, x, u, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NC, NCU, ND, ND, P.nco,
                  P.ncw);
    const double J = Xx[NP * ND * ND];
#pragma unroll
    for (int k = 0; k < NCU; ++k) {
      double sg = s[k];
      if (A.tdep) {
        double fv = 1.0 * sd[k] + (-A.dtfactor) * u[k];
        if (A.tdfunc == 1) fv = 1.0 * fv * td[k];
        sg = 1.0 * sg + 1.0 * fv;
      }
      arr(j, k)[p] = sg * J;
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
        arr(j, (1 + m) * NCU + k)[p] = v;
      }
    }
  }
  // face points: fhat into the u arrays, the trace equation's flux into the uhat arrays
  const double tau0 = A.tau[0];
  for (int t = tid; t < nb * NFE * NPF; t += NT) {
    const int g = t % NPF, l = (t / NPF) % NFE, j = t / (NPF * NFE), e = e0 + j, p = Z::fpos(g);
    const double* fg = A.faceg + ((long long)e * NFE + l) * P.faceg_stride() + g;
    double x[ND], n[ND], u[NC], uq[NC], uh[NCU], f[NCU * ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      x[d] = fg[NPF * d];
      n[d] = fg[NPF * (ND + d)];
    }
    const double jac = fg[NPF * 2 * ND];
#pragma unroll
    for (int c = 0; c < NC; ++c) u[c] = uq[c] = farr(j, l, c)[p];
#pragma unroll
    for (int k = 0; k < NCU; ++k) uh[k] = uq[k] = farr(j, l, NC + k)[p];
#pragma unroll
    for (int q = 0; q < NCU * ND; ++q) f[q] = 0.0;
    Mdl::flux_only(0, f, x, uq, nullptr, nullptr, A.uinf, A.param, A.time, A.modelnumber, 1, NC, NCU, ND, ND, P.nco,
                   P.ncw);
    const int ib = A.bf[l + NFE * e];
    double fb[NCU];
#pragma unroll
    for (int k = 0; k < NCU; ++k) fb[k] = 0.0;
    if (ib > 0)
      Mdl::fbou_only(0, fb, x, u, nullptr, nullptr, uh, n, A.tau, A.uinf, A.param, A.time, A.modelnumber, ib, 1, NC, NCU,
                     ND, ND, P.nco, P.ncw);
#pragma unroll
    for (int k = 0; k < NCU; ++k) {
      double v = f[k] * n[0];
#pragma unroll
      for (int d = 1; d < ND; ++d) v += f[k + NCU * d] * n[d];
      v += tau0 * (u[k] - uh[k]);
      v *= jac;
      farr(j, l, k)[p] = v;
      farr(j, l, NC + k)[p] = ib > 0 ? fb[k] * jac : v;
    }
  }
  __syncthreads();
  // back to the nodes
#pragma unroll
  for (int d = ND - 1; d >= 0; --d) {
    for (int t = tid; t < nb * NCU * NPEN; t += NT) {
      const int q = t % NPEN, k = (t / NPEN) % NCU, j = t / (NPEN * NCU), at = X::pencil(d, q), st = X::stride(d);
      double in[N1], der[N1], o[N1];
      const double* bd = arr(j, (1 + d) * NCU + k) + at;
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = bd[g * st];
      tp_to_nodes<N1>(T.Dw, in, der);
      double* b = arr(j, k) + at;
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = b[g * st];
      tp_to_nodes<N1>(T.Sw, in, o);
#pragma unroll
      for (int g = 0; g < N1; ++g) b[g * st] = o[g] + der[g];
#pragma unroll
      for (int m = 0; m < d; ++m) tp_line<N1, true>(arr(j, (1 + m) * NCU + k) + at, st, T.Sw);
    }
    if (d < ND - 1)
      for (int t = tid; t < nb * NFE * 2 * NCU * Z::FPEN; t += NT) {
        const int q = t % Z::FPEN, r = t / Z::FPEN, k = r % (2 * NCU), l = (r / (2 * NCU)) % NFE, j = r / (2 * NCU * NFE);
        tp_line<N1, true>(farr(j, l, k < NCU ? k : NC + k - NCU) + Z::fpencil(d, q), Z::fstride(d), T.Sw);
      }
    __syncthreads();
  }
  for (int t = tid; t < nb * NCU * NP; t += NT) {
    const int i = t % NP, k = (t / NP) % NCU, j = t / (NP * NCU);
    double v = arr(j, k)[X::point(i)];
#pragma unroll
    for (int c = 0; c < ND; ++c) {  // the faces the node lies on, in order
      const int sl = nslot[ND * i + c];
      if (sl >= 0) v -= farr(j, sl / NPF, k)[Z::fpos(sl % NPF)];
    }
    Ru[(long long)e0 * NP * NCU + t] = v;
  }
  for (int t = tid; t < nb * NFE * NPF * NCU; t += NT) {
    const int k = t % NCU, a = (t / NCU) % NPF, l = (t / (NCU * NPF)) % NFE, j = t / (NCU * NPF * NFE);
    Rh[(long long)e0 * NFE * NPF * NCU + t] = -farr(j, l, NC + k)[Z::fpos(a)];
  }
}

// q from u and uhat (hdgGetQ, qequation.cpp:372-484)
template <int ND, int NCU, int N1>
struct GetqTp {
  using Z = HtpSize<ND, N1>;
  static constexpr int NV = ND * ND * NCU;  // arrays: component r of the moment of q_d, [k][d][r]
  static constexpr int EB = Z::eb(NCU * ND), NT = Z::threads(NCU * ND);
  static constexpr int vol = NV * Z::X::NPAD, face = Z::NFE * NCU * ND * Z::FPAD;
  static constexpr size_t smem = sizeof(double) * EB * (vol + face);
};
template <int ND, int NCU, int N1>
__global__ void __launch_bounds__((GetqTp<ND, NCU, N1>::NT))
    getq_tp_kernel(ExaDims P, const int* nslot, const int* perm, const int* elemcon, const double* elemg,
                   const double* faceg, const double* uh, double* udg, int ne, const __grid_constant__ Tensor1D<N1> T,
                   const __grid_constant__ TensorInv<N1> TI) {
  using H = GetqTp<ND, NCU, N1>;
  using Z = HtpSize<ND, N1>;
  using X = TpIdx<ND, N1>;
  constexpr int NP = X::NP, PAD = X::NPAD, NPEN = X::NPEN, EB = H::EB, NT = H::NT, NPF = Z::NPF, NFE = Z::NFE;
  constexpr int NC = NCU * (ND + 1), L = ND - 1;
  extern __shared__ double hsm[];
  const int e0 = blockIdx.x * EB, nb = min(EB, ne - e0), tid = threadIdx.x;
  auto arr = [&](int j, int k, int d, int r) { return hsm + (((j * NCU + k) * ND + d) * ND + r) * PAD; };
  double* fsm = hsm + EB * H::vol;
  auto farr = [&](int j, int l, int k, int d) { return fsm + (((j * NFE + l) * NCU + k) * ND + d) * Z::FPAD; };
  // u in the arrays (k, 0, 0), uhat in the face arrays (k, 0)
  for (int t = tid; t < nb * NCU * NP; t += NT) {
    const int i = t % NP, k = (t / NP) % NCU, j = t / (NP * NCU);
    arr(j, k, 0, 0)[X::point(i)] = udg[(long long)(e0 + j) * NP * NC + i + NP * k];
  }
  for (int t = tid; t < nb * NFE * NPF; t += NT) {
    const int a = t % NPF, l = (t / NPF) % NFE, j = t / (NPF * NFE);
    const double* h = uh + NCU * (long long)elemcon[a + NPF * l + P.ndf * (e0 + j)];
#pragma unroll
    for (int k = 0; k < NCU; ++k) farr(j, l, k, 0)[Z::fpos(a)] = h[k];
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < ND; ++d) {
    for (int t = tid; t < nb * NCU * NPEN; t += NT) {
      const int q = t % NPEN, k = (t / NPEN) % NCU, j = t / (NPEN * NCU);
      tp_line<N1, false>(arr(j, k, 0, 0) + X::pencil(d, q), X::stride(d), T.S);
    }
    if (d < ND - 1)
      for (int t = tid; t < nb * NFE * NCU * Z::FPEN; t += NT) {
        const int q = t % Z::FPEN, r = t / Z::FPEN, k = r % NCU, l = (r / NCU) % NFE, j = r / (NCU * NFE);
        tp_line<N1, false>(farr(j, l, k, 0) + Z::fpencil(d, q), Z::fstride(d), T.S);
      }
    __syncthreads();
  }
  for (int t = tid; t < nb * NP; t += NT) {
    const int g = t % NP, j = t / NP, p = X::point(g);
    const double* Xx = elemg + (long long)(e0 + j) * P.elemg_stride() + NP * ND + g;
    double u[NCU];
#pragma unroll
    for (int k = 0; k < NCU; ++k) u[k] = arr(j, k, 0, 0)[p];
#pragma unroll
    for (int r = 0; r < ND; ++r)
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        const double x = Xx[NP * (d + ND * r)];
#pragma unroll
        for (int k = 0; k < NCU; ++k) arr(j, k, d, r)[p] = x * u[k];
      }
  }
  for (int t = tid; t < nb * NFE * NPF; t += NT) {
    const int g = t % NPF, l = (t / NPF) % NFE, j = t / (NPF * NFE), p = Z::fpos(g);
    const double* fg = faceg + ((long long)(e0 + j) * NFE + l) * P.faceg_stride() + g;
    const double jac = fg[NPF * 2 * ND];
    double h[NCU];
#pragma unroll
    for (int k = 0; k < NCU; ++k) h[k] = farr(j, l, k, 0)[p];
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const double nj = fg[NPF * (ND + d)] * jac;
#pragma unroll
      for (int k = 0; k < NCU; ++k) farr(j, l, k, d)[p] = nj * h[k];
    }
  }
  __syncthreads();
  // back: component r through the derivative along dimension r, summed into component L = ND - 1
#pragma unroll
  for (int m = ND - 1; m >= 0; --m) {
    for (int t = tid; t < nb * NCU * ND * NPEN; t += NT) {
      const int q = t % NPEN, kd = (t / NPEN) % (NCU * ND), j = t / (NPEN * NCU * ND), at = X::pencil(m, q);
      const int st = X::stride(m);
      double* b = hsm + ((j * NCU * ND + kd) * ND) * PAD + at;  // component 0 of (k, d)
      double in[N1], der[N1], o[N1];
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = b[m * PAD + g * st];
      tp_to_nodes<N1>(T.Dw, in, der);
      if (m < L) {
#pragma unroll
        for (int g = 0; g < N1; ++g) in[g] = b[L * PAD + g * st];
        tp_to_nodes<N1>(T.Sw, in, o);
#pragma unroll
        for (int g = 0; g < N1; ++g) der[g] += o[g];
      }
#pragma unroll
      for (int g = 0; g < N1; ++g) b[L * PAD + g * st] = der[g];
#pragma unroll
      for (int r = 0; r < m; ++r) tp_line<N1, true>(b + r * PAD, st, T.Sw);
    }
    if (m < ND - 1)
      for (int t = tid; t < nb * NFE * NCU * ND * Z::FPEN; t += NT) {
        const int q = t % Z::FPEN;
        tp_line<N1, true>(fsm + (t / Z::FPEN) * Z::FPAD + Z::fpencil(m, q), Z::fstride(m), T.Sw);
      }
    __syncthreads();
  }
  // minus the face terms, in the order of the faces
  for (int t = tid; t < nb * NCU * ND * NP; t += NT) {
    const int i = t % NP, kd = (t / NP) % (NCU * ND), j = t / (NP * NCU * ND), d = kd % ND, k = kd / ND;
    double v = arr(j, k, d, L)[X::point(i)];
#pragma unroll
    for (int c = 0; c < ND; ++c) {
      const int sl = nslot[ND * i + c];
      if (sl >= 0) v -= farr(j, sl / NPF, k, d)[Z::fpos(sl % NPF)];
    }
    arr(j, k, d, L)[X::point(i)] = v;
  }
  __syncthreads();
  // M^-1: S^-T along every dimension, 1 / (w jac) at the points, S^-1 along every dimension
#pragma unroll
  for (int m = 0; m < 2 * ND; ++m) {
    const bool back = m >= ND;
    const int dim = back ? m - ND : m;
    for (int t = tid; t < nb * NCU * ND * NPEN; t += NT) {
      const int q = t % NPEN, kd = (t / NPEN) % (NCU * ND), j = t / (NPEN * NCU * ND);
      double* b = hsm + ((j * NCU * ND + kd) * ND + L) * PAD + X::pencil(dim, q);
      // to_nodes sums over the first index of the table: Si[a + N1 g] over a; to_points over g
      if (back) tp_line<N1, false>(b, X::stride(dim), TI.Si);
      else tp_line<N1, true>(b, X::stride(dim), TI.Si);
    }
    __syncthreads();
    if (m == ND - 1) {
      for (int t = tid; t < nb * NP; t += NT) {
        const int g = t % NP, j = t / NP, p = X::point(g);
        const double J = elemg[(long long)(e0 + j) * P.elemg_stride() + NP * (ND + ND * ND) + g];
        double w = TI.w[g % N1] * TI.w[(g / N1) % N1];
        if (ND == 3) w *= TI.w[g / (N1 * N1)];
        const double s = 1.0 / (w * J);
#pragma unroll
        for (int kd = 0; kd < NCU * ND; ++kd) hsm[((j * NCU * ND + kd) * ND + L) * PAD + p] *= s;
      }
      __syncthreads();
    }
  }
  for (int t = tid; t < nb * NCU * ND * NP; t += NT) {
    const int i = t % NP, d = (t / NP) % ND, k = (t / (NP * ND)) % NCU, j = t / (NP * ND * NCU);
    udg[(long long)(e0 + j) * NP * NC + i + NP * (NCU + k + NCU * d)] = arr(j, k, d, L)[X::point(i)];
  }
}

// the (nd, ncu) pairs of the package's models and p = 2 to 4; false: no instance
template <class Mdl>
bool launch_hdg_resid_tp(const AsmArgs& A, const ExaTensor& T, const int* nslot, double* Ru, double* Rh, cudaStream_t st,
                         int* rc) {
  const ExaDims& P = A.P;
#define EXA_HTP(ND, NCU, NC, N1)                                                                        \
  if (P.nd == ND && P.ncu == NCU && P.nc == NC && T.n1 == N1 && P.nfe == 2 * ND) {                      \
    *rc = [&]() -> int {                                                                                \
      using H = HdgTp<ND, NCU, NC, N1>;                                                                 \
      auto kern = hdg_resid_tp_kernel<Mdl, ND, NCU, NC, N1>;                                            \
      EXA_TRY(exa_allow_smem((const void*)kern, H::smem));                                              \
      kern<<<(P.ne + H::EB - 1) / H::EB, H::NT, H::smem, st>>>(A, nslot, Ru, Rh, P.ne, tensor_1d<N1>(T)); \
      EXA_LAUNCH_CHECK();                                                                               \
      return EXA_OK;                                                                                    \
    }();                                                                                                \
    return true;                                                                                        \
  }
#define EXA_HTP3(ND, NCU, NC) EXA_HTP(ND, NCU, NC, 3) EXA_HTP(ND, NCU, NC, 4) EXA_HTP(ND, NCU, NC, 5)
  EXA_HTP3(2, 1, 3) EXA_HTP3(3, 1, 4) EXA_HTP3(2, 4, 12) EXA_HTP(3, 5, 5, 3) EXA_HTP(3, 5, 5, 4)
#undef EXA_HTP3
#undef EXA_HTP
  return false;
}

// the pairs and orders of launch_getq_tp
inline bool getq_tp_fits(const ExaDims& P, const ExaTensor& T) {
  const bool pair = P.nd == 2 ? P.ncu == 1 || P.ncu == 4 : P.nd == 3 && P.ncu == 1;
  return pair && P.nfe == 2 * P.nd && T.n1 >= 3 && T.n1 <= 5;
}
inline bool launch_getq_tp(const ExaDims& P, const ExaTensor& T, const int* nslot, const int* perm, const int* elemcon,
                           const double* elemg, const double* faceg, const double* uh, double* udg, cudaStream_t st,
                           int* rc) {
#define EXA_QTP(ND, NCU, N1)                                                                                     \
  if (P.nd == ND && P.ncu == NCU && T.n1 == N1 && P.nfe == 2 * ND) {                                             \
    *rc = [&]() -> int {                                                                                         \
      using H = GetqTp<ND, NCU, N1>;                                                                             \
      auto kern = getq_tp_kernel<ND, NCU, N1>;                                                                   \
      EXA_TRY(exa_allow_smem((const void*)kern, H::smem));                                                       \
      kern<<<(P.ne + H::EB - 1) / H::EB, H::NT, H::smem, st>>>(P, nslot, perm, elemcon, elemg, faceg, uh, udg, P.ne, \
                                                               tensor_1d<N1>(T), tensor_inv<N1>(T));             \
      EXA_LAUNCH_CHECK();                                                                                        \
      return EXA_OK;                                                                                             \
    }();                                                                                                         \
    return true;                                                                                                 \
  }
#define EXA_QTP3(ND, NCU) EXA_QTP(ND, NCU, 3) EXA_QTP(ND, NCU, 4) EXA_QTP(ND, NCU, 5)
  EXA_QTP3(2, 1) EXA_QTP3(3, 1) EXA_QTP3(2, 4)
#undef EXA_QTP3
#undef EXA_QTP
  return false;
}
