// Volume blocks D and B of tensor-product elements by sum factorization: for each (k, c) pair,
//   M[i, j] = -sum_g (sum_d shapegw[i, g, d] rgJ[g, d, k, c]) shapegt[g, j]
// (vol_mat_kernel's sums), with the Gauss points contracted one dimension at a time: an element of
// N1^ND nodes costs about 2 N1^(2 ND + 1) products per pair instead of N1^(3 ND) (p = 4 hexahedron:
// 0.2 against 1.95 million), which leaves the FP64 units and the writes of the blocks about even.
// The last pass, most of the work, keeps its 1D tables as constant operands: one lane per
// combination of the upper indexes computes all N1 x N1 entries of the first dimension.
// Measured (B200; before: T factors and DMMA products): p = 4 convection-diffusion, 1331 hexahedra
// 1740 -> 289 us; p = 3 Euler, 1000 hexahedra 2690 -> 486 us (0.82 GB of blocks).  The mixed form keeps
// vol_mat_tc_kernel: B packed by this one took 1.6 ms on 4096 hexahedra, there 1.1 ms.
#pragma once
#include "exa_ldg_tp.cuh"

template <int N1>
struct TensorPair {
  double SS[N1 * N1 * N1], DS[N1 * N1 * N1];  // [g + N1 (i + N1 j)]: weight(g) S or D (g, i), times S(g, j)
};
template <int N1>
TensorPair<N1> tensor_pair(const ExaTensor& T) {
  TensorPair<N1> t;
  for (int j = 0; j < N1; ++j)
    for (int i = 0; i < N1; ++i)
      for (int g = 0; g < N1; ++g) {
        t.SS[g + N1 * (i + N1 * j)] = T.w[g] * T.S[g + N1 * i] * T.S[g + N1 * j];
        t.DS[g + N1 * (i + N1 * j)] = T.w[g] * T.D[g + N1 * i] * T.S[g + N1 * j];
      }
  return t;
}

constexpr int VTP_T = 256;
template <int ND, int N1>
struct VolTp {
  static constexpr int NP = ND == 3 ? N1 * N1 * N1 : N1 * N1, UP = NP / N1;  // UP: values of the upper indexes
  static constexpr int Q = N1 * N1, PR = ND == 3 ? Q * Q : Q;               // pairs (i, j) of one, of the upper dimensions
  static constexpr int LI = UP, GW = 32 / LI;                                // lanes per column group, groups per warp
  static constexpr int ST = N1 * NP;                                         // staged entries per column group
  static constexpr int kA = N1 * PR;                                         // A2, Y1: [g1][pair]
  static constexpr int kZ = ND == 3 ? 3 * N1 * N1 * Q : 0;                   // A, X1, X2: [g1 g2][pair of dim 3]
  static constexpr int doubles = 2 * kA + kZ + (ND + 1) * NP + 2 * Q * N1 + VTP_T / 32 * GW * ST;
};

// One block per (element, pair).
template <int ND, int N1>
__global__ void __launch_bounds__(VTP_T, 2)
    vol_blocks_tp_kernel(ExaDims P, int cfirst, const double* __restrict__ rgJ, double* __restrict__ D, double* __restrict__ B,
                         const __grid_constant__ TensorPair<N1> T) {
  using V = VolTp<ND, N1>;
  constexpr int NP = V::NP, Q = V::Q, PR = V::PR, LI = V::LI, GW = V::GW;
  extern __shared__ double vsm[];
  double* A2 = vsm;                       // [N1][PR]
  double* Y1 = A2 + V::kA;                // [N1][PR]
  double* Z = Y1 + V::kA;                 // [3][N1 N1][Q] (3D)
  double* R = Z + V::kZ;                  // [ND + 1][NP]
  double* tab = R + (ND + 1) * NP;        // SS, DS: [Q][N1] each
  double* stage = tab + 2 * Q * N1;       // [warps][GW][N1][NP]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int le = blockIdx.y, kc = blockIdx.x + P.ncu * cfirst, ncu = P.ncu, n = P.n;
  const int k = kc % ncu, c = kc / ncu;
  const double* Rg = rgJ + ((long long)le * ncu * P.nc + kc) * (ND + 1) * NP;
  for (int t = tid; t < (ND + 1) * NP; t += VTP_T) R[t] = Rg[t];
  for (int t = tid; t < Q * N1; t += VTP_T) {
    tab[t] = T.SS[t];
    tab[Q * N1 + t] = T.DS[t];
  }
  __syncthreads();
  const double *SS = tab, *DS = tab + Q * N1;
  // R: component d at the Gauss points, dimension 1 fastest; component 1 + r goes with the
  // derivative along dimension r
  if constexpr (ND == 3) {
    for (int t = tid; t < Q * Q; t += VTP_T) {  // (g1, g2) x pair of dimension 3
      const int g = t % Q, q = t / Q;
      double a = 0.0, x = 0.0, y = 0.0;
#pragma unroll
      for (int z = 0; z < N1; ++z) {
        const double s = SS[q * N1 + z], d = DS[q * N1 + z];
        a = fma(s, R[g + Q * z], fma(d, R[3 * NP + g + Q * z], a));
        x = fma(s, R[NP + g + Q * z], x);
        y = fma(s, R[2 * NP + g + Q * z], y);
      }
      Z[g + Q * q] = a;
      Z[Q * Q + g + Q * q] = x;
      Z[2 * Q * Q + g + Q * q] = y;
    }
    __syncthreads();
    // (g1, pair of dimension 3) pencils along g2; the pairs of dimension 2 are split over parts
    constexpr int PEN = N1 * Q, PARTS = VTP_T / PEN > 0 ? VTP_T / PEN : 1;
    for (int t = tid; t < PEN * PARTS; t += VTP_T) {
      const int pen = t % PEN, part = t / PEN, g1 = pen % N1, q3 = pen / N1;
      double a[N1], x[N1], y[N1];
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        const double* z = Z + g1 + N1 * g + Q * q3;
        a[g] = z[0];
        x[g] = z[Q * Q];
        y[g] = z[2 * Q * Q];
      }
      for (int q2 = part; q2 < Q; q2 += PARTS) {
        double s = 0.0, v = 0.0;
#pragma unroll
        for (int g = 0; g < N1; ++g) {
          const double w = SS[q2 * N1 + g];
          s = fma(w, a[g], fma(DS[q2 * N1 + g], y[g], s));
          v = fma(w, x[g], v);
        }
        A2[g1 * PR + q2 + Q * q3] = s;
        Y1[g1 * PR + q2 + Q * q3] = v;
      }
    }
  } else {
    for (int t = tid; t < N1 * Q; t += VTP_T) {  // g1 x pair of dimension 2
      const int g1 = t % N1, q = t / N1;
      double s = 0.0, v = 0.0;
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        const double w = SS[q * N1 + g];
        s = fma(w, R[g1 + N1 * g], fma(DS[q * N1 + g], R[2 * NP + g1 + N1 * g], s));
        v = fma(w, R[NP + g1 + N1 * g], v);
      }
      A2[g1 * PR + q] = s;
      Y1[g1 * PR + q] = v;
    }
  }
  __syncthreads();
  // the blocks' place: columns j of D (c < ncu) or of B's gradient component d of trace component nq
  const int qc = c - ncu, nq = c < ncu ? 0 : qc % ncu, d = c < ncu ? 0 : qc / ncu;
  double* out = c < ncu ? D + (long long)le * n * n + (long long)n * NP * c
                        : B + (long long)le * n * NP * P.nd * ncu + (long long)n * (NP * d + (long long)NP * P.nd * nq);
  out += NP * k;
  double* st = stage + warp * GW * V::ST;
  constexpr int GROUPS = V::UP;  // column groups: the upper indexes of j
  for (int g0 = warp * GW; g0 < GROUPS; g0 += VTP_T / 32 * GW) {
    const int sub = lane / LI, li = lane - sub * LI, gr = g0 + sub;
    if (sub < GW && gr < GROUPS) {
      // upper indexes (i2, i3) of this lane, (j2, j3) of its group
      const int pair = ND == 3 ? (li % N1 + N1 * (gr % N1)) + Q * (li / N1 + N1 * (gr / N1)) : li + N1 * gr;
      double a[N1], y[N1];
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        a[g] = A2[g * PR + pair];
        y[g] = Y1[g * PR + pair];
      }
#pragma unroll
      for (int j = 0; j < N1; ++j)
#pragma unroll
        for (int i = 0; i < N1; ++i) {
          double s = 0.0;
#pragma unroll
          for (int g = 0; g < N1; ++g) s = fma(T.SS[g + N1 * (i + N1 * j)], a[g], s);
#pragma unroll
          for (int g = 0; g < N1; ++g) s = fma(T.DS[g + N1 * (i + N1 * j)], y[g], s);
          st[sub * V::ST + j * NP + i + N1 * li] = -s;
        }
    }
    __syncwarp();
    const int ng = min(GW, GROUPS - g0);  // groups g0 .. g0 + ng - 1 are consecutive columns
    for (int t = lane; t < ng * V::ST; t += 32) {
      const int i = t % NP, j = t / NP;
      out[i + (long long)n * (N1 * g0 + j)] = st[t];
    }
    __syncwarp();
  }
}

// Launches it for the pairs of fields c0 .. c1 - 1 where the element's order has an instance; *rc: EXA_OK or the launch's error
inline bool launch_vol_blocks_tp(const ExaDims& P, const ExaTensor& T, const double* rgJ, double* D, double* B, int c0,
                                 int c1, int nb, cudaStream_t st, int* rc) {
#define EXA_VTP(ND, N1)                                                                     \
  if (P.nd == ND && T.n1 == N1) {                                                           \
    *rc = [&]() -> int {                                                                    \
      const size_t sm = sizeof(double) * VolTp<ND, N1>::doubles;                            \
      auto kern = vol_blocks_tp_kernel<ND, N1>;                                             \
      EXA_TRY(exa_allow_smem((const void*)kern, sm));                                       \
      kern<<<dim3(P.ncu * (c1 - c0), nb), VTP_T, sm, st>>>(P, c0, rgJ, D, B, tensor_pair<N1>(T)); \
      EXA_LAUNCH_CHECK();                                                                   \
      return EXA_OK;                                                                        \
    }();                                                                                    \
    return true;                                                                            \
  }
  EXA_VTP(3, 3) EXA_VTP(3, 4) EXA_VTP(3, 5) EXA_VTP(2, 3) EXA_VTP(2, 4) EXA_VTP(2, 5)
#undef EXA_VTP
  return false;
}
