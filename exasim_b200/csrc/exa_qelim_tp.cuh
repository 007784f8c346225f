// The q elimination of scalar models on tensor-product hexahedra without B and G: the columns of
//   D += B MinvC, F -= B MinvE, K += G MinvC, H -= G MinvE
// are the derivative of the element residual with respect to q (volume integrals and the face terms
// of the u rows: B; the trace rows: G) applied to the columns of MinvC and MinvE, and that derivative
// is applied by sum factorization at the stored Jacobians of the Gauss points (uequation.cpp:45-557
// forms B and G, :559-775 multiplies them).
//
// A p = 4 hexahedron takes 19 thousand products per column this way and 275 columns, 5.1 million,
// against 28.4 million of the dense products, and neither B and G (825 KB) nor the passes that write
// them.  Bound: the instructions around the products (shared-memory passes and their addresses: FP64
// units active a quarter of the time).  Measured (B200, 1331 hexahedra, p = 4; before: DMMA products):
// 4.6 ms with the passes that write B and G -> 2.24 ms, whole assembly 7.37 -> 4.97 ms.  The mixed
// form keeps its tensor-core products into D and F (the four took 3.0 ms on 4096 hexahedra, this kernel
// 6.5) and has a kernel of its own for the trace rows.
#pragma once
#include "exa_hdg_tp.cuh"
#include "exa_tc.cuh"
#include "exa_umma.cuh"
#include "exa_vol_tp.cuh"

// Whole planes in registers: a thread takes both in-plane dimensions of a field's plane or of a face
// field at once, and the third dimension there and back around the Gauss points.  The next group's
// columns are copied in while this one is worked on.
template <int N1>
struct Qelim3 {
  static constexpr int NP = N1 * N1 * N1, NPF = N1 * N1, SY = N1 | 1, SZ = N1 * SY, PAD = N1 * SZ, FPAD = N1 * SY;
  static constexpr int VS = (3 * PAD) | 1, FS = (18 * FPAD) | 1;  // per column: nodal (and worked) fields, face fields
  static constexpr int fit = (int)(73000 / (sizeof(double) * (2 * VS + FS)));
  static constexpr int CB = fit > 16 ? 16 : fit;
  static constexpr int NT = 256;
  static constexpr size_t smem = sizeof(double) * CB * (2 * VS + FS);
};
// both dimensions of a plane
template <int N1, bool BACK>
__device__ __forceinline__ void tp_plane(double (&a)[N1][N1], const double (&T)[N1 * N1]) {
#pragma unroll
  for (int y = 0; y < N1; ++y) {
    double o[N1];
    if (BACK) tp_to_nodes<N1>(T, a[y], o);
    else tp_to_points<N1>(T, a[y], o);
#pragma unroll
    for (int x = 0; x < N1; ++x) a[y][x] = o[x];
  }
#pragma unroll
  for (int x = 0; x < N1; ++x) {
    double in[N1], o[N1];
#pragma unroll
    for (int y = 0; y < N1; ++y) in[y] = a[y][x];
    if (BACK) tp_to_nodes<N1>(T, in, o);
    else tp_to_points<N1>(T, in, o);
#pragma unroll
    for (int y = 0; y < N1; ++y) a[y][x] = o[y];
  }
}
// rgJ: volume Jacobian integrands of the chunk; Fq: derivatives of the face fluxes with respect to q
// per element and face [ngf, 3] of the u rows, then of the trace rows.  D, F, K and H hold the volume
// and face terms of the u and uhat columns: D everywhere, F, K and H at the entries that couple a face
// with its own nodes, the only ones read; all are assigned.
template <int N1>
__global__ void __launch_bounds__((Qelim3<N1>::NT), 2)
    qelim3_kernel(ExaDims P, const int* nslot, const int* perm, const int* bf, const double* __restrict__ rgJ,
                  const double* __restrict__ Fq, const double* __restrict__ MC, const double* __restrict__ ME,
                  double* D, double* F, double* K, double* H, const __grid_constant__ Tensor1D<N1> T) {
  using Q = Qelim3<N1>;
  constexpr int NP = Q::NP, NPF = Q::NPF, SY = Q::SY, SZ = Q::SZ, PAD = Q::PAD, FPAD = Q::FPAD, NDF = 6 * NPF;
  constexpr int CB = Q::CB, NT = Q::NT, COLS = NP + NDF;
  extern __shared__ double qsm[];
  double* V = qsm;                  // [CB][3][PAD]: nodal fields
  double* W = V + CB * Q::VS;       // [CB][3][PAD]: worked fields
  double* Fc = W + CB * Q::VS;      // [CB][6][3][FPAD]
  __shared__ int spos[NDF];         // where each face node's value lies in a field
  __shared__ int sout[NDF];         // and in Fc, the trace rows' flux of that node
  __shared__ int snode[3 * NP];     // in Fc, the u rows' fluxes of the faces each node lies on (in order)
  __shared__ unsigned char smask[NP];  // and those faces
  __shared__ int sbnd[6];
  const int le = blockIdx.x, tid = threadIdx.x, n = P.n, m = P.m;
  auto point = [](int i) { return i % N1 + SY * ((i / N1) % N1) + SZ * (i / NPF); };
  auto fpos = [](int a) { return a % N1 + SY * (a / N1); };
  for (int s = tid; s < NDF; s += NT) {
    const int l = s / NPF;
    spos[s] = point(perm[s]);
    sout[s] = (3 * l + (bf[l + 6 * le] > 0 ? 1 : 0)) * FPAD + fpos(s - l * NPF);
  }
  for (int i = tid; i < NP; i += NT) {
    int mask = 0;
    for (int c = 0; c < 3; ++c) {
      const int sl = nslot[3 * i + c], l = sl / NPF;
      snode[3 * i + c] = sl >= 0 ? 3 * l * FPAD + fpos(sl - l * NPF) : -1;
      if (sl >= 0) mask |= 1 << l;
    }
    smask[i] = (unsigned char)mask;
  }
  if (tid < 6) sbnd[tid] = bf[tid + 6 * le] > 0;
  const double* R = rgJ + (long long)le * NP * 4 * 4 + NP * 4;  // the q fields' part
  const double* fq = Fq + (long long)le * 2 * NDF * 3;
  const double* C = MC + (long long)le * NP * 3 * NP;
  const double* E = ME + (long long)le * NP * 3 * NDF;
  const int groups = (COLS + CB - 1) / CB;
  auto fetch = [&](int grp) {
    const int q0 = grp * CB, nb = min(CB, COLS - q0);
    for (int t = tid; t < nb * 3 * NP; t += NT) {
      const int r = t % (3 * NP), j = t / (3 * NP), col = q0 + j;
      const double* src = (col < NP ? C + (long long)3 * NP * col : E + (long long)3 * NP * (col - NP)) + r;
      const unsigned d = (unsigned)__cvta_generic_to_shared(V + j * Q::VS + r / NP * PAD + point(r % NP));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src));
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  if ((int)blockIdx.y < groups) fetch(blockIdx.y);
  for (int grp = blockIdx.y; grp < groups; grp += gridDim.y) {
    const int q0 = grp * CB, nb = min(CB, COLS - q0);
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    // planes of the fields and of the face fields, both in-plane dimensions to the points
    const int planes = nb * 3 * N1;
    for (int t = tid; t < planes + nb * 18; t += NT) {
      double a[N1][N1];
      if (t < planes) {
        const int z = t % N1, d = (t / N1) % 3, j = t / (3 * N1);
        const double* src = V + j * Q::VS + d * PAD + SZ * z;
#pragma unroll
        for (int y = 0; y < N1; ++y)
#pragma unroll
          for (int x = 0; x < N1; ++x) a[y][x] = src[SY * y + x];
        tp_plane<N1, false>(a, T.S);
        double* dst = W + j * Q::VS + d * PAD + SZ * z;
#pragma unroll
        for (int y = 0; y < N1; ++y)
#pragma unroll
          for (int x = 0; x < N1; ++x) dst[SY * y + x] = a[y][x];
      } else {
        const int u = t - planes, ld = u % 18, l = ld / 3, d = ld - 3 * l, j = u / 18;
        const double* src = V + j * Q::VS + d * PAD;
#pragma unroll
        for (int y = 0; y < N1; ++y)
#pragma unroll
          for (int x = 0; x < N1; ++x) a[y][x] = src[spos[l * NPF + N1 * y + x]];
        tp_plane<N1, false>(a, T.S);
        double* dst = Fc + j * Q::FS + ld * FPAD;
#pragma unroll
        for (int y = 0; y < N1; ++y)
#pragma unroll
          for (int x = 0; x < N1; ++x) dst[SY * y + x] = a[y][x];
      }
    }
    __syncthreads();
    if (grp + (int)gridDim.y < groups) fetch(grp + gridDim.y);
    // the third dimension, the Jacobians at the points, and the third dimension back
    for (int t = tid; t < nb * NPF; t += NT) {
      const int p = t % NPF, j = t / NPF;
      double* w = W + j * Q::VS + p % N1 + SY * (p / N1);
      double v[3][N1];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double in[N1];
#pragma unroll
        for (int z = 0; z < N1; ++z) in[z] = w[d * PAD + SZ * z];
        tp_to_points<N1>(T.S, in, v[d]);
      }
      double A[N1], Xa[N1], Ya[N1];
#pragma unroll
      for (int c = 0; c < N1; ++c) A[c] = Xa[c] = Ya[c] = 0.0;
#pragma unroll
      for (int z = 0; z < N1; ++z) {
        double s[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const double* Rr = R + p + NPF * z + NP * r;
          s[r] = fma(Rr[0], v[0][z], fma(Rr[NP * 4], v[1][z], Rr[NP * 8] * v[2][z]));
        }
#pragma unroll
        for (int c = 0; c < N1; ++c) {
          A[c] = fma(T.Sw[z + N1 * c], s[0], fma(T.Dw[z + N1 * c], s[3], A[c]));
          Xa[c] = fma(T.Sw[z + N1 * c], s[1], Xa[c]);
          Ya[c] = fma(T.Sw[z + N1 * c], s[2], Ya[c]);
        }
      }
#pragma unroll
      for (int c = 0; c < N1; ++c) {
        w[SZ * c] = A[c];
        w[PAD + SZ * c] = Xa[c];
        w[2 * PAD + SZ * c] = Ya[c];
      }
    }
    // face points: the u rows' flux, and the trace rows' where a boundary condition makes it another
    for (int t = tid; t < nb * NDF; t += NT) {
      const int s = t % NDF, l = s / NPF, j = t / NDF;
      double* f = Fc + j * Q::FS + 3 * l * FPAD + fpos(s - l * NPF);
      const double* c = fq + (s - l * NPF) + 3 * NPF * l;
      const double v0 = f[0], v1 = f[FPAD], v2 = f[2 * FPAD];
      f[0] = fma(c[0], v0, fma(c[NPF], v1, c[2 * NPF] * v2));
      if (sbnd[l]) {
        const double* cT = c + 3 * NDF;
        f[FPAD] = fma(cT[0], v0, fma(cT[NPF], v1, cT[2 * NPF] * v2));
      }
    }
    __syncthreads();
    // back along the second dimension, lines of the fields; faces whole
    for (int t = tid; t < nb * (NPF + 12); t += NT) {
      if (t < nb * NPF) {
        const int p = t % NPF, j = t / NPF;
        double* w = W + j * Q::VS + p % N1 + SZ * (p / N1);
        double in[N1], o[N1], der[N1];
#pragma unroll
        for (int g = 0; g < N1; ++g) in[g] = w[2 * PAD + SY * g];
        tp_to_nodes<N1>(T.Dw, in, der);
#pragma unroll
        for (int g = 0; g < N1; ++g) in[g] = w[SY * g];
        tp_to_nodes<N1>(T.Sw, in, o);
#pragma unroll
        for (int g = 0; g < N1; ++g) w[SY * g] = o[g] + der[g];
        tp_line<N1, true>(w + PAD, SY, T.Sw);
      } else {
        const int u = t - nb * NPF, ls = u % 12, l = ls >> 1, side = ls & 1, j = u / 12;
        if (side && !sbnd[l]) continue;
        double* f = Fc + j * Q::FS + (3 * l + side) * FPAD;
        double a[N1][N1];
#pragma unroll
        for (int y = 0; y < N1; ++y)
#pragma unroll
          for (int x = 0; x < N1; ++x) a[y][x] = f[SY * y + x];
        tp_plane<N1, true>(a, T.Sw);
#pragma unroll
        for (int y = 0; y < N1; ++y)
#pragma unroll
          for (int x = 0; x < N1; ++x) f[SY * y + x] = a[y][x];
      }
    }
    __syncthreads();
    for (int t = tid; t < nb * NPF; t += NT) {  // the first dimension
      const int p = t % NPF, j = t / NPF;
      double* w = W + j * Q::VS + SY * (p % N1) + SZ * (p / N1);
      double in[N1], o[N1], der[N1];
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = w[PAD + g];
      tp_to_nodes<N1>(T.Dw, in, der);
#pragma unroll
      for (int g = 0; g < N1; ++g) in[g] = w[g];
      tp_to_nodes<N1>(T.Sw, in, o);
#pragma unroll
      for (int g = 0; g < N1; ++g) w[g] = o[g] + der[g];
    }
    __syncthreads();
    // u rows: minus the volume, plus the face terms in the order of the faces
    double* De = D + (long long)le * n * n;
    double* Fe = F + (long long)le * n * m;
    for (int t = tid; t < nb * NP; t += NT) {
      const int i = t % NP, j = t / NP, col = q0 + j;
      const double* f = Fc + j * Q::FS;
      double v = -W[j * Q::VS + point(i)];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int o = snode[3 * i + c];
        if (o >= 0) v += f[o];
      }
      if (col < NP) {
        De[n * col + i] += v;
      } else {
        const int cf = col - NP;
        const double old = (smask[i] >> (cf / NPF)) & 1 ? Fe[n * cf + i] : 0.0;
        Fe[n * cf + i] = old - v;
      }
    }
    // trace rows
    double* Ke = K + (long long)le * m * n;
    double* He = H + (long long)le * m * m;
    for (int t = tid; t < nb * NDF; t += NT) {
      const int s = t % NDF, j = t / NDF, col = q0 + j;
      const double v = Fc[j * Q::FS + sout[s]];
      if (col < NP) {
        const double old = (smask[col] >> (s / NPF)) & 1 ? Ke[m * col + s] : 0.0;
        Ke[m * col + s] = old + v;
      } else {
        const int cf = col - NP;
        const double old = s / NPF == cf / NPF ? He[m * cf + s] : 0.0;
        He[m * cf + s] = old - v;
      }
    }
  }
}

// products per column: the volume part, and the faces'
inline double qelim_tp_volume(const ExaTensor& T) { return (18.0 * T.n1 + 12.0) * T.n1 * T.n1 * T.n1; }
inline double qelim_tp_faces(const ExaTensor& T) { return (48.0 * T.n1 + 18.0) * T.n1 * T.n1; }
// whether a model with q on these elements has an instance
inline bool qelim_tp_fits(const ExaDims& P, const ExaTensor& T) {
  return P.ncq == 3 && P.nd == 3 && P.ncu == 1 && P.nfe == 6 && T.n1 >= 3 && T.n1 <= 5;
}
inline int launch_qelim_tp(const ExaDims& P, const ExaTensor& T, const int* nslot, const int* perm, const int* bf,
                           const double* rgJ, const double* Fq, const double* MC, const double* ME, double* D, double* F,
                           double* K, double* H, int nb, cudaStream_t st) {
#define EXA_Q3(N1)                                                                                                    \
  if (T.n1 == N1) {                                                                                                   \
    using Q = Qelim3<N1>;                                                                                             \
    auto kern = qelim3_kernel<N1>;                                                                                    \
    EXA_TRY(exa_allow_smem((const void*)kern, Q::smem));                                                              \
    /* small meshes: several blocks per element, about two waves of two per SM */                                     \
    const int parts = std::max(1, std::min((P.npe + P.ndf + Q::CB - 1) / Q::CB, 592 / nb));                           \
    kern<<<dim3(nb, parts), Q::NT, Q::smem, st>>>(P, nslot, perm, bf, rgJ, Fq, MC, ME, D, F, K, H, tensor_1d<N1>(T)); \
    EXA_LAUNCH_CHECK();                                                                                               \
    return EXA_OK;                                                                                                    \
  }
  EXA_Q3(3) EXA_Q3(4) EXA_Q3(5)
#undef EXA_Q3
  exa_set_error("q elimination: no tensor-product instance");
  return EXA_ERR_UNSUPPORTED;
}

// The same for the trace rows alone in the mixed form: K = K + G MinvC and H = H - G MinvE in FP32,
//   G x = Sw (x) Sw sum_d f_d (S (x) S) x_d   on the nodes of each face,
// in place of products with G, whose rows meet the nodes of one face only (75 of 375 columns at p = 4)
// and whose 150 rows fill two tensor-core tiles of 128.  One warp per face, one column of MinvC or
// MinvE per lane, a face's plane in registers, the 1D tables in constant memory: 1075 products per face
// and column against 9.4 thousand.  Bound: instructions and the latency of the loads (2.9 GB, 0.44 ms at
// the copy rate).  Measured (B200, 4096 hexahedra, p = 4; before: two 3xTF32 products): 1.87 -> 0.90 ms,
// and 0.15 ms in the face kernel, which writes no G; the assembly 8.70 -> 7.64 ms.  Three blocks per SM
// instead of four: 1.10 ms.  Without the prefetch of the columns 64 elements on the assembly takes
// 7.69 ms.
constexpr int TRQ_COLS = 32, TRQ_LD = 34;  // columns of a block; row stride (its quads land in other banks)
constexpr int TRQ_AHEAD = 64;
template <int N1>
struct TraceTables {
  float S[N1 * N1], Sw[N1 * N1];
};
template <int N1>
__global__ void __launch_bounds__(192, 4)
    trace_q_kernel(ExaDims P, int kg, const int* nslot, const int* perm, const double* __restrict__ Fq, UPacked MC,
                   UPacked ME, const double* __restrict__ K, const double* __restrict__ H, float* K32, float* H32,
                   UPacked Kp, const __grid_constant__ TraceTables<N1> T) {
  constexpr int NP = N1 * N1 * N1, NPF = N1 * N1, M = 6 * NPF, MR = M | 1, FP = (N1 + 3) / 4 * 4;
  extern __shared__ __align__(16) float xs[];  // [3 kg, whole chunks][TRQ_LD], then the results [TRQ_COLS][MR]
  __shared__ __align__(16) float sf[6][3][N1][FP];  // derivatives of the trace flux at the points [x][y]
  __shared__ int sp[M];                        // rows of xs of the face nodes
  __shared__ unsigned char son[NP];            // faces each node lies on
  const int le = blockIdx.y, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int cblocks = (NP + TRQ_COLS - 1) / TRQ_COLS;
  const bool trace = (int)blockIdx.x >= cblocks;  // columns of MinvE
  const int c0 = (trace ? blockIdx.x - cblocks : blockIdx.x) * TRQ_COLS;
  const int ncol = min(TRQ_COLS, (trace ? M : NP) - c0);
  const UPacked X = trace ? ME : MC;
  {
    const float* src = X.hi + (long long)le * X.sb;
    const int ng = (X.R + 7) / 8, g0 = c0 >> 3;
    const int blocks = (3 * kg + exa_tc::PK - 1) / exa_tc::PK * 4;
    float* dl = xs + 4 * (lane >> 3) * TRQ_LD + (lane & 7);
#pragma unroll 4
    for (int b = w; b < blocks; b += 6) {  // 8 columns x 16 k, 512 contiguous bytes
      const int g = b & 3, kb = b >> 2;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (g0 + g < ng) v = *reinterpret_cast<const float4*>(src + (kb * ng + g0 + g) * 128 + 4 * lane);
      float* d = dl + 16 * kb * TRQ_LD + 8 * g;
      d[0] = v.x;
      d[TRQ_LD] = v.y;
      d[2 * TRQ_LD] = v.z;
      d[3 * TRQ_LD] = v.w;
    }
    // the columns of the same block TRQ_AHEAD elements on into L2
    if (le + TRQ_AHEAD < (int)gridDim.y) {
      const float* nx = src + TRQ_AHEAD * X.sb;
      for (int t = tid; t < blocks * 4; t += 192) {
        const int b = t >> 2, g = b & 3, kb = b >> 2;
        if (g0 + g < ng)
          asm volatile("prefetch.global.L2 [%0];\n" ::"l"(nx + (kb * ng + g0 + g) * 128 + 32 * (t & 3)));
      }
    }
    const double* fq = Fq + (long long)le * 2 * M * 3 + M * 3;
    for (int t = tid; t < M * 3; t += 192) {
      const int l = t / (3 * NPF), d = t / NPF % 3, p = t % NPF;
      sf[l][d][p % N1][p / N1] = (float)fq[t];
    }
    for (int t = tid; t < M; t += 192) sp[t] = perm[t] * TRQ_LD;
    for (int i = tid; i < NP; i += 192) {
      int mask = 0;
      for (int c = 0; c < 3; ++c)
        if (nslot[3 * i + c] >= 0) mask |= 1 << (nslot[3 * i + c] / NPF);
      son[i] = (unsigned char)mask;
    }
  }
  __syncthreads();
  float acc[N1][N1];
#pragma unroll
  for (int y = 0; y < N1; ++y)
#pragma unroll
    for (int x = 0; x < N1; ++x) acc[y][x] = 0.f;
  int at[NPF];
#pragma unroll
  for (int i = 0; i < NPF; ++i) at[i] = sp[w * NPF + i];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float* xd = xs + d * kg * TRQ_LD + lane;
    float a[N1][N1];
#pragma unroll
    for (int y = 0; y < N1; ++y) {  // the first dimension of the face, row by row
      float in[N1];
#pragma unroll
      for (int x = 0; x < N1; ++x) in[x] = xd[at[N1 * y + x]];
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        float o = 0.f;
#pragma unroll
        for (int x = 0; x < N1; ++x) o = fmaf(T.S[g + N1 * x], in[x], o);
        a[y][g] = o;
      }
    }
#pragma unroll
    for (int x = 0; x < N1; ++x) {
      __align__(16) float f[FP];
#pragma unroll
      for (int i = 0; i < FP; i += 4) *reinterpret_cast<float4*>(f + i) = *reinterpret_cast<const float4*>(&sf[w][d][x][i]);
#pragma unroll
      for (int g = 0; g < N1; ++g) {
        float o = 0.f;
#pragma unroll
        for (int y = 0; y < N1; ++y) o = fmaf(T.S[g + N1 * y], a[y][x], o);
        acc[g][x] = fmaf(f[g], o, acc[g][x]);
      }
    }
  }
  // back to the nodes
  float out[N1][N1];
#pragma unroll
  for (int y = 0; y < N1; ++y)
#pragma unroll
    for (int x = 0; x < N1; ++x) {
      float o = 0.f;
#pragma unroll
      for (int g = 0; g < N1; ++g) o = fmaf(T.Sw[g + N1 * x], acc[y][g], o);
      out[y][x] = o;
    }
  __syncthreads();  // the columns have been read: the results take their place
#pragma unroll
  for (int x = 0; x < N1; ++x)
#pragma unroll
    for (int y = 0; y < N1; ++y) {
      float o = 0.f;
#pragma unroll
      for (int g = 0; g < N1; ++g) o = fmaf(T.Sw[g + N1 * y], out[g][x], o);
      xs[lane * MR + w * NPF + N1 * y + x] = o;
    }
  __syncthreads();
  // a column per warp; an entry that couples a face with its own nodes adds to what the face kernel left
  if (trace) {
    for (int j = w; j < ncol; j += 6) {
      const int cf = c0 + j, r0 = cf / NPF * NPF;
      const long long o = (long long)le * M * M + (long long)M * cf;
#pragma unroll
      for (int i = 0; i < (M + 31) / 32; ++i) {
        const int r = lane + 32 * i;
        if (r >= M) break;
        const float v = xs[j * MR + r];
        H32[o + r] = r >= r0 && r < r0 + NPF ? (float)(H[o + r] - (double)v) : -v;
      }
    }
    return;
  }
  for (int j = w; j < ncol; j += 6) {
    const int mask = son[c0 + j];
    const long long o = (long long)le * M * NP + (long long)M * (c0 + j);
#pragma unroll
    for (int i = 0; i < (M + 31) / 32; ++i) {
      const int r = lane + 32 * i;
      if (r >= M) break;
      float v = xs[j * MR + r];
      if ((mask >> (r / NPF)) & 1) xs[j * MR + r] = v = (float)(K[o + r] + (double)v);
      K32[o + r] = v;
    }
  }
  __syncthreads();
  // the packed operand of K D^-1 F, row r and k = column: 8 rows x 4 columns per warp
  const int nkc = (Kp.K + exa_tc::PK - 1) / exa_tc::PK, ng0 = (min(M, Kp.TR) + 7) / 8, ng1 = (M - Kp.TR + 7) / 8;
  float* kp = Kp.hi + (long long)le * Kp.sb + lane;
  const int k3 = lane & 3, r7 = lane >> 2;
  for (int b = w; b < (M + 7) / 8 * (TRQ_COLS / 4); b += 6) {
    const int q = b & (TRQ_COLS / 4 - 1), r8 = b / (TRQ_COLS / 4), r = 8 * r8 + r7, k = 4 * q + k3, kk = c0 + 4 * q;
    if (r >= M || k >= ncol) continue;
    const int base = 8 * r8 >= Kp.TR ? (Kp.TR / 8) * nkc * 128 + ((kk >> 4) * ng1 + r8 - Kp.TR / 8) * 128
                                     : ((kk >> 4) * ng0 + r8) * 128;
    kp[base + ((kk >> 2) & 3) * 32] = xs[k * MR + r];
  }
}
inline size_t trace_q_smem(const ExaDims& P, int kg) {
  return sizeof(float) * std::max((size_t)(3 * kg + exa_tc::PK - 1) / exa_tc::PK * exa_tc::PK * TRQ_LD, (size_t)TRQ_COLS * (P.m | 1));
}
inline int launch_trace_q(const ExaDims& P, const ExaTensor& T, const int* nslot, const int* perm, const double* Fq,
                          const UPacked& MC, const UPacked& ME, const double* K, const double* H, float* K32, float* H32,
                          const UPacked& Kp, int nb, cudaStream_t st) {
  const int kg = exa_tc::qk_group(P.npe);
  const int blocks = exa_ceil_div(P.npe, TRQ_COLS) + exa_ceil_div(P.ndf, TRQ_COLS);
  const size_t sm = trace_q_smem(P, kg);
#define EXA_TRQ(N1)                                                                                                 \
  if (T.n1 == N1) {                                                                                                 \
    TraceTables<N1> t;                                                                                              \
    const Tensor1D<N1> d = tensor_1d<N1>(T);                                                                        \
    for (int i = 0; i < N1 * N1; ++i) {                                                                             \
      t.S[i] = (float)d.S[i];                                                                                       \
      t.Sw[i] = (float)d.Sw[i];                                                                                     \
    }                                                                                                               \
    auto kern = trace_q_kernel<N1>;                                                                                 \
    EXA_TRY(exa_allow_smem((const void*)kern, sm));                                                                 \
    kern<<<dim3(blocks, nb), 192, sm, st>>>(P, kg, nslot, perm, Fq, MC, ME, K, H, K32, H32, Kp, t);                 \
    EXA_LAUNCH_CHECK();                                                                                             \
    return EXA_OK;                                                                                                  \
  }
  EXA_TRQ(3) EXA_TRQ(4) EXA_TRQ(5)
#undef EXA_TRQ
  exa_set_error("q elimination: no tensor-product instance");
  return EXA_ERR_UNSUPPORTED;
}

// B of the chunk from the same data, for callers that read it (the solver does not form it): the
// volume pairs of the q fields, then the face terms face by face.
__global__ void face_b_kernel(ExaDims P, const double* shapfgt, const double* shapfgw, const int* perm, const double* Fq,
                              double* B) {
  const int le = blockIdx.x, npe = P.npe, npf = P.npf, ngf = P.ngf, ncu = P.ncu, nd = P.nd, n = P.n;
  const int ncq = ncu * nd;
  const double* fq = Fq + (long long)le * 2 * P.nfe * ngf * ncu * ncq;
  double* Be = B + (long long)le * n * npe * nd * ncu;
  for (int l = 0; l < P.nfe; ++l) {
    for (int t = threadIdx.x; t < npf * npf * ncu * ncq; t += blockDim.x) {
      const int a = t % npf, b = (t / npf) % npf, k = (t / (npf * npf)) % ncu, c = t / (npf * npf * ncu);
      double s = 0.0;
      for (int g = 0; g < ngf; ++g)
        s = fma(shapfgw[a + npf * g] * shapfgt[g + ngf * b], fq[g + ngf * (k + ncu * c) + ngf * ncu * ncq * l], s);
      const int nq = c % ncu, d = c / ncu;
      Be[perm[a + npf * l] + npe * k + (long long)n * (perm[b + npf * l] + npe * d + npe * nd * nq)] += s;
    }
    __syncthreads();
  }
}
