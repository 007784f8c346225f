// Model-specific translation unit: instantiates the assembly kernels for one
// generated model (header produced by exasim_b200/modelc.py, selected at build time
// with -DEXA_MODEL_HEADER="..." -DEXA_MODEL_NS=exa_model_<name>) and runs the
// element-block loop of hdgAssembleLinearSystem / hdgAssembleResidual
// (backend/Discretization/uequation.cpp:778-787, 1080-1088).
#include <vector>

#include "exa_assembly.cuh"
#include "exa_ldg.cuh"
#include "exa_ldg_tp.cuh"
#include "exa_hdg_tp.cuh"
#include "exa_qelim_tp.cuh"
#include "exa_vol_tp.cuh"
#include "exa_solver.cuh"
#include "exa_umma.cuh"
#include EXA_MODEL_HEADER

EXA_BIND_MODEL(EXA_MODEL_NS)

namespace {

AsmArgs make_args(const ExaCtx& c, int e0) {
  AsmArgs A{};
  A.P = c.P;
  A.shapegt = c.shapegt; A.shapegw = c.shapegw; A.shapfgt = c.shapfgt; A.shapfgw = c.shapfgw;
  A.perm = c.perm; A.elemcon = c.elemcon; A.bf = c.bf;
  A.elemg = c.elemg; A.faceg = c.faceg;
  A.uinf = c.uinf; A.param = c.param; A.tau = c.tau;
  A.udg = c.udg; A.uh = c.uh; A.sdg = c.sdg;
  A.time = c.time; A.dtfactor = c.dtfactor;
  A.tdep = c.tdep; A.tdfunc = c.tdfunc; A.sourcefunc = c.sourcefunc; A.modelnumber = c.modelnumber;
  A.e0 = e0;
  return A;
}

int smem_attr(const void* fn, size_t bytes) {
  EXA_TRY(exa_allow_smem(fn, bytes));
  return EXA_OK;
}

// The element inverse needs D alone, so once the q-elimination product into D is done it
// runs on the context's second stream, beside the three products into F, K and H: its pivot
// loop is latency-bound and the products are HBM- or tensor-bound.  With phase profiling on,
// everything stays on the context stream, so the phase events time each step alone.
// Blocks of a warp's inverse (order up to 32) are too short a step to pay for the two events.
bool overlap_inverse(const ExaCtx& c) { return c.P.ncq > 0 && c.st2 && !c.prof.on && c.P.n > 32; }

// The context stream joins the second stream before any later work, on every path out of a
// Schur step (an early error return included), so nothing it runs next can overlap it.
struct InverseJoin {
  ExaCtx& c;
  bool pending = false;
  ~InverseJoin() {
    if (pending) cudaStreamWaitEvent(c.st, c.ev_inv, 0);
  }
  int join() {
    pending = false;
    EXA_CUDA(cudaStreamWaitEvent(c.st, c.ev_inv, 0));
    return EXA_OK;
  }
};

template <class Fn>
int inverse_beside(ExaCtx& c, InverseJoin& j, Fn&& fn) {
  EXA_CUDA(cudaEventRecord(c.ev_q, c.st));
  EXA_CUDA(cudaStreamWaitEvent(c.st2, c.ev_q, 0));
  j.pending = true;
  const int st = fn(c.st2);
  // recorded whatever fn returned, so the join covers whatever it enqueued; if the record
  // itself fails, the second stream is drained here, so that nothing left on it can outlive
  // this step (the join would otherwise wait on the previous step's event)
  const cudaError_t e = cudaEventRecord(c.ev_inv, c.st2);
  if (e != cudaSuccess) {
    j.pending = false;
    cudaStreamSynchronize(c.st2);
    exa_set_error("cudaEventRecord on the second stream: %s", cudaGetErrorString(e));
    return EXA_ERR_CUDA;
  }
  return st;
}

// the plain form's q elimination by sum factorization (exa_qelim_tp.cuh)
bool tp_qelim(const ExaCtx& c) { return c.wFq && c.precision != 1; }
// its trace rows in the mixed form (B is packed there by the volume kernel)
bool tp_trace(const ExaCtx& c) { return c.wFq && c.precision == 1 && c.Sp.hi; }

// Schur condensation of one chunk (uequation.cpp:559-775): q-elimination, D^-1, DinvF,
// Ru <- D^-1 Ru, H += K DinvF, Rh -= K Ru.
int schur_chunk(ExaCtx& c, int e0, int nb) {
  const ExaDims& P = c.P;
  const int n = P.n, m = P.m, npe = P.npe, nd = P.nd, ncu = P.ncu, ndf = P.ndf;
  const long long nqn = (long long)npe * nd * ncu;
  double* Hc = c.H + (long long)e0 * m * m;
  const bool overlap = overlap_inverse(c) && !tp_qelim(c);
  InverseJoin join{c};
  if (tp_qelim(c)) {
    ExaProfScope ps(c, EXA_PH_QELIM);
    exa_prof_flops(c, EXA_PH_QELIM, 2.0 * nb * (qelim_tp_volume(c.tensor) + qelim_tp_faces(c.tensor)) * (npe + ndf));
    const double* MC = c.MC + (long long)e0 * npe * npe * nd;
    const double* ME = c.ME + (long long)e0 * npe * ndf * nd;
    EXA_TRY(launch_qelim_tp(P, c.tensor, c.tp_nslot, c.perm, c.bf + (long long)e0 * P.nfe, c.wRg,
                                    c.wFq, MC, ME, c.wD, c.wF, c.wK, Hc, nb, c.st));
  } else if (P.ncq > 0) {
    ExaProfScope ps(c, EXA_PH_QELIM);
    // four GEMMs per trace component with K = npe*nd: (n + m) rows x (npe + ndf) columns in all
    exa_prof_flops(c, EXA_PH_QELIM, 2.0 * nb * ncu * (double)npe * nd * (double)(n + m) * (npe + ndf));
    const double* MC = c.MC + (long long)e0 * npe * npe * nd;
    const double* ME = c.ME + (long long)e0 * npe * ndf * nd;
    // contraction over the stacked (l, d) rows of MinvC / MinvE (K = npe*nd), one GEMM per
    // block and per trace component b (batch2 = ncu)
    const long long kq = (long long)npe * nd;
    GemmBatch g{};
    g.batch = nb; g.batch2 = ncu;
    g.K = (int)kq; g.beta = 1.0;
    GemmBatch q4[EXA_GEMM_GROUP];
    // D(:, j + npe*b) += sum_(l,d) B(:, l + npe*d + npe*nd*b) MinvC(l, d, j)
    g.M = n; g.N = npe; g.alpha = 1.0;
    g.A = c.wB; g.lda = n; g.sA = (long long)n * nqn; g.sA2 = (long long)n * kq;
    g.B = MC; g.ldb = kq; g.sB = kq * npe; g.sB2 = 0;
    g.C = c.wD; g.ldc = n; g.sC = (long long)n * n; g.sC2 = (long long)n * npe;
    q4[0] = g;
    // F(:, b + ncu*jf) -= sum_(l,d) B(:, l + npe*d + npe*nd*b) MinvE(l, d, jf)
    g.N = ndf; g.alpha = -1.0;
    g.B = ME; g.ldb = kq; g.sB = kq * ndf;
    g.C = c.wF; g.ldc = (long long)n * ncu; g.sC = (long long)n * m; g.sC2 = n;
    q4[1] = g;
    // K(:, j + npe*b) += sum_(l,d) G(:, l + npe*d + npe*nd*b) MinvC(l, d, j)
    g.M = m; g.N = npe; g.alpha = 1.0;
    g.A = c.wG; g.lda = m; g.sA = (long long)m * nqn; g.sA2 = (long long)m * kq;
    g.B = MC; g.ldb = kq; g.sB = kq * npe;
    g.C = c.wK; g.ldc = m; g.sC = (long long)m * n; g.sC2 = (long long)m * npe;
    q4[2] = g;
    // H(:, b + ncu*jf) -= sum_(l,d) G(:, l + npe*d + npe*nd*b) MinvE(l, d, jf)
    g.N = ndf; g.alpha = -1.0;
    g.B = ME; g.ldb = kq; g.sB = kq * ndf;
    g.C = Hc; g.ldc = (long long)m * ncu; g.sC = (long long)m * m; g.sC2 = m;
    q4[3] = g;
    if (overlap) {
      EXA_TRY(exa_gemm(q4[0], c.st));
      EXA_TRY(inverse_beside(c, join, [&](cudaStream_t s) {
        return exa_inverse_ws(c.wD, n, (long long)n * n, nb, c.wInv, c.d_flag, s);
      }));
      for (int i = 1; i < 4; ++i) EXA_TRY(exa_gemm(q4[i], c.st));
    } else {
      EXA_TRY(exa_gemm_group(q4, 4, c.st));
    }
  }
  if (overlap) {
    EXA_TRY(join.join());
  } else {
    ExaProfScope ps(c, EXA_PH_INVERSE);
    EXA_TRY(exa_inverse_ws(c.wD, n, (long long)n * n, nb, c.wInv, c.d_flag, c.st));
  }
  ExaProfScope ps(c, EXA_PH_SCHUR);
  // D^-1 F and K D^-1 F run over the k that face_k lists, a face's unknowns, where it does
  const double kf = c.face_k ? (double)P.npf * ncu : (double)n;
  exa_prof_flops(c, EXA_PH_SCHUR, 2.0 * nb * ((double)n * m * kf + (double)n * n + (double)m * m * kf + (double)m * n));
  GemmBatch g{};
  g.batch = nb; g.batch2 = 1;
  // DinvF = -Dinv F.  Without q the columns of F on face l have entries at that face's nodes only,
  // and so have the rows of K below: the products run over those k, face by face (B200, 1000
  // hexahedra of 3D Euler at p = 3, 80 of 320: assembly 18.0 -> 13.7 ms)
  const int ncf = P.npf * ncu;
  g.M = n; g.N = m; g.K = n; g.alpha = -1.0; g.beta = 0.0;
  g.A = c.wD; g.lda = n; g.sA = (long long)n * n;
  g.B = c.wF; g.ldb = n; g.sB = (long long)n * m;
  g.C = c.F + (long long)e0 * n * m; g.ldc = n; g.sC = (long long)n * m;
  if (c.face_k) {
    g.N = ncf; g.K = ncf; g.batch2 = P.nfe;
    g.kidx = c.face_k; g.skidx = ncf;
    g.sB2 = (long long)n * ncf; g.sC2 = (long long)n * ncf;
  }
  EXA_TRY(exa_gemm(g, c.st));
  g.batch2 = 1; g.kidx = nullptr; g.sB2 = g.sC2 = 0; g.K = n;
  // Ru = Dinv Ru
  double* Ruc = c.Ru + (long long)e0 * n;
  EXA_CUDA(cudaMemcpyAsync(c.wRu, Ruc, sizeof(double) * (size_t)n * nb, cudaMemcpyDeviceToDevice, c.st));
  g.N = 1; g.alpha = 1.0;
  g.B = c.wRu; g.ldb = n; g.sB = n;
  g.C = Ruc; g.ldc = n; g.sC = n;
  EXA_TRY(exa_gemm(g, c.st));
  // H += K DinvF
  g.M = m; g.N = m; g.K = n; g.alpha = 1.0; g.beta = 1.0;
  g.A = c.wK; g.lda = m; g.sA = (long long)m * n;
  g.B = c.F + (long long)e0 * n * m; g.ldb = n; g.sB = (long long)n * m;
  g.C = Hc; g.ldc = m; g.sC = (long long)m * m;
  if (c.face_k) {
    g.M = ncf; g.K = ncf; g.batch2 = P.nfe;
    g.kidx = c.face_k; g.skidx = ncf;
    g.sA2 = ncf; g.sC2 = ncf;
    g.cown = ncf;  // the face kernel fills H's diagonal face blocks only
  }
  EXA_TRY(exa_gemm(g, c.st));
  g.M = m; g.K = n; g.batch2 = 1; g.kidx = nullptr; g.sA2 = g.sC2 = 0; g.cown = 0;
  // Rh -= K Ru
  g.N = 1; g.alpha = -1.0;
  g.B = Ruc; g.ldb = n; g.sB = n;
  g.C = c.Rh + (long long)e0 * m; g.ldc = m; g.sC = m;
  EXA_TRY(exa_gemm(g, c.st));
  return EXA_OK;
}

// Mixed-precision Schur condensation of one chunk: the steps of schur_chunk with the
// products in 3xTF32 on the tensor cores (FP32 accumulation) over operands packed in the
// tensor-core layout, and the results kept in FP32: Dinv32 = D^-1, F32 = -D^-1 F,
// K32 = K, H32 = H + K D^-1 F.  The GEMM epilogues write each result both where the
// solver reads it and packed for the next product.  Ru <- D^-1 Ru and Rh <- Rh - K Ru stay
// FP64 vectors (FP32 matrices, FP64 accumulation).
int schur_chunk_mixed(ExaCtx& c, int e0, int nb) {
  const ExaDims& P = c.P;
  const int n = P.n, m = P.m, npe = P.npe, nd = P.nd, ncu = P.ncu, ndf = P.ndf;
  const long long nqn = (long long)npe * nd * ncu;
  float* D32 = c.Dinv32 + (long long)e0 * n * n;
  float* K32 = c.K32 + (long long)e0 * m * n;
  float* H32 = c.H32 + (long long)e0 * m * m;
  float* F32 = c.F32 + (long long)e0 * n * m;
  const double* Hc = c.fp64_full ? c.H + (long long)e0 * m * m : c.H;  // per-chunk staging in the mixed form
  const bool overlap = overlap_inverse(c);
  InverseJoin join{c};
  // D^-1 in FP32 (the recursive blocked form with its products on the tensor cores where
  // the order exceeds the register kernel's, else the register kernel), then packed
  auto inverse = [&](cudaStream_t s) -> int {
    if (c.wInvPk)
      EXA_TRY(exa_inverse_tc32(D32, n, (long long)n * n, nb, c.wInv32, c.wInvPk, c.d_flag, c.d_uflag, s));
    else
      EXA_TRY(exa_inverse_ws(D32, n, (long long)n * n, nb, reinterpret_cast<float*>(c.wInv), c.d_flag, s));
    return EXA_OK;
  };
  auto pack_dinv = [&](cudaStream_t s) { return exa_pack(D32, 0, 1, n, (long long)n * n, 0, nb, 1, c.Dinvp, s); };
  auto at = [](UPacked u, long long e) {  // operand of element e of the set
    u.hi += e * u.sb;
    if (u.lo) u.lo += e * u.sb;
    return u;
  };
  UPackOut toF{c.wFp, 1, 1, 0}, toK{c.Kp, 0, 1, 0};
  if (P.ncq > 0) {
    const long long kq = (long long)npe * nd;   // the contraction, and B's columns per component
    const int kg = exa_tc::qk_group(npe);       // packed K: a group of kg per gradient component
    if (!c.Sp.hi) {
      // B per trace component b: row r, packed k = l + kg*d from column l + npe*d + npe*nd*b.
      // With the tensor-core volume kernel B is already packed (volume and face kernels write
      // it so), and G always is (the face kernel writes it in this layout in the mixed form)
      ExaProfScope pp(c, EXA_PH_PACK);
      EXA_TRY(exa_pack(c.wB, 1, 1, n, (long long)n * nqn, (long long)n * kq, nb, ncu, c.wBp, c.st, kg, npe));
    }
    ExaProfScope ps(c, EXA_PH_QELIM);
    exa_prof_flops(c, EXA_PH_QELIM, tp_trace(c) ? 2.0 * nb * (npe + ndf) * ((double)npe * nd * n + qelim_tp_faces(c.tensor))
                                                : 2.0 * nb * ncu * (double)npe * nd * (double)(n + m) * (npe + ndf));
    UGemmP u{};
    u.batch = nb; u.batch2 = ncu; u.K = kg * nd; u.beta = 1.0;
    u.tci = EXA_T_F64; u.tco = EXA_T_F32;
    // D(:, j + npe*b) = D + B_b MinvC
    u.M = n; u.N = npe; u.alpha = 1.0;
    u.A = c.wBp; u.B = at(c.MCp, e0); u.B.sb2 = 0;
    u.Cin = c.wD; u.ldci = n; u.sCi = (long long)n * n; u.sCi2 = (long long)n * npe;
    u.C = D32; u.ldc = n; u.sC = (long long)n * n; u.sC2 = (long long)n * npe;
    u.nout = 0;
    EXA_TRY(exa_gemm_3xtf32(u, c.d_uflag, c.st));
    if (overlap) EXA_TRY(inverse_beside(c, join, [&](cudaStream_t s) {
      EXA_TRY(inverse(s));
      return pack_dinv(s);
    }));
    // F(:, b + ncu*jf) = F - B_b MinvE, packed only (B operand of D^-1 F)
    u.N = ndf; u.alpha = -1.0;
    u.B = at(c.MEp, e0); u.B.sb2 = 0;
    u.Cin = c.wF; u.ldci = (long long)n * ncu; u.sCi = (long long)n * m; u.sCi2 = n;
    u.C = nullptr;
    toF.cmul = ncu; toF.cadd = 1;
    u.out[0] = toF; u.nout = 1;
    EXA_TRY(exa_gemm_3xtf32(u, c.d_uflag, c.st));
    // K and H: G is applied from the flux derivatives where the elements are tensor products
    if (tp_trace(c)) {
      ExaProfScope pt(c, EXA_PH_QTRACE);
      EXA_TRY(launch_trace_q(P, c.tensor, c.tp_nslot, c.perm, c.wFq, at(c.MCp, e0), at(c.MEp, e0), c.wK, Hc, K32, H32,
                             c.Kp, nb, c.st));
    }
    // K(:, j + npe*b) = K + G_b MinvC, plain and packed (A operand of K D^-1 F)
    u.M = m; u.N = npe; u.alpha = 1.0;
    u.A = c.wGp; u.B = at(c.MCp, e0); u.B.sb2 = 0;
    u.Cin = c.wK; u.ldci = m; u.sCi = (long long)m * n; u.sCi2 = (long long)m * npe;
    u.C = K32; u.ldc = m; u.sC = (long long)m * n; u.sC2 = (long long)m * npe;
    toK.cmul = 1; toK.cadd = npe;
    u.out[0] = toK; u.nout = 1;
    if (!tp_trace(c)) EXA_TRY(exa_gemm_3xtf32(u, c.d_uflag, c.st));
    // H(:, b + ncu*jf) = H - G_b MinvE
    u.N = ndf; u.alpha = -1.0;
    u.B = at(c.MEp, e0); u.B.sb2 = 0;
    u.Cin = Hc; u.ldci = (long long)m * ncu; u.sCi = (long long)m * m; u.sCi2 = m;
    u.C = H32; u.ldc = (long long)m * ncu; u.sC = (long long)m * m; u.sC2 = m;
    u.nout = 0;
    if (!tp_trace(c)) EXA_TRY(exa_gemm_3xtf32(u, c.d_uflag, c.st));
  } else {
    EXA_TRY(exa_k_to_f32(c.wD, D32, (long long)nb * n * n, c.st));
    EXA_TRY(exa_k_to_f32(c.wK, K32, (long long)nb * m * n, c.st));
    EXA_TRY(exa_k_to_f32(Hc, H32, (long long)nb * m * m, c.st));
    // F as the B operand of D^-1 F (row = column of F, k = row), K as an A operand
    EXA_TRY(exa_pack(c.wF, 1, n, 1, (long long)n * m, 0, nb, 1, c.wFp, c.st));
    EXA_TRY(exa_pack(c.wK, 1, 1, m, (long long)m * n, 0, nb, 1, c.Kp, c.st));
  }
  if (overlap) {
    EXA_TRY(join.join());
  } else {
    {
      ExaProfScope ps(c, EXA_PH_INVERSE);
      EXA_TRY(inverse(c.st));
    }
    ExaProfScope pp(c, EXA_PH_PACK);
    EXA_TRY(pack_dinv(c.st));
  }
  ExaProfScope ps(c, EXA_PH_SCHUR);
  exa_prof_flops(c, EXA_PH_SCHUR, 2.0 * nb * ((double)n * n * m + (double)n * n + (double)m * m * n + (double)m * n));
  UGemmP u{};
  u.batch = nb; u.batch2 = 1;
  u.tci = EXA_T_F32; u.tco = EXA_T_F32;
  // DinvF = -Dinv F: plain (Newton update) and packed (B operand of K DinvF)
  u.M = n; u.N = m; u.K = n; u.alpha = -1.0; u.beta = 0.0;
  u.A = c.Dinvp; u.B = c.wFp;
  u.Cin = nullptr;
  u.C = F32; u.ldc = n; u.sC = (long long)n * m;
  u.out[0] = UPackOut{c.DinvFp, 1, 1, 0}; u.nout = 1;
  EXA_TRY(exa_gemm_3xtf32(u, c.d_uflag, c.st));
  // H += K DinvF
  u.M = m; u.N = m; u.K = n; u.alpha = 1.0; u.beta = 1.0;
  u.A = c.Kp; u.B = c.DinvFp;
  u.Cin = H32; u.ldci = m; u.sCi = (long long)m * m;
  u.C = H32; u.ldc = m; u.sC = (long long)m * m;
  u.nout = 0;
  EXA_TRY(exa_gemm_3xtf32(u, c.d_uflag, c.st));
  // Ru = Dinv Ru; Rh -= K Ru
  double* Ruc = c.Ru + (long long)e0 * n;
  EXA_CUDA(cudaMemcpyAsync(c.wRu, Ruc, sizeof(double) * (size_t)n * nb, cudaMemcpyDeviceToDevice, c.st));
  EXA_TRY(exa_k_gemv32(n, n, nb, 1.0, D32, (long long)n * n, c.wRu, n, 0.0, Ruc, n, c.st, c.d_uflag));
  EXA_TRY(exa_k_gemv32(m, n, nb, -1.0, K32, (long long)m * n, Ruc, n, 1.0, c.Rh + (long long)e0 * m, m, c.st,
                       c.d_uflag));
  return EXA_OK;
}

}  // namespace

namespace {

// udg (and the stage source) at the Gauss points of elements e0 .. e0 + nb - 1 by GEMMs with the
// shared basis shapegt: the volume kernel then reads them instead of forming them per element
int volume_gauss_values(ExaCtx& c, AsmArgs& A, int e0, int nb) {
  const ExaDims& P = c.P;
  GemmBatch g{};
  g.M = P.nge; g.K = P.npe; g.alpha = 1.0; g.beta = 0.0;
  g.A = c.shapegt; g.lda = P.nge;
  g.B = c.udg + (long long)e0 * P.npe * P.nc; g.ldb = P.npe; g.N = P.nc * nb;
  g.C = c.wUG; g.ldc = P.nge;
  g.batch = 1; g.batch2 = 1;
  EXA_TRY(exa_gemm(g, c.st));
  A.ugpre = c.wUG;
  if (c.tdep) {
    g.B = c.sdg + (long long)e0 * P.npe * P.ncu; g.N = P.ncu * nb;
    g.C = c.wSG;
    EXA_TRY(exa_gemm(g, c.st));
    A.sgpre = c.wSG;
  }
  A.rgout = c.wRG;
  return EXA_OK;
}

// The FP64 volume blocks D and B of the chunk on the DMMA tensor cores: for each field c, the
// products T_(k,c) shapegt[:, :, 0] of all (element, k) pairs in one batched GEMM, written into
// the columns of D (c < ncu) or B, elements in parts of c.wT_elems (vol_mat_kernel's sums).
int volume_blocks_gemm(ExaCtx& c, int nb) {
  const ExaDims& P = c.P;
  const int npe = P.npe, nge = P.nge, ncu = P.ncu, nd = P.nd, n = P.n, nblk = P.ncu * P.nc;
  const long long nqn = (long long)npe * nd * ncu, blk = (long long)npe * nge;
  for (int le0 = 0; le0 < nb; le0 += c.wT_elems) {
    const int nbs = std::min(c.wT_elems, nb - le0);
    const long long tot = blk * nblk * nbs;
    vol_t_kernel<<<(unsigned)std::min<long long>((tot + 255) / 256, 8192), 256, 0, c.st>>>(P, c.shapegw, c.wRg, le0,
                                                                                         nbs, c.wT);
    EXA_LAUNCH_CHECK();
    std::vector<GemmBatch> gs;
    for (int cc = 0; cc < P.nc; ++cc) {
      GemmBatch g{};
      g.M = npe; g.N = npe; g.K = nge; g.alpha = 1.0; g.beta = 0.0;
      g.A = c.wT + (long long)ncu * cc * blk; g.lda = npe; g.sA = nblk * blk; g.sA2 = blk;
      g.B = c.shapegt; g.ldb = nge;
      if (cc < ncu) {
        g.C = c.wD + (long long)le0 * n * n + (long long)n * npe * cc;
        g.ldc = n; g.sC = (long long)n * n;
      } else {
        const int qc = cc - ncu, nq = qc % ncu, d = qc / ncu;
        g.C = c.wB + (long long)le0 * n * nqn + (long long)n * ((long long)npe * d + (long long)npe * nd * nq);
        g.ldc = n; g.sC = (long long)n * nqn;
      }
      g.sC2 = npe;  // trace component k: rows npe k
      g.batch = nbs; g.batch2 = ncu;
      gs.push_back(g);
    }
    for (size_t i = 0; i < gs.size(); i += EXA_GEMM_GROUP)
      EXA_TRY(exa_gemm_group(&gs[i], (int)std::min<size_t>(EXA_GEMM_GROUP, gs.size() - i), c.st));
  }
  return EXA_OK;
}

// Ru of the chunk = shapegw (npe x nge (nd + 1)) times the volume kernel's integrands
int volume_residual_gemm(ExaCtx& c, double* Ruc, int nb) {
  const ExaDims& P = c.P;
  GemmBatch g{};
  g.M = P.npe; g.K = P.nge * (P.nd + 1); g.N = P.ncu * nb; g.alpha = 1.0; g.beta = 0.0;
  g.A = c.shapegw; g.lda = P.npe;
  g.B = c.wRG; g.ldb = (long long)P.nge * (P.nd + 1);
  g.C = Ruc; g.ldc = P.npe;
  g.batch = 1; g.batch2 = 1;
  return exa_gemm(g, c.st);
}

}  // namespace

int exa_model_assemble(ExaCtx& c, bool jacobian) {
  const ExaDims& P = c.P;
  const int n = P.n, m = P.m;
  const long long nqn = (long long)P.npe * P.nd * P.ncu;
  if (!jacobian && c.tp_nslot) {
    ExaProfScope ps(c, EXA_PH_RESIDUAL);
    int rc = EXA_OK;
    if (launch_hdg_resid_tp<ExaModel>(make_args(c, 0), c.tensor, c.tp_nslot, c.Ru, c.Rh, c.st, &rc)) return rc;
  }
  const size_t vs = jacobian ? vol_points_smem<true>(P) : vol_points_smem<false>(P);
  const size_t fs = face_smem(P, jacobian);
  if (jacobian) {
    EXA_TRY(smem_attr((const void*)vol_points_kernel<ExaModel, true>, vs));
    EXA_TRY(smem_attr((const void*)face_kernel<ExaModel, true>, fs));
  } else {
    EXA_TRY(smem_attr((const void*)vol_points_kernel<ExaModel, false>, vs));
    EXA_TRY(smem_attr((const void*)face_kernel<ExaModel, false>, fs));
  }
  const int tpb_v = P.nge <= 64 ? 64 : (P.nge <= 128 ? 128 : 256);
  const int tpb_f = 128;
  for (int e0 = 0; e0 < P.ne; e0 += c.neb) {
    const int nb = std::min(c.neb, P.ne - e0);
    AsmArgs A = make_args(c, e0);
    double* Ruc = c.Ru + (long long)e0 * n;
    double* Rhc = c.Rh + (long long)e0 * m;
    if (jacobian) {
      {
        ExaProfScope ps(c, EXA_PH_VOLUME);
        if (c.wRG) EXA_TRY(volume_gauss_values(c, A, e0, nb));
        vol_points_kernel<ExaModel, true><<<nb, tpb_v, vs, c.st>>>(A, Ruc, c.wRg);
        EXA_LAUNCH_CHECK();
        if (c.wRG) EXA_TRY(volume_residual_gemm(c, Ruc, nb));
        // B straight into its packed FP32 form where the mixed form's q elimination takes it (the
        // face kernel adds its terms there too).  The volume kernel assigns every entry of B, so
        // only the layout's padding needs zeros, and nothing writes there after the zeroing at
        // allocation.
        const bool packed = c.precision == 1 && c.Sp.hi;
        UPacked bp{};
        if (packed && nqn > 0 && P.ncq > 0) {
          bp = c.wBp;
          A.Bp = c.wBp;
        }
        int rc = EXA_OK;
        if (packed) {
          EXA_TRY(exa_k_vol_mat_tc(P, c.shapegw32, c.Sp, c.wRg, c.wD, c.wB, bp, nb, c.d_uflag, c.st));
        } else if (exa_tensor_blocks(P, c.tensor) &&
                   launch_vol_blocks_tp(P, c.tensor, c.wRg, c.wD, c.wB, 0, tp_qelim(c) ? P.ncu : P.nc, nb, c.st, &rc)) {
          EXA_TRY(rc);
        } else if (c.wT) {
          EXA_TRY(volume_blocks_gemm(c, nb));
        } else {
          const int tiles = exa_ceil_div(P.npe, 64);
          dim3 grid(tiles * tiles, nb, P.ncu * P.nc);
          vol_mat_kernel<<<grid, 256, 0, c.st>>>(P, c.shapegw, c.shapegt, c.wRg, c.wD, c.wB);
          EXA_LAUNCH_CHECK();
        }
      }
      double* Hc = c.fp64_full ? c.H + (long long)e0 * m * m : c.H;
      {
        ExaProfScope ps(c, EXA_PH_FACE);
        // F, K and H of the chunk: the face kernel assigns their face blocks, at the same
        // positions at every assembly (face l's rows or columns, the same master-face node
        // lists for every element); the rest is structurally zero.  The plain form's products
        // overwrite these arrays, so it zeroes them each time; in the mixed form the products
        // only read them, and the zeros of the switch to that form (exa_ctx_set_precision) stay.
        // The tensor-product q elimination reads the face blocks of F, K and H only and assigns every
        // entry.
        const bool zero_blocks = c.precision != 1 && !tp_qelim(c);
        // Without q the products read F at those entries only and take H's other blocks as zero
        // (face_k); K's other entries are never written.  1000 p = 3 hexahedra of the Euler equations:
        // 5 GB not written, assembly 13.31 -> 12.59 ms.
        if (zero_blocks && (!c.face_k || c.k_given)) {
          EXA_CUDA(cudaMemsetAsync(c.wF, 0, sizeof(double) * (size_t)nb * n * m, c.st));
          EXA_CUDA(cudaMemsetAsync(c.wK, 0, sizeof(double) * (size_t)nb * m * n, c.st));
        }
        if (tp_qelim(c)) {
          A.fqout = c.wFq;
          c.b_pending = c.neb == P.ne;
        } else if (tp_trace(c)) {
          A.fqout = c.wFq;
        } else if (nqn > 0 && P.ncq > 0) {
          if (c.precision == 1 && c.wGp.hi) {
            // G written packed by the face kernel.  Each element slot gets the same entries
            // assigned at every assembly (face l's trace rows against face l's nodes, the same
            // master-face node lists for every element); the rest of G is structurally zero and
            // keeps the zeros of the allocation, since nothing else writes there.
            A.Gp = c.wGp;
          } else {
            EXA_CUDA(cudaMemsetAsync(c.wG, 0, sizeof(double) * (size_t)nb * m * nqn, c.st));
          }
        }
        if (zero_blocks && !c.face_k) EXA_CUDA(cudaMemsetAsync(Hc, 0, sizeof(double) * (size_t)nb * m * m, c.st));
        face_kernel<ExaModel, true><<<nb, tpb_f, fs, c.st>>>(A, Ruc, Rhc, c.wD, c.wB, c.wF, c.wK, c.wG, Hc);
        EXA_LAUNCH_CHECK();
      }
      EXA_TRY(c.precision == 1 ? schur_chunk_mixed(c, e0, nb) : schur_chunk(c, e0, nb));
      if (c.b_given) EXA_TRY(exa_model_form_b(c));
    } else {
      ExaProfScope ps(c, EXA_PH_RESIDUAL);
      if (c.wRG) EXA_TRY(volume_gauss_values(c, A, e0, nb));
      if (!launch_vol_pointwise<ExaModel>(A, nb, c.st))
        vol_points_kernel<ExaModel, false><<<nb, tpb_v, vs, c.st>>>(A, Ruc, nullptr);
      EXA_LAUNCH_CHECK();
      if (c.wRG) EXA_TRY(volume_residual_gemm(c, Ruc, nb));
      face_kernel<ExaModel, false><<<nb, tpb_f, fs, c.st>>>(A, Ruc, Rhc, nullptr, nullptr, nullptr, nullptr, nullptr,
                                                           nullptr);
      EXA_LAUNCH_CHECK();
    }
  }
  return EXA_OK;
}

bool exa_model_getq_tp(ExaCtx& c, int* rc) {
  return c.tp_nslot && launch_getq_tp(c.P, c.tensor, c.tp_nslot, c.perm, c.elemcon, c.elemg, c.faceg, c.uh, c.udg, c.st, rc);
}

bool exa_model_has_getq_tp(const ExaDims& P, const ExaTensor& t) { return P.ncq > 0 && getq_tp_fits(P, t); }

// the mixed form's volume kernel then packs B itself, so neither form stores B and G
bool exa_model_qelim_tp(const ExaDims& P, const ExaTensor& t) {
  return exa_tensor_blocks(P, t) && qelim_tp_fits(P, t) && exa_vol_mat_tc_fits(P);
}

int exa_model_form_b(ExaCtx& c) {
  const ExaDims& P = c.P;
  int rc = EXA_OK;
  if (!c.b_pending || !c.wB) return EXA_OK;
  c.b_pending = false;
  if (!launch_vol_blocks_tp(P, c.tensor, c.wRg, c.wD, c.wB, P.ncu, P.nc, P.ne, c.st, &rc))
    return EXA_OK;
  EXA_TRY(rc);
  face_b_kernel<<<P.ne, 128, 0, c.st>>>(P, c.shapfgt, c.shapfgw, c.perm, c.wFq, c.wB);
  EXA_LAUNCH_CHECK();
  return EXA_OK;
}

bool exa_model_has_ldg_boundary() { return ExaModel::has_ldg_boundary; }

namespace {

LdgArgs ldg_args(const ExaCtx& c, const double* u) {
  LdgArgs L{};
  L.P = c.P;
  L.shapfgt = c.shapfgt; L.shapfgw = c.shapfgw; L.shapfnt = c.shapfnt;
  L.f2e = c.f2e; L.perm = c.perm; L.bf = c.bf; L.fcon = c.ldg_fcon;
  L.xdg = c.xdg; L.faceg = c.faceg; L.uinf = c.uinf; L.param = c.param; L.tau = c.tau;
  L.ntau = c.ntau; L.modelnumber = c.modelnumber; L.time = c.time;
  L.u = u; L.Rh = c.ldg_Rh;
  return L;
}

// the general face kernel over faces f0 .. nf - 1
int ldg_faces_general(const ExaCtx& c, LdgArgs L, int f0) {
  if (c.P.nf <= f0) return EXA_OK;
  const size_t fs = ldg_face_smem(c.P);
  EXA_TRY(smem_attr((const void*)ldg_face_kernel<ExaModel>, fs));
  L.f0 = f0;
  ldg_face_kernel<ExaModel><<<c.P.nf - f0, 64, fs, c.st>>>(L);
  EXA_LAUNCH_CHECK();
  return EXA_OK;
}

// out = U.cr R(u) + U.c0 U.R0 (or R(u)) by the tensor-product kernels; false where they do not apply.
// Boundary faces take their states from L.u alone, so U.v is given on meshes without them only.
bool ldg_residual_tp(ExaCtx& c, const LdgState& U, double* out, int* rc) {
  if (!c.ldg_fslot || !c.ldg_split) return false;
  struct Boundary {
    ExaCtx& c;
    LdgArgs L;
  } b{c, ldg_args(c, U.u)};
  auto boundary = [](void* p) -> int {
    Boundary& q = *static_cast<Boundary*>(p);
    return ldg_faces_general(q.c, q.L, q.c.P.nf0);
  };
  return launch_ldg_tp<ExaModel>(b.L, make_args(c, 0), U, c.tensor, c.tp_nslot, c.ldg_fslot, out, c.st, boundary, &b,
                                 rc);
}

}  // namespace

// The LDG residual of the element states u (the layout of udg: nc = ncu without q): the volume
// integrals of the HDG residual (RuElem, uresidual.cpp:45-130, is the same quadrature), the
// face residuals of every face, and their sum into the elements with the sign and scaling of
// Residual (residual.cpp:589-617).
int exa_model_ldg_residual(ExaCtx& c, const double* u, double* Ru) {
  const ExaDims& P = c.P;
  ExaProfScope ps(c, EXA_PH_RESIDUAL);
  int rc = EXA_OK;
  if (ldg_residual_tp(c, LdgState{u, nullptr, nullptr, 0.0, 1.0, 0.0}, Ru, &rc)) return rc;
  double* saved = c.udg;
  c.udg = const_cast<double*>(u);
  auto body = [&]() -> int {
    const size_t vs = vol_points_smem<false>(P);
    EXA_TRY(smem_attr((const void*)vol_points_kernel<ExaModel, false>, vs));
    const int tpb_v = P.nge <= 64 ? 64 : (P.nge <= 128 ? 128 : 256);
    for (int e0 = 0; e0 < P.ne; e0 += c.neb) {
      const int nb = std::min(c.neb, P.ne - e0);
      AsmArgs A = make_args(c, e0);
      double* Ruc = c.Ru + (long long)e0 * P.n;
      if (c.wRG) EXA_TRY(volume_gauss_values(c, A, e0, nb));
      if (!launch_vol_pointwise<ExaModel>(A, nb, c.st))
        vol_points_kernel<ExaModel, false><<<nb, tpb_v, vs, c.st>>>(A, Ruc, nullptr);
      EXA_LAUNCH_CHECK();
      if (c.wRG) EXA_TRY(volume_residual_gemm(c, Ruc, nb));
    }
    LdgArgs L = ldg_args(c, u);
    // interior faces by the pointwise kernel where the model's (nd, ncu) has one, the boundary
    // faces (and otherwise all) by the general one
    int fgen = 0;
    if (c.ldg_split && launch_ldg_face_inner<ExaModel>(L, P.nf0, c.st)) {
      EXA_LAUNCH_CHECK();
      fgen = P.nf0;
    }
    EXA_TRY(ldg_faces_general(c, L, fgen));
    return exa_k_ldg_gather(P, c.f2e, c.perm, c.elemcon, c.Ru, c.ldg_Rh, Ru, c.tdep, c.dtfactor, c.st);
  };
  const int st = body();
  c.udg = saved;
  return st;
}

int exa_model_ldg_jv(ExaCtx& c, const double* v, double* w) {
  const long long N = c.sysN();
  const double eps = c.matvec_eps;
  const bool bnd = c.P.nf > c.P.nf0;
  if (bnd) EXA_TRY(exa_lincomb(c.ldg_w, 1.0, c.udg, eps, v, N, c.st));
  {
    ExaProfScope ps(c, EXA_PH_RESIDUAL);
    LdgState U{c.udg, v, c.ldg_R, eps, 1.0 / eps, -1.0 / eps};
    if (bnd) {
      U.u = c.ldg_w;
      U.v = nullptr;
    }
    int rc = EXA_OK;
    if (ldg_residual_tp(c, U, w, &rc)) return rc;
  }
  if (!bnd) EXA_TRY(exa_lincomb(c.ldg_w, 1.0, c.udg, eps, v, N, c.st));
  EXA_TRY(exa_model_ldg_residual(c, c.ldg_w, c.ldg_Rw));
  return exa_lincomb(w, 1.0 / eps, c.ldg_Rw, -1.0 / eps, c.ldg_R, N, c.st);
}

// initial u from the model's cpuInitu at the element nodes (readsolstruct, readbinaryfiles.cpp:546-556)
int exa_model_init_udg(ExaCtx& c, double* host_udg) {
  const ExaDims& P = c.P;
  const int np = P.npe * P.ne;
  std::vector<double> f((size_t)np * P.nc, 0.0);
  EXA_MODEL_NS::cpuInitu(f.data(), c.h_xdg.data(), c.h_uinf.data(), c.h_param.data(), c.modelnumber, np, P.ncx,
                         P.nc, P.npe, P.ne);
  for (int e = 0; e < P.ne; ++e)
    for (int k = 0; k < P.ncu; ++k)
      for (int i = 0; i < P.npe; ++i)
        host_udg[i + P.npe * k + P.npe * P.nc * e] = f[i + P.npe * k + (size_t)P.npe * P.nc * e];
  return EXA_OK;
}
