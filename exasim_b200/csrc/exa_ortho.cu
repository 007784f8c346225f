// Gram-Schmidt of the Krylov loop: one vector against the basis, two passes over the basis.
//
// Modified Gram-Schmidt takes h_k = <v_k, w - sum_{j<k} h_j v_j> one basis vector at a time
// (Exasim's MGS, backend/Solver/getpoly.cpp:36-45), which reads and writes w for every vector
// and orders k launches one after another.  Expanding the bracket, h solves
//   (I + L) h = V^T w,   L_kj = <v_k, v_j> for j < k  (strictly lower triangular),
// the triangular form of the same recurrence (Bjorck 1967; Swirydowicz, Langou, Ananthan, Yang,
// Thomas 2020): the coefficients, and the loss of orthogonality, are those of MGS up to rounding,
// but all products with w come from one pass over V and the update from a second.  Row k of L
// needs <v_k, v_j>, which the same pass forms when v_k is the newest basis vector.  Panels of OP
// vectors bound the triangle; between panels w is updated, as MGS does.
//
// Bound: HBM (or L2) reads of V, 2 n k doubles per step against 4 n k of a launch per vector; for
// short vectors the launches, 1 or 3 against k + 2.  Three forms of one reduction order per size:
// vectors up to OC_MAX_N entries run in one thread-block cluster that keeps w in registers (one
// launch, partial sums through distributed shared memory), longer ones as three launches over the
// GPU.  Every sum has a fixed partition and order, so results do not depend on scheduling.
// Measured (B200, before: one launch per vector): 4800 unknowns, restart 50, 245 steps of a served
// 2D solve 22.9 -> 5.2 ms for the call, with the face-by-face operator (face_op_kernel) at the same time;
// 553k unknowns, restart 50, 150 steps of an LDG solve 41.9 -> 23.5 ms.
#include <cooperative_groups.h>

#include <algorithm>
#include <utility>

#include "exa_common.cuh"

namespace cg = cooperative_groups;

namespace {
constexpr int OP = EXA_ORTHO_PANEL;  // basis vectors per panel
constexpr int OT = 256;              // threads of the whole-GPU kernels
constexpr int OB = EXA_ORTHO_BLOCKS; // their blocks: two per SM
constexpr int OCT = 512;             // threads of a cluster's CTAs
constexpr int OC_MAX = 8;            // CTAs of a cluster (the portable limit)
// one cluster reads V at the L2 rate of 8 SMs, about 1 TB/s: at 16384 entries and 25 vectors that is
// 3 us a pass, what the two extra launches of the whole-GPU form cost
constexpr long long OC_MAX_N = 16384;

// Sums NV values per lane over the warp by halving exchanges (NV - 1 + the remaining butterfly
// shuffles instead of 5 NV): lane l ends with the total of value idx(l).
template <int NV>
__device__ __forceinline__ double warp_sum_many(double (&v)[NV], int lane) {
  int off = 16;
#pragma unroll
  for (int m = NV / 2; m >= 1; m >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int t = 0; t < m; ++t) {
      const double send = up ? v[t] : v[t + m];
      const double keep = up ? v[t + m] : v[t];
      v[t] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    off >>= 1;
  }
  double s = v[0];
  for (; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
  return s;
}
template <int NV>
__device__ __forceinline__ int warp_sum_index(int lane) {
  return NV == 16 ? lane >> 1 : lane >> 2;
}
template <int NV>
__device__ __forceinline__ bool warp_sum_owner(int lane) {
  return NV == 16 ? (lane & 1) == 0 : (lane & 3) == 0;
}

// acc[2 j] += <w, V_j>, acc[2 j + 1] += <u, V_j> over this thread's R rows r0 + q stride (the
// first `rows` of them inside the range), j < kp; acc is the warp's own.  The loads of JG vectors
// are in flight at once.
template <int R>
__device__ __forceinline__ void panel_dots(const double* V, long long n, int kp, long long r0, int stride, int rows,
                                           const double (&w)[R], const double (&u)[R], double* acc, int lane) {
  constexpr int JG = R <= 4 ? 8 : 4, NV = 2 * JG;
  for (int j0 = 0; j0 < kp; j0 += JG) {
    double t[JG][R];
#pragma unroll
    for (int g = 0; g < JG; ++g)
#pragma unroll
      for (int q = 0; q < R; ++q)
        t[g][q] = (j0 + g < kp && q < rows) ? V[n * (j0 + g) + r0 + (long long)q * stride] : 0.0;
    double v[NV];
#pragma unroll
    for (int g = 0; g < JG; ++g) {
      double a = 0.0, b = 0.0;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        a = fma(w[q], t[g][q], a);
        b = fma(u[q], t[g][q], b);
      }
      v[2 * g] = a;
      v[2 * g + 1] = b;
    }
    const double s = warp_sum_many<NV>(v, lane);
    if (warp_sum_owner<NV>(lane)) {
      const int at = 2 * j0 + warp_sum_index<NV>(lane);
      if (at < 2 * kp) acc[at] += s;
    }
  }
}

// w_q += sgn h_j V_j over this thread's rows, vector by vector
template <int R>
__device__ __forceinline__ void panel_update(const double* V, long long n, int kp, long long r0, int stride, int rows,
                                             const double* h, double sgn, double (&w)[R]) {
  constexpr int JG = R <= 4 ? 8 : 4;
  for (int j0 = 0; j0 < kp; j0 += JG) {
    double t[JG][R];
#pragma unroll
    for (int g = 0; g < JG; ++g)
#pragma unroll
      for (int q = 0; q < R; ++q)
        t[g][q] = (j0 + g < kp && q < rows) ? V[n * (j0 + g) + r0 + (long long)q * stride] : 0.0;
#pragma unroll
    for (int g = 0; g < JG; ++g) {
      const double hg = j0 + g < kp ? sgn * h[j0 + g] : 0.0;
#pragma unroll
      for (int q = 0; q < R; ++q) w[q] = fma(hg, t[g][q], w[q]);
    }
  }
}

// g <- (I + L)^-1 g, g[2 j] in shared memory, L column-major with leading dimension OP in shared
// memory; one warp, lane l holds rows l and l + 32.  The result goes to h[0 .. kp).
__device__ __forceinline__ void forward_solve(const double* g, const double* Ls, int kp, double* h, int lane) {
  static_assert(OP == 64, "two rows per lane");
  double a = lane < kp ? g[2 * lane] : 0.0, b = lane + 32 < kp ? g[2 * (lane + 32)] : 0.0;
  for (int j = 0; j < kp; ++j) {
    const double hj = __shfl_sync(0xffffffffu, j < 32 ? a : b, j & 31);
    if (lane > j) a = fma(-Ls[j * OP + lane], hj, a);
    if (lane + 32 > j) b = fma(-Ls[j * OP + lane + 32], hj, b);
  }
  if (lane < kp) h[lane] = a;
  if (lane + 32 < kp) h[lane + 32] = b;
}

// cpuApplyGivensRotation (backend/Common/cpuimpl.h:167-196) on column i of the Hessenberg
// matrix, by one block: the old rotations come through shared memory in chunks, one thread
// applies them.  H[0 .. i] and hn = H[i + 1] are ready; *rel and *rel_host get |s[i + 1]| / nrmb.
__device__ __forceinline__ void givens_column(const ExaGivens& G, int i, double* H, double hn, double* sh) {
  constexpr int C = 64;
  const int tid = threadIdx.x;
  double carry = H[0];
  for (int b = 0; b < i; b += C) {
    const int cnt = min(C, i - b);
    if (tid < cnt) {
      sh[tid] = H[b + tid + 1];
      sh[C + tid] = G.cs[b + tid];
      sh[2 * C + tid] = G.sn[b + tid];
    }
    __syncthreads();
    if (tid == 0) {
      for (int k = 0; k < cnt; ++k) {
        const double c = sh[C + k], s = sh[2 * C + k], next = sh[k];
        sh[k] = c * carry + s * next;
        carry = -s * carry + c * next;
      }
    }
    __syncthreads();
    if (tid < cnt) H[b + tid] = sh[tid];
    __syncthreads();
  }
  if (tid != 0) return;
  double c, s;
  if (hn == 0.0) {
    c = 1.0;
    s = 0.0;
  } else if (fabs(hn) > fabs(carry)) {
    const double t = carry / hn;
    s = 1.0 / sqrt(1.0 + t * t);
    c = t * s;
  } else {
    const double t = hn / carry;
    c = 1.0 / sqrt(1.0 + t * t);
    s = t * c;
  }
  G.cs[i] = c;
  G.sn[i] = s;
  const double si = G.s[i], sn1 = -s * si;
  G.s[i + 1] = sn1;
  G.s[i] = c * si;
  H[i] = c * carry + s * hn;
  H[i + 1] = 0.0;
  const double rel = fabs(sn1) / *G.nrmb;
  *G.rel = rel;
  *G.rel_host = rel;
}

// the panel's part of the whole-GPU kernels' rows: block b takes rows [b rpb, (b + 1) rpb)
template <int R>
__global__ void __launch_bounds__(OT, 2)
    ortho_dots_kernel(const double* V, const double* w, const double* u, long long n, int kp, long long rpb,
                      double* part, unsigned* ticket, double* L, double* h, double* hcol) {
  __shared__ double acc[OT / 32][2 * OP];
  __shared__ double Ls[OP * OP];
  __shared__ double tot[2 * OP];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int t = lane; t < 2 * OP; t += 32) acc[warp][t] = 0.0;
  __syncwarp();
  const long long end = min(n, (blockIdx.x + 1) * rpb);
  for (long long base = blockIdx.x * rpb; base < end; base += (long long)OT * R) {
    const long long r0 = base + tid;
    const int rows = r0 < end ? (int)min((long long)R, (end - r0 + OT - 1) / OT) : 0;
    double wr[R], ur[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      wr[q] = q < rows ? w[r0 + (long long)q * OT] : 0.0;
      ur[q] = (u && q < rows) ? u[r0 + (long long)q * OT] : 0.0;
    }
    panel_dots<R>(V, n, kp, r0, OT, rows, wr, ur, acc[warp], lane);
  }
  __syncthreads();
  for (int t = tid; t < 2 * kp; t += OT) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < OT / 32; ++q) s += acc[q][t];
    part[(size_t)t * gridDim.x + blockIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the last block adds the partial sums in block order and solves for h
  for (int t = tid; t < OP * OP; t += OT)
    if (t / OP < kp && t % OP < kp) Ls[t] = L[t];
  for (int t = warp; t < 2 * kp; t += OT / 32) {
    double s = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(part + (size_t)t * gridDim.x + b);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) tot[t] = s;
  }
  __syncthreads();
  if (u)  // the newest vector's row of L
    for (int j = tid; j < kp - 1; j += OT) Ls[j * OP + kp - 1] = L[j * OP + kp - 1] = tot[2 * j + 1];
  __syncthreads();
  if (warp == 0) {
    forward_solve(tot, Ls, kp, h, lane);
    __syncwarp();
    for (int j = lane; j < kp; j += 32) hcol[j] = h[j];
  }
  if (tid == 0) *ticket = 0u;
}

// w += sgn V h on the block's rows.  With hnext, the norm of the result goes there (the last
// block, in block order) and the Givens update of the Hessenberg column follows.
template <int R>
__global__ void __launch_bounds__(OT, 2)
    ortho_update_kernel(const double* V, double* w, long long n, int kp, long long rpb, const double* h, double sgn,
                        double* part, unsigned* ticket, double* hnext, ExaGivens G, int i, double* hcol) {
  __shared__ double hs[OP];
  __shared__ double red[OT / 32];
  __shared__ double sh[3 * 64];
  __shared__ double hn;
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < kp) hs[tid] = h[tid];
  __syncthreads();
  double ss = 0.0;
  const long long beg = blockIdx.x * rpb, end = min(n, beg + rpb), step = (long long)OT * R;
  // tiles from the end of the range: the first pass read them last, so they are still in L2
  for (long long base = beg + (end > beg ? (end - 1 - beg) / step * step : -step); base >= beg; base -= step) {
    const long long r0 = base + tid;
    const int rows = r0 < end ? (int)min((long long)R, (end - r0 + OT - 1) / OT) : 0;
    double wr[R];
#pragma unroll
    for (int q = 0; q < R; ++q) wr[q] = q < rows ? w[r0 + (long long)q * OT] : 0.0;
    panel_update<R>(V, n, kp, r0, OT, rows, hs, sgn, wr);
#pragma unroll
    for (int q = 0; q < R; ++q)
      if (q < rows) {
        w[r0 + (long long)q * OT] = wr[q];
        ss = fma(wr[q], wr[q], ss);
      }
  }
  if (!hnext) return;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if (lane == 0) red[warp] = ss;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < OT / 32; ++q) s += red[q];
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp == 0) {
    double s = 0.0;
    for (int b = lane; b < (int)gridDim.x; b += 32) s += __ldcg(part + b);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) {
      hn = sqrt(s);
      *hnext = hn;
      G.inv[0] = 1.0 / hn;
      *ticket = 0u;
    }
  }
  __syncthreads();
  if (G.cs) givens_column(G, i, hcol, hn, sh);
}

__global__ void __launch_bounds__(OT) ortho_scale_kernel(double* w, const double* inv, long long n) {
  const double r = *inv;
  const long long stride = (long long)gridDim.x * OT;
  long long i = blockIdx.x * (long long)OT + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {
    double a[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) a[q] = w[i + q * stride];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[i + q * stride] = a[q] * r;
  }
  for (; i < n; i += stride) w[i] *= r;
}

// The whole step in one cluster: CTA c of the cluster keeps rows [c rpc, (c + 1) rpc) of w (and
// of the newest basis vector) in registers; each CTA writes its partial sums into every CTA's
// shared memory, and after one cluster barrier all of them add these in CTA order and solve the
// same triangle.  The exchange buffer alternates, so one barrier per panel is enough.
constexpr int OC_SMEM = sizeof(double) * (OCT / 32 * 2 * OP + 2 * OC_MAX * 2 * OP + OP * OP + 2 * OP + OP + OC_MAX + 3 * 64);
template <int R>
__global__ void __launch_bounds__(OCT, 1)
    ortho_cluster_kernel(const double* V, double* w, long long n, int k, long long rpc, double* L, double* hcol,
                         ExaGivens G) {
  extern __shared__ double osm[];
  double* acc = osm;                          // [warps][2 OP]
  double* xch = acc + OCT / 32 * 2 * OP;      // [2][OC_MAX][2 OP]
  double* Ls = xch + 2 * OC_MAX * 2 * OP;     // [OP][OP]
  double* tot = Ls + OP * OP;                 // [2 OP]
  double* hs = tot + 2 * OP;                  // [OP]
  double* xn = hs + OP;                       // [OC_MAX]
  double* sh = xn + OC_MAX;                   // [3 64]
  cg::cluster_group cl = cg::this_cluster();
  auto started = cl.barrier_arrive();  // before the first write into another CTA's shared memory
  const int rank = (int)cl.block_rank(), nc = (int)cl.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long beg = rank * rpc, end = min(n, beg + rpc), r0 = beg + tid;
  const int rows = r0 < end ? (int)min((long long)R, (end - r0 + OCT - 1) / OCT) : 0;
  const double* vi = V + n * (k - 1);
  double wr[R], ur[R];
#pragma unroll
  for (int q = 0; q < R; ++q) {
    wr[q] = q < rows ? w[r0 + (long long)q * OCT] : 0.0;
    ur[q] = q < rows ? vi[r0 + (long long)q * OCT] : 0.0;
  }
  for (int p = 0; p * OP < k; ++p) {
    const int kp = min(OP, k - p * OP);
    const bool newest = p * OP + kp == k;
    const double* Vp = V + n * (long long)(p * OP);
    double* Lp = L + (long long)p * OP * OP;
    for (int t = lane; t < 2 * kp; t += 32) acc[warp * 2 * OP + t] = 0.0;
    for (int t = tid; t < OP * kp; t += OCT)
      if (t % OP < kp) Ls[t] = Lp[t];  // rows below the newest, from earlier steps
    __syncwarp();
    panel_dots<R>(Vp, n, kp, r0, OCT, rows, wr, ur, acc + warp * 2 * OP, lane);
    __syncthreads();
    if (p == 0) cl.barrier_wait(std::move(started));
    double* xp = xch + (p & 1) * OC_MAX * 2 * OP;
    for (int t = tid; t < 2 * kp; t += OCT) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < OCT / 32; ++q) s += acc[q * 2 * OP + t];
      for (int c = 0; c < nc; ++c) *cl.map_shared_rank(xp + rank * 2 * OP + t, c) = s;
    }
    cl.sync();
    for (int t = tid; t < 2 * kp; t += OCT) {
      double s = 0.0;
      for (int c = 0; c < nc; ++c) s += xp[c * 2 * OP + t];
      tot[t] = s;
      if (newest && (t & 1) && t / 2 < kp - 1) {
        Ls[(t / 2) * OP + kp - 1] = s;
        if (rank == 0) Lp[(t / 2) * OP + kp - 1] = s;
      }
    }
    __syncthreads();
    if (warp == 0) forward_solve(tot, Ls, kp, hs, lane);
    __syncthreads();
    panel_update<R>(Vp, n, kp, r0, OCT, rows, hs, -1.0, wr);
    if (rank == 0 && tid < kp) hcol[p * OP + tid] = hs[tid];
  }
  double ss = 0.0;
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (q < rows) ss = fma(wr[q], wr[q], ss);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  __syncthreads();
  if (lane == 0) tot[warp] = ss;
  __syncthreads();
  if (tid < nc) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < OCT / 32; ++q) s += tot[q];
    *cl.map_shared_rank(xn + rank, tid) = s;
  }
  cl.sync();
  double s = 0.0;
  for (int c = 0; c < nc; ++c) s += xn[c];
  const double hn = sqrt(s), inv = 1.0 / hn;
#pragma unroll
  for (int q = 0; q < R; ++q)
    if (q < rows) w[r0 + (long long)q * OCT] = wr[q] * inv;
  if (rank != 0) return;
  if (tid == 0) hcol[k] = hn;
  __syncthreads();
  if (G.cs) givens_column(G, k - 1, hcol, hn, sh);
}

// blocks and rows per block of the whole-GPU kernels, and their rows per thread
struct Split {
  int blocks, r;
  long long rpb;
};
Split split_rows(long long n) {
  Split s;
  const long long g = std::min<long long>(OB, (n + OT - 1) / OT);
  s.rpb = ((n + g - 1) / g + 31) / 32 * 32;
  s.blocks = (int)((n + s.rpb - 1) / s.rpb);
  s.r = (int)std::min<long long>(8, (s.rpb + OT - 1) / OT);
  return s;
}

#define EXA_BY_ROWS(r, CALL)  \
  do {                        \
    if ((r) <= 1) CALL(1);    \
    else if ((r) <= 2) CALL(2); \
    else if ((r) <= 3) CALL(3); \
    else if ((r) <= 4) CALL(4); \
    else if ((r) <= 5) CALL(5); \
    else if ((r) <= 6) CALL(6); \
    else CALL(8);             \
  } while (0)

int update_panel(const double* V, double* w, long long n, int kp, const Split& s, const double* h, double sgn,
                 double* part, unsigned* ticket, double* hnext, const ExaGivens& G, int i, double* hcol,
                 cudaStream_t st) {
#define EXA_CALL(R) \
  ortho_update_kernel<R><<<s.blocks, OT, 0, st>>>(V, w, n, kp, s.rpb, h, sgn, part, ticket, hnext, G, i, hcol)
  EXA_BY_ROWS(s.r, EXA_CALL);
#undef EXA_CALL
  EXA_LAUNCH_CHECK();
  return EXA_OK;
}
}  // namespace

size_t exa_ortho_work(int restart) {
  const size_t panels = ((size_t)restart + OP) / OP;
  return panels * OP * OP + (size_t)2 * OP * OB + OP + 4;
}

int exa_mgs(double* w, const double* V, long long n, int k, double* hcol, double* work, int restart,
            const ExaGivens* givens, cudaStream_t st) {
  if (n <= 0 || k <= 0) return EXA_OK;
  double* L = work;
  double* part = L + (((size_t)restart + OP) / OP) * OP * OP;
  double* h = part + (size_t)2 * OP * OB;
  ExaGivens G = givens ? *givens : ExaGivens{};
  G.inv = h + OP;
  unsigned* ticket = reinterpret_cast<unsigned*>(h + OP + 1);  // zero between launches
  if (n <= OC_MAX_N) {
    // as many CTAs as give each at least 512 rows, up to 8
    int nc = 1;
    while (nc < OC_MAX && n > (long long)nc * OCT) nc *= 2;
    const long long rpc = ((n + nc - 1) / nc + 31) / 32 * 32;
    const int r = (int)((rpc + OCT - 1) / OCT);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nc);
    cfg.blockDim = dim3(OCT);
    cfg.dynamicSmemBytes = OC_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = nc;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
#define EXA_CALL(R)                                                                                     \
  do {                                                                                                  \
    EXA_TRY(exa_allow_smem((const void*)ortho_cluster_kernel<R>, OC_SMEM));                             \
    EXA_CUDA(cudaLaunchKernelEx(&cfg, ortho_cluster_kernel<R>, V, w, n, k, rpc, L, hcol, G));           \
  } while (0)
    if (r <= 1) EXA_CALL(1);
    else if (r <= 2) EXA_CALL(2);
    else EXA_CALL(4);
#undef EXA_CALL
    EXA_LAUNCH_CHECK();
    return EXA_OK;
  }
  const Split s = split_rows(n);
  for (int p = 0; p * OP < k; ++p) {
    const int kp = std::min(OP, k - p * OP);
    const bool newest = p * OP + kp == k;
    const double* Vp = V + n * (long long)(p * OP);
    const double* u = newest ? V + n * (long long)(k - 1) : nullptr;
#define EXA_CALL(R)                                                                                               \
  ortho_dots_kernel<R><<<s.blocks, OT, 0, st>>>(Vp, w, u, n, kp, s.rpb, part, ticket, L + (long long)p * OP * OP, h, \
                                                hcol + p * OP)
    EXA_BY_ROWS(s.r, EXA_CALL);
#undef EXA_CALL
    EXA_LAUNCH_CHECK();
    EXA_TRY(update_panel(Vp, w, n, kp, s, h, -1.0, part, ticket + 1, newest ? hcol + k : nullptr, G, k - 1, hcol, st));
  }
  ortho_scale_kernel<<<s.blocks, OT, 0, st>>>(w, G.inv, n);
  EXA_LAUNCH_CHECK();
  return EXA_OK;
}

int exa_gemv_add(double* x, const double* V, const double* y, long long n, int k, cudaStream_t st) {
  if (k <= 0 || n <= 0) return EXA_OK;
  const Split s = split_rows(n);
  for (int p = 0; p * OP < k; ++p)
    EXA_TRY(update_panel(V + n * (long long)(p * OP), x, n, std::min(OP, k - p * OP), s, y + p * OP, 1.0, nullptr,
                         nullptr, nullptr, ExaGivens{}, 0, nullptr, st));
  return EXA_OK;
}
