// BP-gauge truncation of every edge, FP64 on the device, one block per edge.
//
// Follows truncation.h:57-219 and SquareRootAndInverse (root.h:66-148):
//   M_a = E[m] (computed at site a), M_b = E[m + ne]
//   M = U diag(s) Vh                        (SVD, descending s)
//   R = U diag(sqrt s  | s > sv_min) Vh
//   S = Vh^H diag(1/sqrt s | sqrt s > sqrt sv_min) U^H
//   T = R_a^T R_b / ||R_a^T R_b||_F
//   T = X diag(s) Y, keep s_i > sv_min, at most chi_max, at least one
//   P_a = S_a^T X diag(sqrt s)   (D x chi, applied to V_a's leg)
//   P_b = (diag(sqrt s) Y S_b)^T (D x chi, applied to V_b's leg)
//   E[m] = E[m + ne] = diag(s)
// The SVD is a one-sided (Hestenes) Jacobi SVD: column pairs are rotated in
// a round-robin order, 16 lanes per pair, until no pair is rotated; the
// sweep count is bounded and a non-converged edge is reported, never spun on.
//
// What bounds it: a serial chain (about 8 sweeps of n - 1 rounds, each a dot
// product, a reduction and two reciprocal square roots before the columns
// can be rotated and the next round may start).  So the matrices stay in
// shared memory, a round's pairs all run at once, both columns and the
// rotation's columns of V are held in registers, the rotation needs two
// rsqrt instead of three square roots and four divisions, and the two
// messages of an edge are decomposed by two CTAs before a third SVD joins
// them.  Per launch, before (one warp per pair, matrices in global memory,
// the three SVDs in one CTA) and after: 264 edges at D = 32 4.34 -> 1.38 ms,
// 40 edges at D = 64 18.8 -> 3.9 ms, 49 edges at D <= 16 0.27 -> 0.08 ms.
#pragma once
#include "kernels.cuh"

namespace tnbp {

struct TruncTask {
  const void* Ma;   // D x D, storage precision
  const void* Mb;
  int D;
  double2* work;    // 8 * D * D scratch: R_a, S_a^T, R_b, S_b^T and four matrices of the large-D path
  void* Pa;         // D x D capacity, storage precision (first keep columns valid)
  void* Pb;
  double* s_keep;   // D: kept singular values of T
  int* keep_out;
  double* err_out;
  int* status;      // 3 values (SVDs of Ma, Mb, T): 0 ok, 1 SVD sweep limit reached, 2 non-finite values
};

constexpr int kTruncSmemMaxD = 80;  // two D x (D | 1) matrices in shared memory: 203 KB
constexpr int kTruncMaxD = 128;     // as every leg contraction
__host__ __device__ inline size_t trunc_smem_bytes(int max_d) {
  const int d = max_d < kTruncSmemMaxD ? max_d : kTruncSmemMaxD;
  return (size_t)2 * d * (d | 1) * sizeof(double2) + (size_t)max_d * (3 * sizeof(double) + sizeof(int)) + 16;
}
// 16 lanes per column pair: D = 16 fills 128 threads, D = 32 256, above that
// 512 (D = 64 has 32 pairs).
__host__ __device__ inline int trunc_threads(int max_d) { return max_d <= 16 ? 128 : max_d <= 32 ? 256 : 512; }

// One-sided Jacobi on the n x n matrix A (column-major, leading dimension
// ld); V accumulates the rotations so that A_in = A_out * V^H.  Returns
// sweeps used, -1 if the sweep limit was reached.  n <= 16 NR rows are held
// as NR registers per lane; larger n walk their rows in memory (NR = 0).
template <int NR>
__device__ __forceinline__ int block_jacobi(double2* A, double2* V, int n, int ld, int* flag, double* red) {
  double fro = 0.0;
  for (int i = threadIdx.x; i < n * n; i += blockDim.x) {
    const int r = i % n, c = i / n;
    V[r + ld * c] = r == c ? make_double2(1.0, 0.0) : make_double2(0.0, 0.0);
    fro += abs2(A[r + ld * c]);
  }
  fro = block_sum(fro, red);
  const int np = n + (n & 1), half = np / 2;
  const int ngrp = blockDim.x >> 4, grp = threadIdx.x >> 4, lane = threadIdx.x & 15;
  // Pairs count as orthogonal once |a_i^H a_j| <= n eps |a_i| |a_j|: the
  // rounding of the dot product itself is about sqrt(n) eps, so a tighter
  // threshold could keep rotating noise forever.  A column whose norm is at
  // the rounding level of the matrix (<= n eps ||A||_F) is numerically zero
  // and is not rotated (its singular value is noise, far below any cut).
  const double eps = 2.220446049250313e-16;
  const double tol = eps * (double)max(n, 8);
  const double tol2 = tol * tol, zero2 = tol2 * fro;
  constexpr int kReg = NR > 0 ? NR : 1;
  for (int sweep = 0; sweep < kSvdMaxSweeps; ++sweep) {
    __syncthreads();
    if (threadIdx.x == 0) *flag = 0;
    __syncthreads();
    bool rotated = false;
    for (int round = 0; round < np - 1; ++round) {
      for (int p0 = 0; p0 < half; p0 += ngrp) {
        const int pi = p0 + grp;
        int a = np - 1, b = round;
        if (pi > 0) {
          a = round + pi;
          b = round - pi;
          if (a >= np - 1) a -= np - 1;
          if (b < 0) b += np - 1;
        }
        const bool act = pi < half && a < n && b < n;
        const int i = act ? min(a, b) : 0, j = act ? max(a, b) : 0;
        double2* ai = A + ld * i;
        double2* aj = A + ld * j;
        double2 x[kReg], y[kReg];
        double al = 0.0, be = 0.0;
        double2 ga = make_double2(0.0, 0.0);
        if constexpr (NR > 0) {
#pragma unroll
          for (int k = 0; k < NR; ++k) {
            const int r = lane + 16 * k;
            x[k] = y[k] = make_double2(0.0, 0.0);
            if (act && r < n) { x[k] = ai[r]; y[k] = aj[r]; }
            al += abs2(x[k]);
            be += abs2(y[k]);
            cfma(ga, conj(x[k]), y[k]);
          }
        } else if (act) {
          for (int r = lane; r < n; r += 16) {
            const double2 u = ai[r], w = aj[r];
            al += abs2(u);
            be += abs2(w);
            cfma(ga, conj(u), w);
          }
        }
        for (int o = 8; o > 0; o >>= 1) {  // every lane of the pair gets the same sums
          al += __shfl_xor_sync(0xffffffffu, al, o);
          be += __shfl_xor_sync(0xffffffffu, be, o);
          ga.x += __shfl_xor_sync(0xffffffffu, ga.x, o);
          ga.y += __shfl_xor_sync(0xffffffffu, ga.y, o);
        }
        const double g2 = abs2(ga);
        if (!act || !(g2 > 0.0) || g2 <= tol2 * (al * be) || min(al, be) <= zero2) continue;
        // tan 2 theta = g / d, d = (|a_j|^2 - |a_i|^2) / 2, theta the smaller
        // angle: c^2 = (1 + |d| / h) / 2, s = g / (2 h c), h^2 = d^2 + g^2
        const double d = 0.5 * (be - al);
        const double rh = rsqrt(d * d + g2);
        const double c2 = 0.5 + 0.5 * fabs(d) * rh, rc = rsqrt(c2), c = c2 * rc;
        const double f = (d >= 0.0 ? 0.5 : -0.5) * rh * rc;
        const double2 sph = f * ga, sphc = f * conj(ga);
        if (abs2(sph) < eps * eps * c2) continue;  // the rotation would not change a bit
        rotated = true;
        double2* vi = V + ld * i;
        double2* vj = V + ld * j;
        if constexpr (NR > 0) {
#pragma unroll
          for (int k = 0; k < NR; ++k) {
            const int r = lane + 16 * k;
            if (r < n) {
              const double2 u = vi[r], w = vj[r];
              ai[r] = c * x[k] - sphc * y[k];
              aj[r] = sph * x[k] + c * y[k];
              vi[r] = c * u - sphc * w;
              vj[r] = sph * u + c * w;
            }
          }
        } else {
          for (int r = lane; r < n; r += 16) {
            const double2 p = ai[r], q = aj[r], u = vi[r], w = vj[r];
            ai[r] = c * p - sphc * q;
            aj[r] = sph * p + c * q;
            vi[r] = c * u - sphc * w;
            vj[r] = sph * u + c * w;
          }
        }
      }
      __syncthreads();
    }
    if (rotated) *flag = 1;
    __syncthreads();
    if (*flag == 0) return sweep + 1;
  }
  return -1;
}

// After block_jacobi: s[k] sorted descending, perm[k] = source column.
__device__ __forceinline__ void block_sv_sort(const double2* A, int n, int ld, double* s_tmp, double* s, int* perm) {
  const int lane = threadIdx.x & 15, grp = threadIdx.x >> 4, ngrp = blockDim.x >> 4;
  for (int c0 = 0; c0 < n; c0 += ngrp) {
    const int c = c0 + grp;
    double acc = 0.0;
    if (c < n)
      for (int r = lane; r < n; r += 16) acc += abs2(A[ld * c + r]);
    for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (c < n && lane == 0) s_tmp[c] = sqrt(acc);
  }
  __syncthreads();
  // Non-finite values (from non-finite messages) sort last as -1, so that
  // the ranks stay a permutation and every perm[] entry is a valid column;
  // the caller reports them.
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const double si = s_tmp[i];
    const double ki = isfinite(si) ? si : -1.0;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double kj = isfinite(s_tmp[j]) ? s_tmp[j] : -1.0;
      rank += (kj > ki) || (kj == ki && j < i);
    }
    s[rank] = si;
    perm[rank] = i;
  }
  __syncthreads();
}

// The shared memory of one CTA: two matrices (D up to kTruncSmemMaxD), then
// values, sorted values, weights and ranks.
struct TruncSmem {
  double2 *A, *V;
  double *s_tmp, *s, *w;
  int* perm;
  int ld;
};
__device__ __forceinline__ TruncSmem trunc_smem(unsigned char* raw, int n, int max_d, double2* gA, double2* gV) {
  const int d = max_d < kTruncSmemMaxD ? max_d : kTruncSmemMaxD;
  TruncSmem m;
  double2* base = reinterpret_cast<double2*>(raw);
  m.ld = n <= kTruncSmemMaxD ? n | 1 : n;  // odd: rows of consecutive columns on distinct banks
  m.A = n <= kTruncSmemMaxD ? base : gA;
  m.V = n <= kTruncSmemMaxD ? base + (size_t)d * (d | 1) : gV;
  m.s_tmp = reinterpret_cast<double*>(base + (size_t)2 * d * (d | 1));
  m.s = m.s_tmp + max_d;
  m.w = m.s + max_d;
  m.perm = reinterpret_cast<int*>(m.w + max_d);
  return m;
}

__device__ __forceinline__ int jacobi_any(unsigned char* raw, const TruncSmem& m, int n, int max_d, int* flag,
                                          double* red) {
  if (n > kTruncSmemMaxD) return block_jacobi<0>(m.A, m.V, n, m.ld, flag, red);
  const int d = max_d < kTruncSmemMaxD ? max_d : kTruncSmemMaxD;
  double2* A = reinterpret_cast<double2*>(raw);  // m.A and m.V, known to be shared memory
  double2* V = A + d * (d | 1);
  if (n <= 16) return block_jacobi<1>(A, V, n, m.ld, flag, red);
  if (n <= 32) return block_jacobi<2>(A, V, n, m.ld, flag, red);
  if (n <= 64) return block_jacobi<4>(A, V, n, m.ld, flag, red);
  return block_jacobi<5>(A, V, n, m.ld, flag, red);
}

// SquareRootAndInverse of one message per CTA (blockIdx.x = 2 edge + side):
// R and the transpose of S, written to the edge's scratch.
template <typename R>
__global__ void __launch_bounds__(512) k_trunc_roots(const TruncTask* __restrict__ tasks, double sv_min, int max_d) {
  using C = typename cvec<R>::type;
  extern __shared__ __align__(16) unsigned char trunc_raw[];
  __shared__ double red[32];
  __shared__ int flag;
  const TruncTask tk = tasks[blockIdx.x >> 1];
  const int side = blockIdx.x & 1, n = tk.D, nn = n * n;
  double2* const big = tk.work + (size_t)(4 + 2 * side) * nn;  // matrices of the large-D path
  const TruncSmem m = trunc_smem(trunc_raw, n, max_d, big, big + nn);
  double2* Rout = tk.work + (size_t)(2 * side) * nn;
  double2* Sout = Rout + nn;
  const C* M = static_cast<const C*>(side ? tk.Mb : tk.Ma);
  double mx = 0.0;
  for (int i = threadIdx.x; i < nn; i += blockDim.x) {
    const double2 v = to_d2(M[i]);
    m.A[i % n + m.ld * (i / n)] = v;
    mx += fabs(v.x) + fabs(v.y);
  }
  // scale by a power of two to a norm near one, so that squares neither
  // overflow nor vanish whatever the message's scale; taken back in s
  mx = block_sum(mx, red);
  const int ex = mx > 0.0 && isfinite(mx) ? ilogb(mx) : 0;
  if (ex != 0)
    for (int i = threadIdx.x; i < nn; i += blockDim.x) {
      double2& v = m.A[i % n + m.ld * (i / n)];
      v = make_double2(scalbn(v.x, -ex), scalbn(v.y, -ex));
    }
  __syncthreads();
  const int done = jacobi_any(trunc_raw, m, n, max_d, &flag, red);
  block_sv_sort(m.A, n, m.ld, m.s_tmp, m.s, m.perm);
  // R[i,j] = sum_k U[i,k] sq_k conj(V[j,k]);  U[:,k] = A[:,perm k] / s_k
  // S[i,j] = sum_k V[i,k] isq_k conj(U[j,k])
  // with the scaled A and s' = s / 2^ex: sq / s' = sqrt(s) / s' and
  // 1 / (sq s') per k, zero where the reference drops the value
  const double sq_min = sqrt(sv_min);
  int bad = done < 0 ? 1 : 0;
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    const double sp = m.s[k], sk = scalbn(sp, ex), sq = sqrt(sk);
    const bool keep = sk > sv_min;  // sqrt(s) := 0 (root.h:316-318)
    m.s_tmp[k] = keep ? sq / sp : 0.0;
    m.w[k] = keep && sq > sq_min ? 1.0 / (sq * sp) : 0.0;  // root.h:324-326
    if (!isfinite(sk)) bad = 2;
  }
  if (threadIdx.x == 0) flag = 0;
  __syncthreads();
  if (bad) atomicMax(&flag, bad);
  for (int idx = threadIdx.x; idx < nn; idx += blockDim.x) {
    const int i = idx % n, j = idx / n;
    double2 r = make_double2(0.0, 0.0), q = make_double2(0.0, 0.0);
    for (int k = 0; k < n; ++k) {
      const double w1 = m.s_tmp[k];
      if (w1 == 0.0) continue;
      const int pk = m.perm[k] * m.ld;
      const double2 a_i = m.A[pk + i], v_j = m.V[pk + j];
      cfma(r, w1 * a_i, conj(v_j));
      cfma(q, m.w[k] * conj(a_i), v_j);  // S[j,i]
    }
    Rout[idx] = r;
    Sout[idx] = q;
  }
  __syncthreads();
  if (threadIdx.x == 0) tk.status[side] = flag;
}

// T of one edge per CTA, its SVD, the kept rank and both projectors.
template <typename R>
__global__ void __launch_bounds__(512) k_truncate_edges(const TruncTask* __restrict__ tasks, int chi_max, double sv_min,
                                                        int max_d) {
  using C = typename cvec<R>::type;
  extern __shared__ __align__(16) unsigned char trunc_raw[];
  __shared__ double red[32];
  __shared__ int flag;
  const TruncTask tk = tasks[blockIdx.x];
  const int n = tk.D, nn = n * n;
  const double2* RA = tk.work;
  const double2* SA = RA + nn;  // transposed
  const double2* RB = SA + nn;
  const double2* SB = RB + nn;
  double2* T = tk.work + (size_t)4 * nn;
  const TruncSmem m = trunc_smem(trunc_raw, n, max_d, tk.work + (size_t)5 * nn, tk.work + (size_t)6 * nn);
  // T = RA^T RB, normalized (truncation.h:110-121)
  for (int i = threadIdx.x; i < nn; i += blockDim.x) {
    m.A[i % n + m.ld * (i / n)] = RA[i];
    m.V[i % n + m.ld * (i / n)] = RB[i];
  }
  __syncthreads();
  double ss = 0.0;
  for (int idx = threadIdx.x; idx < nn; idx += blockDim.x) {
    const double2* ra = m.A + m.ld * (idx % n);
    const double2* rb = m.V + m.ld * (idx / n);
    double2 acc = make_double2(0.0, 0.0);
    for (int k = 0; k < n; ++k) cfma(acc, ra[k], rb[k]);
    T[idx] = acc;
    ss += abs2(acc);
  }
  const double tn = sqrt(block_sum(ss, red));
  const double inv_tn = tn > 0.0 ? 1.0 / tn : 1.0;
  __syncthreads();
  for (int i = threadIdx.x; i < nn; i += blockDim.x) m.A[i % n + m.ld * (i / n)] = inv_tn * T[i];
  __syncthreads();
  const int done = jacobi_any(trunc_raw, m, n, max_d, &flag, red);
  block_sv_sort(m.A, n, m.ld, m.s_tmp, m.s, m.perm);
  int keep = 0;
  while (keep < n && keep < chi_max && m.s[keep] > sv_min) ++keep;
  if (keep == 0) keep = 1;
  // P_a[i,c] = sum_k SA[k,i] X[k,c] sqrt(s_c);  X[:,c] = A[:,perm c]/s_c
  // P_b[j,c] = sqrt(s_c) sum_k Y[c,k] SB[k,j];  Y[c,k] = conj(V[k, perm c])
  C* Pa = static_cast<C*>(tk.Pa);
  C* Pb = static_cast<C*>(tk.Pb);
  for (int idx = threadIdx.x; idx < n * keep; idx += blockDim.x) {
    const int i = idx % n, c = idx / n;
    const double sc = m.s[c];
    const double2* x = m.A + m.ld * m.perm[c];
    const double2* y = m.V + m.ld * m.perm[c];
    const double xs = sc > 0.0 ? sqrt(sc) / sc : 0.0;
    double2 a = make_double2(0.0, 0.0), b = make_double2(0.0, 0.0);
    for (int k = 0; k < n; ++k) {
      cfma(a, SA[(size_t)n * k + i], x[k]);
      cfma(b, conj(y[k]), SB[(size_t)n * k + i]);
    }
    Pa[idx] = from_d2<C>(xs * a);
    Pb[idx] = from_d2<C>(sqrt(sc) * b);
  }
  for (int c = threadIdx.x; c < keep; c += blockDim.x) tk.s_keep[c] = m.s[c];
  if (threadIdx.x == 0) {
    double tot = 0.0, cut = 0.0;
    int bad = done < 0 ? 1 : 0;
    for (int k = 0; k < n; ++k) {
      const double s2 = m.s[k] * m.s[k];
      tot += s2;
      if (k >= keep) cut += s2;
      if (!isfinite(m.s[k])) bad = 2;  // non-finite message or T
    }
    *tk.keep_out = keep;
    *tk.err_out = tot > 0.0 ? cut / tot : 0.0;
    tk.status[2] = bad;
  }
}

// Messages after truncation: E = diag(s) (truncation.h:137-149).
struct DiagTask {
  const double* s;
  void* out;
  int n;
};
template <typename R>
__global__ void k_write_diag(const DiagTask* __restrict__ tasks) {
  using C = typename cvec<R>::type;
  const DiagTask tk = tasks[blockIdx.x];
  C* out = static_cast<C*>(tk.out);
  for (int i = threadIdx.x; i < tk.n * tk.n; i += blockDim.x) {
    const int r = i % tk.n, c = i / tk.n;
    out[i] = r == c ? from_d2<C>(make_double2(tk.s[r], 0.0)) : czero<C>();
  }
}

}  // namespace tnbp
