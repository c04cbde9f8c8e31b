// Leg contraction and Gram in FP64 on the tensor pipe (mma.sync m8n8k4 .f64):
// the complex128 sweeps, the truncation's projector chains, the measurement
// chains and environments of every complex128-stored job, and the
// no-allocation message.
//
// What bounds them: one complex multiply-add is 8 flops and 16 bytes per
// operand element, so a leg at D = 32 needs 16 flops per byte moved, just
// above the ratio of the FP64 peak (36.8 TFLOP/s measured for both DFMA and
// DMMA) to the copy bandwidth: arithmetic and HBM both matter.  The previous
// CUDA-core kernels ran two shared-memory loads per complex FMA (10 TFLOP/s)
// and were bound by shared memory; a DMMA fragment is loaded once for 4
// (leg) or 2 (Gram) tiles, which leaves the FP64 pipe as the bound.  FP64
// products and sums as before (IEEE FMAs), only their order differs.
//
// Operand elements are complex (16 bytes, re and im together): one 16-byte
// shared load feeds the re and the im fragment.  A fragment load touches 8
// rows x 4 k; strides of 4 (mod 8) elements along the row, or 2 (mod 8)
// along k, put the 8 lanes of each quarter warp on distinct banks.
#pragma once
#include <cstdint>

#include "kernels.cuh"

namespace tnbp {
namespace dm {

constexpr int kLegThreads = 128;
constexpr int kLegRows = 64;     // 4 warps x 16 rows
constexpr int kLegCols = 32;     // output columns per pass
constexpr int kGramThreads = 128;
constexpr int kGramStage = 1152; // elements of one operand's stage

// Rows of one CTA's tile.  For L <= 32 a tile holds whole (l, j) blocks, so
// its input and output are contiguous ranges of memory whatever L is (odd
// and small L would otherwise touch a sector per element); above that a
// row's neighbours along l are themselves runs of 512 bytes.
__host__ __device__ inline int leg_rows_per_tile(long long L) {
  return L <= 32 ? (int)((kLegRows / (int)L) * (int)L) : kLegRows;
}
__host__ __device__ inline long long leg_tiles(long long L, long long R) {
  const long long rpt = leg_rows_per_tile(L);
  return (L * R + rpt - 1) / rpt;
}
// Row stride of an operand of Din columns: Din rounded up to the MMA's K of
// 4, then to 4 (mod 8).
__host__ __device__ inline int leg_ld(int Din) {
  const int k4 = (Din + 3) & ~3;
  return (k4 & 7) == 4 ? k4 : k4 + 4;
}
// The tile's elements in either order (rows of leg_ld, or columns of 66).
__host__ __device__ inline int leg_tile_elems(int Din) {
  const int k4 = (Din + 3) & ~3, a = kLegRows * leg_ld(Din), b = (kLegRows + 2) * k4;
  return a > b ? a : b;
}
// D = 32 takes 54 KB (four CTAs per SM), the largest Din of 128 198 KB.
__host__ __device__ inline size_t leg_smem_bytes(int max_din) {
  return (size_t)(leg_tile_elems(max_din) + kLegCols * leg_ld(max_din)) * sizeof(double2);
}
constexpr size_t gram_smem_bytes() { return (size_t)4 * kGramStage * sizeof(double2); }

__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
// 16 bytes global -> shared, zeros when !valid (nothing is read then).
__device__ __forceinline__ void cp16(double2* dst, const double2* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// find_task by a whole warp: 32 probes per step, so at most two dependent
// loads for up to 1024 tasks instead of ten.
__device__ __forceinline__ int find_task_warp(const long long* begins, int n, long long b) {
  const int lane = threadIdx.x & 31;
  int lo = 0;
  while (n > 1) {
    const int step = (n + 31) / 32, i = lane * step;
    const unsigned m = __ballot_sync(0xffffffffu, i < n && begins[lo + i] <= b);
    const int k = 31 - __clz((int)m);
    lo += k * step;
    n = min(step, n - k * step);
  }
  return lo;
}

}  // namespace dm

// out[l, k, r] = sum_j in[l, j, r] * mat[j, k] (the contraction of
// k_leg_apply), complex128.  One CTA: one tile of up to 64 rows with all of
// Din, output columns in passes of 32.  16 rows x 32 columns per warp: 6
// shared loads feed 32 DMMAs.
static __global__ void __launch_bounds__(dm::kLegThreads, 4)
    k_leg_apply_f64(const LegTask* __restrict__ tasks, const long long* __restrict__ begins, int ntask, int max_din) {
  using namespace dm;
  extern __shared__ __align__(16) unsigned char dm_smem[];
  const int ti = find_task_warp(begins, ntask, blockIdx.x);
  const LegTask tk = tasks[ti];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t L = (uint32_t)tk.L, rows = (uint32_t)(tk.L * tk.R);
  const int Din = tk.Din, Dout = tk.Dout, k4 = (Din + 3) & ~3, ld = leg_ld(Din);
  const uint32_t rpt = (uint32_t)leg_rows_per_tile(tk.L);
  const uint32_t q0 = (uint32_t)(blockIdx.x - tk.block_begin) * rpt;
  const int nrow = (int)min(rpt, rows - q0);
  double2* As = reinterpret_cast<double2*>(dm_smem);
  double2* Bs = As + leg_tile_elems(max_din);
  // element (row, j) at row sr + j sj: along j for L = 1, along l otherwise,
  // as the memory runs
  const int sr = L == 1 ? ld : 1, sj = L == 1 ? 1 : kLegRows + 2;
  const double2* __restrict__ in = static_cast<const double2*>(tk.in);
  const double2* __restrict__ mat = static_cast<const double2*>(tk.mat);

  if (L <= 32) {  // whole blocks: one contiguous range
    const double2* base = in + (size_t)q0 * Din;
    const uint32_t n = (uint32_t)(nrow * Din);
    for (uint32_t idx = tid; idx < n; idx += kLegThreads) {
      const uint32_t t = fast_div(idx, tk.div_l), l = idx - t * L;
      const uint32_t rr = fast_div(t, tk.div_din), j = t - rr * (uint32_t)Din;
      cp16(As + (int)(rr * L + l) * sr + (int)j * sj, base + idx, true);
    }
  } else {
    const int row = tid & (kLegRows - 1);
    if (row < nrow) {
      const uint32_t q = q0 + (uint32_t)row, r = fast_div(q, tk.div_l), l = q - r * L;
      const double2* p = in + (size_t)l + (size_t)L * (size_t)Din * r;
      for (int j = tid / kLegRows; j < Din; j += kLegThreads / kLegRows) cp16(As + row + j * sj, p + (size_t)L * j, true);
    }
  }
  if (k4 > Din)  // the K padding multiplies to zero
    for (int i = tid; i < kLegRows * (k4 - Din); i += kLegThreads)
      As[(i & (kLegRows - 1)) * sr + (Din + i / kLegRows) * sj] = make_double2(0.0, 0.0);

  const int r0 = warp * 16 + (lane >> 2), kl = lane & 3;
  for (int c0 = 0; c0 < Dout; c0 += kLegCols) {
    const int kc = min(kLegCols, Dout - c0);
    if (c0) __syncthreads();  // the last pass has read Bs
    for (int i = tid; i < kc * Din; i += kLegThreads) {
      const int c = (int)fast_div((uint32_t)i, tk.div_din), j = i - c * Din;
      cp16(Bs + c * ld + j, mat + (size_t)c0 * Din + i, true);
    }
    if (k4 > Din)
      for (int i = tid; i < kLegCols * (k4 - Din); i += kLegThreads)
        Bs[(i & (kLegCols - 1)) * ld + Din + i / kLegCols] = make_double2(0.0, 0.0);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    const int nf = (kc + 7) >> 3;
    if (warp * 16 >= nrow) continue;  // every warp reaches the barriers above
    double cr[2][4][2], ci[2][4][2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int f = 0; f < 4; ++f) cr[m][f][0] = cr[m][f][1] = ci[m][f][0] = ci[m][f][1] = 0.0;
    const double2* ap = As + r0 * sr + kl * sj;
    const double2* bp = Bs + (lane >> 2) * ld + kl;
    for (int k = 0; k < k4; k += 4) {
      const double2 a0 = ap[0], a1 = ap[8 * sr];
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        if (f < nf) {
          const double2 b = bp[f * 8 * ld];
          mma_f64(cr[0][f][0], cr[0][f][1], a0.x, b.x);
          mma_f64(ci[0][f][0], ci[0][f][1], a0.x, b.y);
          mma_f64(cr[1][f][0], cr[1][f][1], a1.x, b.x);
          mma_f64(ci[1][f][0], ci[1][f][1], a1.x, b.y);
          mma_f64(cr[0][f][0], cr[0][f][1], -a0.y, b.y);
          mma_f64(ci[0][f][0], ci[0][f][1], a0.y, b.x);
          mma_f64(cr[1][f][0], cr[1][f][1], -a1.y, b.y);
          mma_f64(ci[1][f][0], ci[1][f][1], a1.y, b.x);
        }
      }
      ap += 4 * sj;
      bp += 4;
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int row = r0 + 8 * m;
      if (row >= nrow) continue;
      const uint32_t q = q0 + (uint32_t)row, r = fast_div(q, tk.div_l), l = q - r * L;
      double2* o = static_cast<double2*>(tk.out) + (size_t)l + (size_t)L * ((size_t)Dout * r + c0);
#pragma unroll
      for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = 8 * f + 2 * kl + e;
          if (c < kc) o[(size_t)L * c] = make_double2(cr[m][f][e], ci[m][f][e]);
        }
    }
  }
}

// N[c, c'] = sum_q A[q, c] conj(B[q, c']), the contraction of k_gram, in
// complex128: one CTA per (row chunk, 32 x 32 tile of N), the chunk walked
// in stages of 32, 64 or 128 rows (fewer columns, more rows: a stage stays
// near 16 KB per operand) loaded one stage ahead with cp.async.  Above 16
// columns each warp owns a 16 x 16 quarter of N; up to 16 columns the warps
// share the rows and their sums are added in warp order at the end.
static __global__ void __launch_bounds__(dm::kGramThreads, 3)
    k_gram_f64(const GramTask* __restrict__ tasks, const long long* __restrict__ begins, int ntask) {
  using namespace dm;
  extern __shared__ __align__(16) unsigned char dm_smem[];
  double2* st = reinterpret_cast<double2*>(dm_smem);  // [stage][operand][kGramStage]
  const GramTask tk = tasks[find_task_warp(begins, ntask, blockIdx.x)];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long b = blockIdx.x - tk.block_begin;
  const int tiles2 = tk.ctiles * tk.ctiles, chunk = (int)(b / tiles2), tt = (int)(b % tiles2);
  const int ca0 = (tt % tk.ctiles) * kColTile, cb0 = (tt / tk.ctiles) * kColTile;
  const int na = min(kColTile, tk.C - ca0), nb = min(kColTile, tk.C - cb0), nc = max(na, nb);
  const uint32_t qbeg = (uint32_t)(chunk * tk.chunk_rows), qend = (uint32_t)min(tk.Q, chunk * tk.chunk_rows + tk.chunk_rows);
  const uint32_t L = (uint32_t)tk.L;
  const size_t LD = (size_t)tk.L * tk.D, LDM = (size_t)tk.L * tk.D * tk.M;
  const double2* __restrict__ A = static_cast<const double2*>(tk.A);
  const double2* __restrict__ B = static_cast<const double2*>(tk.B);
  const bool split = nc <= 16;  // warps split the rows
  const int TQ = nc > 16 ? 32 : nc > 8 ? 64 : 128;
  // element (q, c) at c sc + q sq: along q when the memory runs along l,
  // along c for L = 1
  const int sq = L == 1 ? (nc > 16 ? 34 : nc > 8 ? 18 : 9) : 1, sc = L == 1 ? 1 : TQ + 4;

  const bool one = tk.P == 1;
  auto col = [&](int x) { return one ? (size_t)L * x : (size_t)L * (x % tk.D) + LDM * (x / tk.D); };
  auto load = [&](uint32_t q0, double2* dst) {
    if (L == 1) {  // every thread walks the (q, c) plane of the stage, c fastest
      int c = tid % nc, q = tid / nc;
      const int dc = kGramThreads % nc, dq = kGramThreads / nc;
      for (; q < TQ; q += dq) {
        const bool ok = q0 + (uint32_t)q < qend;
        const size_t row = ok ? LD * (q0 + (uint32_t)q) : 0;
        if (c < na) cp16(dst + c * sc + q * sq, A + row + col(ca0 + c), ok);
        if (c < nb) cp16(dst + kGramStage + c * sc + q * sq, B + row + col(cb0 + c), ok);
        c += dc;
        if (c >= nc) { c -= nc; ++q; }
      }
    } else {
      const int qi = tid & (TQ - 1);
      const uint32_t q = q0 + (uint32_t)qi;
      const bool ok = q < qend;
      const uint32_t m = ok ? q / L : 0, l = ok ? q - m * L : 0;
      const size_t row = (size_t)l + LD * m;
      for (int c = tid / TQ; c < nc; c += kGramThreads / TQ) {
        if (c < na) cp16(dst + c * sc + qi, A + row + col(ca0 + c), ok);
        if (c < nb) cp16(dst + kGramStage + c * sc + qi, B + row + col(cb0 + c), ok);
      }
    }
    cp_commit();
  };

  const int wa = split ? 0 : (warp & 1) * 16, wb = split ? 0 : (warp >> 1) * 16;
  const int fa = min(2, (na - wa + 7) >> 3), fb = min(2, (nb - wb + 7) >> 3);  // may be <= 0: nothing to do
  double nr[2][2][2], ni[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) nr[i][j][0] = nr[i][j][1] = ni[i][j][0] = ni[i][j][1] = 0.0;
  const int k_step = split ? 16 : 4, k_first = (split ? 4 * warp : 0) + (lane & 3);
  load(qbeg, st);
  int s = 0;
  for (uint32_t q0 = qbeg; q0 < qend; q0 += (uint32_t)TQ, s ^= 1) {
    if (q0 + (uint32_t)TQ < qend) {
      load(q0 + (uint32_t)TQ, st + (s ^ 1) * 2 * kGramStage);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    const double2* as = st + s * 2 * kGramStage + (wa + (lane >> 2)) * sc;
    const double2* bs = st + s * 2 * kGramStage + kGramStage + (wb + (lane >> 2)) * sc;
#pragma unroll 4
    for (int k = k_first; k < TQ; k += k_step) {
      double2 a[2], bb[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i] = i < fa ? as[8 * i * sc + k * sq] : make_double2(0.0, 0.0);
        bb[i] = i < fb ? bs[8 * i * sc + k * sq] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (i < fa && j < fb) {
            mma_f64(nr[i][j][0], nr[i][j][1], a[i].x, bb[j].x);
            mma_f64(ni[i][j][0], ni[i][j][1], a[i].y, bb[j].x);
            mma_f64(nr[i][j][0], nr[i][j][1], a[i].y, bb[j].y);
            mma_f64(ni[i][j][0], ni[i][j][1], -a[i].x, bb[j].y);
          }
    }
    __syncthreads();  // the stage is free for the load after next
  }
  double2* part = tk.partial + (long long)chunk * tk.C * tk.C;
  if (!split) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int a = wa + 8 * i + (lane >> 2), c = wb + 8 * j + 2 * (lane & 3) + e;
          if (a < na && c < nb) part[ca0 + a + (long long)tk.C * (cb0 + c)] = make_double2(nr[i][j][e], ni[i][j][e]);
        }
    return;
  }
  // 4 warps x 16 x 16 sums in the stages, added in warp order
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        st[warp * 256 + 8 * i + (lane >> 2) + 16 * (8 * j + 2 * (lane & 3) + e)] = make_double2(nr[i][j][e], ni[i][j][e]);
  __syncthreads();
  for (int o = tid; o < 256; o += kGramThreads) {
    const int a = o & 15, c = o >> 4;
    if (a < na && c < nb)
      part[ca0 + a + (long long)tk.C * (cb0 + c)] = ((st[o] + st[256 + o]) + st[512 + o]) + st[768 + o];
  }
}

}  // namespace tnbp
