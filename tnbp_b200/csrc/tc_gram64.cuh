// Message Gram on tcgen05 for 32 < C <= 64 (chi = 32 requests), complex64:
//   N[c, c'] = sum_q A[q, c] * conj(B[q, c'])
// with the element and row conventions of k_gram_tc (tc_gram.cuh).
//
// Real form: X = [A_re ; A_im] and Y = [B_re ; B_im], 64 rows each, hi and lo
// (3xTF32 with the fourth product): per 8 contraction rows one M = 128, N =
// 256 MMA X_hi [Y_hi | Y_lo] and one N = 128 MMA X_lo Y_hi into the same first
// 128 columns.  D = columns 0-127 plus columns 128-255;
//   N_re = D[c, c'] + D[64+c, 64+c'],  N_im = D[64+c, c'] - D[c, 64+c'].
//
// What bounds it: the MMAs take 1536 cycles per 64 rows; reading A and B takes
// 2800 of HBM's share of an SM and splitting them about as long as the MMAs.
// The kernel before this one had one operand buffer and 256 threads and
// waited for each tile's MMAs before it converted the next; here 32-row tiles
// alternate between two operand buffers and 64-row sums between two
// accumulators, so loads (two tiles ahead, in registers), conversion, MMAs
// and the FP64 additions of finished sums overlap, and warps meet only through
// barriers of the operands.  A thread's four rows of a column come in one
// 32-byte load (in two of 16 each half of every sector: 3250 -> 2700 cycles
// per 32 rows at L > 1; 2600 at L = 1).  Per 5x5 sweep at D = 64: 14.3 -> 5.8
// ms (3.4 TB/s).
//
// One CTA (512 threads) per split-K chunk.  Every wait is bounded: on timeout
// the CTA records g_tc_error, waits once more (bounded) for its MMAs, frees
// its TMEM and returns.
#pragma once
#include <cstdint>

#include "tc_pair.cuh"

namespace tnbp {
namespace tc {
constexpr int kGram64Threads = 512;
constexpr int kGram64Q = 32;                    // contraction rows per tile
constexpr uint32_t kGram64X = 128 * kGram64Q * 4;  // X_hi or X_lo of a tile; Y (256 rows) is twice that
__host__ __device__ constexpr size_t gram64_smem_bytes() { return 1024 + 8 * (size_t)kGram64X + 64; }
__host__ __device__ inline bool gram64_ok(int C, int P) { return P == 1 && C > kTcMaxD && C <= 64; }
// 32 aligned bytes, a whole sector, in one load
__device__ __forceinline__ void ldg32(const float2* p, float4& a, float4& b) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
               : "l"(p));
}
}  // namespace tc

__global__ void __launch_bounds__(tc::kGram64Threads, 1) k_gram_tc64(const GramTask* __restrict__ tasks,
                                                                     const long long* __restrict__ begins, int ntask) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char g64_smem_raw[];
  unsigned char* op = g64_smem_raw + ((1024 - (smem_u32(g64_smem_raw) & 1023)) & 1023);  // per buffer: X_hi, X_lo, Y
  uint64_t* bars = reinterpret_cast<uint64_t*>(op + 8 * kGram64X);                        // per buffer: written, MMAs done
  const uint32_t bar_ready = smem_u32(bars), bar_done = bar_ready + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 4);
  volatile int* fail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const GramTask& tk = tasks[find_task(begins, ntask, blockIdx.x)];
  const int chunk = (int)(blockIdx.x - tk.block_begin), C = tk.C;
  const uint32_t qbeg = (uint32_t)(chunk * tk.chunk_rows), qend = (uint32_t)min(tk.Q, chunk * tk.chunk_rows + tk.chunk_rows);
  const uint32_t ntile = (qend - qbeg + kGram64Q - 1) / kGram64Q;
  const uint32_t L = (uint32_t)tk.L, LC = L * (uint32_t)C;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < 4; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bars + i)), "r"(i < 2 ? kGram64Threads / 32u : 1u));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *fail = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot, base = uniform(tmem);

  // This thread's part of a tile: four rows 4 q4 .. of column c, one 16-byte
  // operand chunk per re / im and hi / lo; eight lanes run along c (a
  // quarter warp's stores are 128 contiguous bytes), four along q.
  const uint32_t c = (uint32_t)((lane & 7) + 8 * (warp & 7)), q4 = (uint32_t)((lane >> 3) + 4 * (warp >> 3));
  const uint32_t place = q4 * (128 * 16) + (c >> 3) * 128 + (c & 7) * 16;   // X: 128 rows
  const uint32_t place_y = q4 * (256 * 16) + (c >> 3) * 128 + (c & 7) * 16;  // Y: 256 rows
  const bool mine = c < (uint32_t)C;
  // four rows of a column are 32 contiguous, aligned bytes
  const bool wide = (L & 3) == 0 && ((reinterpret_cast<uintptr_t>(tk.A) | reinterpret_cast<uintptr_t>(tk.B)) & 31) == 0;
  const float2* __restrict__ A = static_cast<const float2*>(tk.A) + (size_t)L * c;
  const float2* __restrict__ B = static_cast<const float2*>(tk.B) + (size_t)L * c;

  struct Part {
    float4 a01, a23, b01, b23;
  };
  Part part[2];  // of tiles t and t + 1
  // (l, m) of the next even and odd tile's first row, advanced by two tiles
  const uint32_t dm = 2 * kGram64Q / L, dl = 2 * kGram64Q - dm * L;
  uint32_t ms[2], ls[2];
#pragma unroll
  for (uint32_t i = 0; i < 2; ++i) {
    const uint32_t q = qbeg + i * kGram64Q + 4 * q4;
    ms[i] = q / L;
    ls[i] = q - ms[i] * L;
  }
  auto load = [&](uint32_t t, Part& p, uint32_t& mt, uint32_t& lt) {
    uint32_t q = qbeg + t * kGram64Q + 4 * q4, m = mt, l = lt;
    mt += dm;
    lt += dl;
    if (lt >= L) {
      lt -= L;
      ++mt;
    }
    p.a01 = p.a23 = p.b01 = p.b23 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!mine) return;
    if (wide && q + 3 < qend) {
      const size_t off = (size_t)l + (size_t)LC * m;
      ldg32(A + off, p.a01, p.a23);
      ldg32(B + off, p.b01, p.b23);
      return;
    }
    float2 a[4], b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] = b[j] = make_float2(0.f, 0.f);
      if (q < qend) {
        const size_t off = (size_t)l + (size_t)LC * m;
        a[j] = __ldg(A + off);
        b[j] = __ldg(B + off);
      }
      ++q;
      if (++l == L) { l = 0; ++m; }
    }
    p.a01 = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
    p.a23 = make_float4(a[2].x, a[2].y, a[3].x, a[3].y);
    p.b01 = make_float4(b[0].x, b[0].y, b[1].x, b[1].y);
    p.b23 = make_float4(b[2].x, b[2].y, b[3].x, b[3].y);
  };
  auto convert = [&](const Part& p, unsigned char* o) {
    float4 h, l;
    split4(make_float4(p.a01.x, p.a01.z, p.a23.x, p.a23.z), h, l);
    *reinterpret_cast<float4*>(o + place) = h;
    *reinterpret_cast<float4*>(o + kGram64X + place) = l;
    split4(make_float4(p.a01.y, p.a01.w, p.a23.y, p.a23.w), h, l);
    *reinterpret_cast<float4*>(o + place + 64 * 16) = h;
    *reinterpret_cast<float4*>(o + kGram64X + place + 64 * 16) = l;
    unsigned char* y = o + 2 * kGram64X + place_y;
    split4(make_float4(p.b01.x, p.b01.z, p.b23.x, p.b23.z), h, l);
    *reinterpret_cast<float4*>(y) = h;
    *reinterpret_cast<float4*>(y + 128 * 16) = l;
    split4(make_float4(p.b01.y, p.b01.w, p.b23.y, p.b23.w), h, l);
    *reinterpret_cast<float4*>(y + 64 * 16) = h;
    *reinterpret_cast<float4*>(y + 192 * 16) = l;
  };
  auto mma = [&](uint32_t t) {  // by warp 0
    const uint32_t o = uniform(smem_u32(op)) + (t & 1u) * 4 * kGram64X, d = base + ((t >> 1) & 1u) * 256;
    const uint64_t xh = smem_desc(o, 128 * 16, 128), xl = smem_desc(o + kGram64X, 128 * 16, 128),
                   y = smem_desc(o + 2 * kGram64X, 256 * 16, 128);
    if (elect_one()) {
#pragma unroll
      for (uint32_t s = 0; s < kGram64Q / 8; ++s) {
        mma_tf32(d, xh + 256 * s, y + 512 * s, idesc_tf32(128, 256), (t & 1u) | s);
        mma_tf32(d, xl + 256 * s, y + 512 * s, idesc_tf32(128, 128), 1u);
      }
      mma_commit(bar_done + 8u * (t & 1u));
    }
    __syncwarp();
  };
  // Bounded waits by a whole warp; false (for the whole warp) when it or any
  // other warp gave up.  Warps meet only through these barriers, so one may
  // be two tiles ahead of another.
  auto wait_bar = [&](uint32_t bar, uint32_t phase) -> bool {
    bool r = __all_sync(0xffffffffu, mbar_try(bar, phase));
    for (int i = 0; i < kPairWaitLimit && !r; ++i) {
      r = __all_sync(0xffffffffu, mbar_try(bar, phase));
      if (!r && (i & 1023) == 1023 && __any_sync(0xffffffffu, *fail)) break;
    }
    if (!r) *fail = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return r;
  };
  auto wait = [&](uint32_t t) { return wait_bar(bar_done + 8u * (t & 1u), (t >> 1) & 1u); };  // for tile t's MMAs
  // FP64 sums of this thread's row of D (lane of tensor memory), 32 columns
  const int row = 32 * (warp & 3) + lane, cg = warp >> 2;
  double acc[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) acc[i] = 0.0;
  auto drain = [&](uint32_t pair) {
    const uint32_t d = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (pair & 1u) * 256 + 32u * (uint32_t)cg;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      float v[8], u[8];
      tmem_ld4_async(d + 8 * h, v);
      tmem_ld4_async(d + 8 * h + 4, v + 4);
      tmem_ld4_async(d + 128 + 8 * h, u);
      tmem_ld4_async(d + 128 + 8 * h + 4, u + 4);
      tmem_ld_wait16(v, v + 4, u, u + 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[8 * h + i] += (double)(v[i] + u[i]);
    }
  };
  auto step = [&](uint32_t t, Part& p, uint32_t& m, uint32_t& l) -> bool {
    if (t >= 2 && !wait(t - 2)) return false;
    convert(p, op + (t & 1u) * 4 * kGram64X);
    if (t + 2 < ntile) load(t + 2, p, m, l);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_ready + 8u * (t & 1u));
    if (warp == 0) {
      if (!wait_bar(bar_ready + 8u * (t & 1u), (t >> 1) & 1u)) return false;
      mma(t);
    }
    // the sums of the two tiles before an even tile, while its MMAs run
    if (t >= 2 && (t & 1u) == 0) {
      if (!wait(t - 1)) return false;
      drain((t >> 1) - 1);
    }
    return true;
  };
  load(0, part[0], ms[0], ls[0]);
  if (ntile > 1) load(1, part[1], ms[1], ls[1]);
  bool ok = true;
  for (uint32_t t = 0; t < ntile && ok; t += 2) {
    ok = step(t, part[0], ms[0], ls[0]);
    if (ok && t + 1 < ntile) ok = step(t + 1, part[1], ms[1], ls[1]);
  }
  if (ok && wait(ntile - 1)) drain((ntile - 1) >> 1);
  __syncthreads();
  if (*fail == 0) {
    // D, then N, through shared memory (the operands are free), element (r, c) at 128 c + r
    double* dsum = reinterpret_cast<double*>(op);
#pragma unroll
    for (int i = 0; i < 32; ++i) dsum[128 * (32 * cg + i) + row] = acc[i];
    __syncthreads();
    double2* out = tk.partial + (long long)chunk * C * C;
    for (int o = tid; o < C * C; o += kGram64Threads) {
      const int a = o % C, b = o / C;
      out[o] = make_double2(dsum[128 * b + a] + dsum[128 * (64 + b) + 64 + a], dsum[128 * b + 64 + a] - dsum[128 * (64 + b) + a]);
    }
  } else if (tid == 0) {
    atomicExch(&g_tc_error, 1);
    for (uint32_t i = 0; i < 4; ++i) mbar_wait(bar_done + 8u * (i >> 1), i & 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

}  // namespace tnbp
