// Leg contraction on tcgen05 for bond dimensions above 32 (chi = 32 requests
// run BP at D = 64):  out[l, k, r] = sum_j in[l, j, r] * M[j, k],
// complex64 tensors, 32 < max(Din, Dout) <= 64, 3xTF32 as in k_leg_apply_tc.
//
// What bounds it: at D = 64 a 128-row tile moves 128 KB, about 5600 cycles of
// an SM's share of HBM, and its MMAs take 3100.  The kernel before this one
// converted straight from global loads into shared-memory operands with one
// tile in flight and waited for every chunk's MMAs (23000 cycles per tile).
// Here a tile arrives by cp.async while the one before it is worked on; its
// rows go to tensor memory as the A operand (shared memory then holds only
// M: [M_re | M_im], D1 = A_re M', D2 = A_im M'), K in two halves with an
// operand each, so that the next tile's first half is converted during this
// tile's second MMAs; the result returns over the tile it came from and is
// written out as memory runs.  Per 5x5 sweep at D = 64: 24.9 -> 10.2 ms (9000
// cycles per tile, 4 TB/s; 9400 at L = 1, whose tiles go out through shared
// memory).
//
// 512 threads, persistent, one CTA per SM (194 KB of shared memory, all of
// tensor memory).  Every wait is bounded: on timeout the CTA records
// g_tc_error, waits once more (bounded) for its MMAs, frees its TMEM and
// returns.
#pragma once
#include <cstdint>

#include "tc_pair.cuh"

namespace tnbp {
namespace tc {

constexpr int kTcMaxD64 = 64;
constexpr int kLeg64Threads = 512;
constexpr int kLeg64Pitch = kTcRows + 1;  // of a tile's columns: odd, see leg64_form
constexpr uint32_t kLeg64Op = 128 * 64 * 4;

__host__ __device__ constexpr size_t leg64_smem_bytes() {
  return 1024 + 2 * (size_t)kLeg64Op + 2 * (size_t)kTcMaxD64 * kLeg64Pitch * 8 + 64;
}
__host__ __device__ inline bool leg64_ok(int Din, int Dout) {
  return Din <= kTcMaxD64 && Dout <= kTcMaxD64 && (Din > kTcMaxD || Dout > kTcMaxD);
}
// Rows per tile: whole (l, j) blocks for L <= 32, so that the tile is one
// contiguous range of memory; above that 128, each run of l contiguous.
__host__ __device__ inline int leg64_rows(long long L) { return L <= 32 ? (int)(kTcRows / L * L) : kTcRows; }
__host__ __device__ inline long long leg64_tiles(long long L, long long R) {
  const long long rows = leg64_rows(L);
  return (L * R + rows - 1) / rows;
}

// How a tile lies in shared memory.  Rows that are contiguous in memory (L =
// 1, even dimensions) stay rows of 64, pairs swizzled by the row; where lanes
// run along memory (even L above 32) element (row, j) lies at 128 j + row.
// Both are copied 16 bytes at a time, and read without bank conflicts (D =
// 64, cycles per tile: 10900 -> 9400 at L = 1, 9300 -> 9100 above).  The
// rest, at 129 j + row, takes eight.
enum : uint32_t { kLeg64Any, kLeg64Row, kLeg64Col };
__device__ __forceinline__ uint32_t leg64_form(const LegTask& t) {
  if ((reinterpret_cast<uintptr_t>(t.in) | reinterpret_cast<uintptr_t>(t.out)) & 15) return kLeg64Any;
  if (t.L == 1) return ((t.Din | t.Dout) & 1) == 0 ? kLeg64Row : kLeg64Any;
  return t.L > 32 && (t.L & 1) == 0 ? kLeg64Col : kLeg64Any;
}

}  // namespace tc

template <typename MR>
__global__ void __launch_bounds__(tc::kLeg64Threads, 1) k_leg_apply_tc64(const LegTask* __restrict__ tasks,
                                                                        const long long* __restrict__ begins, int ntask,
                                                                        long long total_tiles) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char t64_smem_raw[];
  unsigned char* b_op = t64_smem_raw + ((1024 - (smem_u32(t64_smem_raw) & 1023)) & 1023);  // M: hi, lo
  float2* raw = reinterpret_cast<float2*>(b_op + 2 * kLeg64Op);                             // two tiles
  // per half: operand written, MMAs done; per tile parity: tile arrived
  uint64_t* bars = reinterpret_cast<uint64_t*>(raw + 2 * kTcMaxD64 * kLeg64Pitch);
  const uint32_t bar_ready = smem_u32(bars), bar_done = bar_ready + 16, bar_full = bar_ready + 32;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);
  volatile int* fail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const long long per = (total_tiles + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per, last = min(total_tiles, first + per);
  if (first >= last) return;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < 6; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bars + i)),
                   "r"(i < 2 ? kLeg64Threads / 32u : i < 4 ? 1u : (uint32_t)kLeg64Threads));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *fail = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot, base = uniform(tmem);
  constexpr uint32_t kColD = 256;  // A halves at 0 and 128 ([re_hi | im_hi | re_lo | im_lo] of 32 columns), D1 at 256, D2 at 384

  const int row = 32 * (warp & 3) + lane;
  const uint32_t g = (uint32_t)warp >> 2;  // groups of four columns, j: those with j % 4 == g
  const uint32_t lanes = tmem + ((uint32_t)(32 * (warp & 3)) << 16);

  // of the current task
  LegTask tk{};
  uint32_t L = 1, rows = 0, rpt = kTcRows, Din = 0, Dout = 0, Np = 8, nk = 1, nk0 = 1;  // K steps of 8, of the first half
  uint32_t form = kLeg64Any, pitch = kLeg64Pitch;
  const uint32_t swz = 2 * ((uint32_t)row & 7), at_row = 64 * (uint32_t)row;  // kLeg64Row

  auto load_tile = [&](uint32_t lt, int stage) {
    float2* d = raw + (size_t)stage * kTcMaxD64 * kLeg64Pitch;
    const float2* in = static_cast<const float2*>(tk.in);
    const uint32_t q0 = lt * rpt, n = min(rpt, rows - q0);
    if (form == kLeg64Row) {
      const float2* p = in + (size_t)q0 * Din;
      for (uint32_t i = 2 * (uint32_t)tid; i < n * Din; i += 2 * kLeg64Threads) {
        const uint32_t r = fast_div(i, tk.div_din), j = i - r * Din;
        cp16(d + 64 * r + (j ^ (2 * (r & 7))), p + i, true);
      }
    } else if (form == kLeg64Col) {
      const uint32_t i = 2 * ((uint32_t)tid & 63), j0 = (uint32_t)tid >> 6;
      if (i < n) {
        const uint32_t q = q0 + i, r = fast_div(q, tk.div_l), l = q - r * L;
        const float2* p = in + (size_t)l + (size_t)L * ((size_t)Din * r + j0);
        float2* e = d + j0 * kTcRows + i;
#pragma unroll 4
        for (uint32_t j = j0; j < Din; j += 8) {
          cp16(e, p, true);
          p += (size_t)L * 8;
          e += 8 * kTcRows;
        }
      }
    } else if (L <= 32) {
      const float2* p = in + (size_t)q0 * Din;
      for (uint32_t i = (uint32_t)tid; i < n * Din; i += kLeg64Threads) {
        const uint32_t c = fast_div(i, tk.div_l), l = i - c * L, r = fast_div(c, tk.div_din), j = c - r * Din;
        cp8(d + j * kLeg64Pitch + r * L + l, p + i, true);
      }
    } else if ((uint32_t)row < n) {
      const uint32_t q = q0 + (uint32_t)row, r = fast_div(q, tk.div_l), l = q - r * L;
      const float2* p = in + (size_t)l + (size_t)L * ((size_t)Din * r + g);
      float2* e = d + g * kLeg64Pitch + row;
#pragma unroll 4
      for (uint32_t j = g; j < Din; j += 4) {
        cp8(e, p, true);
        p += (size_t)L * 4;
        e += 4 * kLeg64Pitch;
      }
    }
    // this thread's arrival, when its copies have landed
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_full + 8u * stage) : "memory");
  };
  // columns j .. j + 3 of this row, zero from Din on
  auto read4 = [&](const float2* t, uint32_t j, float2* e) {
    if (form == kLeg64Row) {
      const uint32_t i = at_row + (j ^ swz);
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 a = j < Din ? *reinterpret_cast<const float4*>(t + i) : z;
      const float4 b = j + 2 < Din ? *reinterpret_cast<const float4*>(t + (i ^ 2)) : z;
      e[0] = make_float2(a.x, a.y);
      e[1] = make_float2(a.z, a.w);
      e[2] = make_float2(b.x, b.y);
      e[3] = make_float2(b.z, b.w);
      return;
    }
    const float2* p = t + j * pitch + row;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) e[k] = j + k < Din ? p[k * pitch] : make_float2(0.f, 0.f);
  };
  auto put_a = [&](const float2* t, uint32_t half) {
    const uint32_t j0 = half ? 2 * nk0 : 0, n = 2 * (half ? nk - nk0 : nk0);  // groups
    const uint32_t a = lanes + 128 * half;
#pragma unroll
    for (uint32_t i = g; i < 8; i += 4)
      if (i < n) {
        const uint32_t j = 4 * (j0 + i);
        float2 e[4];
        read4(t, j, e);
        float4 rh, rl, ih, il;
        split4(make_float4(e[0].x, e[1].x, e[2].x, e[3].x), rh, rl);
        split4(make_float4(e[0].y, e[1].y, e[2].y, e[3].y), ih, il);
        tmem_st4(a + 4 * i, rh);
        tmem_st4(a + 4 * i + 32u, ih);
        tmem_st4(a + 4 * i + 64u, rl);
        tmem_st4(a + 4 * i + 96u, il);
      }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  };
  auto mma_half = [&](uint32_t half) {  // by warp 0
    const uint32_t N2 = uniform(2 * Np), s0 = uniform(half ? nk0 : 0), n = uniform(half ? nk - nk0 : nk0);
    const uint32_t idesc = idesc_tf32(128, 0) | ((N2 >> 3) << 17), op = uniform(smem_u32(b_op));
    const uint64_t dh0 = smem_desc(op, N2 * 16, 128) + s0 * 2 * N2, dl0 = smem_desc(op + kLeg64Op, N2 * 16, 128) + s0 * 2 * N2;
    if (elect_one()) {
#pragma unroll
      for (uint32_t part = 0; part < 2; ++part)
#pragma unroll
        for (uint32_t s = 0; s < 4; ++s)
          if (s < n) {
            const uint32_t d = base + kColD + 128u * part, ah = base + 128u * half + 32u * part + 8u * s;
            const uint64_t dh = dh0 + s * 2 * N2, dl = dl0 + s * 2 * N2;
            mma_tf32_ts(d, ah, dh, idesc, half + s);
            mma_tf32_ts(d, ah, dl, idesc, 1u);
            mma_tf32_ts(d, ah + 64u, dh, idesc, 1u);
          }
      mma_commit(bar_done + 8u * half);
    }
    __syncwarp();
  };
  // Warps meet only through barriers.  A bounded wait by a whole warp; false
  // (for the whole warp) when it or any other warp gave up.
  auto wait = [&](uint32_t bar, uint32_t phase) -> bool {
    bool r = __all_sync(0xffffffffu, mbar_try(bar, phase));
    for (int i = 0; i < kPairWaitLimit && !r; ++i) {
      r = __all_sync(0xffffffffu, mbar_try(bar, phase));
      if (!r && (i & 1023) == 1023 && __any_sync(0xffffffffu, *fail)) break;
    }
    if (!r) *fail = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return r;
  };
  // this warp's part of a half's operand is written (and the last tile's D
  // read); warp 0 issues when every warp's is
  uint32_t ready_ph[2] = {0u, 0u}, done_ph[2] = {0u, 0u}, full_ph[2] = {0u, 0u};
  auto publish = [&](uint32_t half) -> bool {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_ready + 8u * half);
    if (warp != 0) return true;
    if (!wait(bar_ready + 8u * half, half ? ready_ph[1] : ready_ph[0])) return false;
    if (half) ready_ph[1] ^= 1u; else ready_ph[0] ^= 1u;
    mma_half(half);
    return true;
  };
  auto done = [&](uint32_t half) {
    const bool r = wait(bar_done + 8u * half, half ? done_ph[1] : done_ph[0]);
    if (half) done_ph[1] ^= 1u; else done_ph[0] ^= 1u;
    return r;
  };
  auto arrived = [&](int stage) {
    const bool r = wait(bar_full + 8u * stage, stage ? full_ph[1] : full_ph[0]);
    if (stage) full_ph[1] ^= 1u; else full_ph[0] ^= 1u;
    return r;
  };
  bool ok = true;

  int ti = find_task(begins, ntask, first) - 1;
  long long task_end = first;
  uint32_t lt = 0;
  bool loaded = false;   // this tile's copies are on their way
  bool halved = false;   // and its first half is in tensor memory
  for (long long tile = first; tile < last; ++tile, ++lt) {
    const int stage = (int)(tile - first) & 1;
    float2* t = raw + (size_t)stage * kTcMaxD64 * kLeg64Pitch;
    float2* t2 = raw + (size_t)(stage ^ 1) * kTcMaxD64 * kLeg64Pitch;
    if (tile == task_end) {  // the next task: this warp waited for the last one's MMAs
      tk = tasks[++ti];
      L = (uint32_t)tk.L;
      rows = (uint32_t)(tk.L * tk.R);
      rpt = (uint32_t)leg64_rows(tk.L);
      Din = (uint32_t)tk.Din;
      Dout = (uint32_t)tk.Dout;
      Np = (Dout + 7u) & ~7u;
      nk = (Din + 7u) / 8;
      nk0 = (nk + 1) / 2;
      form = uniform(leg64_form(tk));
      pitch = form == kLeg64Col ? kTcRows : kLeg64Pitch;
      task_end = begins[ti] + leg64_tiles(tk.L, tk.R);
      lt = (uint32_t)(tile - begins[ti]);
      loaded = halved = false;
      // element (n, k) of 2 Np rows (re, im), K = 8 nk columns
      const typename cvec<MR>::type* __restrict__ mat = static_cast<const typename cvec<MR>::type*>(tk.mat);
      for (uint32_t n = (uint32_t)warp; n < 2 * Np; n += kLeg64Threads / 32)
        for (uint32_t k = (uint32_t)lane; k < 8 * nk; k += 32) {
          const uint32_t c = n < Np ? n : n - Np;
          double v = 0.0;
          if (k < Din && c < Dout) {
            const double2 m = to_d2(mat[k + (size_t)Din * c]);
            v = n < Np ? m.x : m.y;
          }
          // the remainder in FP64, so that complex128 messages keep their low bits
          const float h = to_tf32((float)v), l = to_tf32((float)(v - (double)h));
          *reinterpret_cast<float*>(b_op + kmajor_off((int)n, (int)k, (int)(2 * Np))) = h;
          *reinterpret_cast<float*>(b_op + kLeg64Op + kmajor_off((int)n, (int)k, (int)(2 * Np))) = l;
        }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // A stage is free once the MMAs of its tile are done (every warp has read
    // it by then) or, where results go back over it, after the barrier below.
    if (!loaded) load_tile(lt, stage);
    const bool more = tile + 1 < task_end && tile + 1 < last;
    if (!halved) {
      if (!(ok = arrived(stage))) break;
      put_a(t, 0);
    }
    if (!(ok = publish(0))) break;
    if (more) load_tile(lt + 1, stage ^ 1);
    loaded = more;
    if (nk > nk0) {
      put_a(t, 1);
      if (!(ok = publish(1))) break;
    }
    if (!(ok = done(0))) break;
    // the next tile's first half, during this one's second MMAs
    halved = more;
    if (more) {
      if (!(ok = arrived(stage ^ 1))) break;
      put_a(t2, 0);
    }
    if (nk > nk0 && !(ok = done(1))) break;
    // D1, D2 of this row: back over the tile (both halves were read), or
    // straight out where lanes run along memory
    const uint32_t q0 = lt * rpt, n = min(rpt, rows - q0);
    const bool direct = L > 32;
    float2* out = static_cast<float2*>(tk.out);
    size_t off = 0;
    if (direct) {
      const uint32_t q = q0 + (uint32_t)row, r = fast_div(q, tk.div_l), l = q - r * L;
      off = (size_t)l + (size_t)L * (size_t)Dout * r;
    }
#pragma unroll
    for (uint32_t i = g; i < 16; i += 4)
      if (4 * i < Np) {
        float rr[4], ri[4], ir[4], ii[4];
        const uint32_t c = lanes + kColD + 4 * i;
        tmem_ld4_async(c, rr);             // A_re M_re
        tmem_ld4_async(c + Np, ri);        // A_re M_im
        tmem_ld4_async(c + 128, ir);       // A_im M_re
        tmem_ld4_async(c + 128 + Np, ii);  // A_im M_im
        tmem_ld_wait16(rr, ri, ir, ii);
        if ((uint32_t)row < n && form == kLeg64Row) {
          float2* p = t + at_row;
          *reinterpret_cast<float4*>(p + ((4 * i) ^ swz)) = make_float4(rr[0] - ii[0], ri[0] + ir[0], rr[1] - ii[1], ri[1] + ir[1]);
          *reinterpret_cast<float4*>(p + ((4 * i + 2) ^ swz)) = make_float4(rr[2] - ii[2], ri[2] + ir[2], rr[3] - ii[3], ri[3] + ir[3]);
        } else if ((uint32_t)row < n) {
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k) {
            const float2 v = make_float2(rr[k] - ii[k], ri[k] + ir[k]);
            if (!direct) t[(4 * i + k) * kLeg64Pitch + row] = v;
            else if (4 * i + k < Dout) out[off + (size_t)L * (4 * i + k)] = v;
          }
        }
      }
    if (!direct) {
      __syncthreads();
      float2* o = out + (size_t)q0 * Dout;
      if (form == kLeg64Row) {
        for (uint32_t i = 2 * (uint32_t)tid; i < n * Dout; i += 2 * kLeg64Threads) {
          const uint32_t r = Dout == Din ? fast_div(i, tk.div_din) : i / Dout, k = i - r * Dout;
          *reinterpret_cast<float4*>(o + i) = *reinterpret_cast<const float4*>(t + 64 * r + (k ^ (2 * (r & 7))));
        }
      } else
      for (uint32_t i = (uint32_t)tid; i < n * Dout; i += kLeg64Threads) {
        const uint32_t c = fast_div(i, tk.div_l), l = i - c * L;
        const uint32_t r = Dout == Din ? fast_div(c, tk.div_din) : c / Dout, k = c - r * Dout;
        o[i] = t[k * kLeg64Pitch + r * L + l];
      }
      __syncthreads();
    }
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  if (*fail && tid == 0) {
    // MMAs in flight get one more bounded wait before TMEM is freed
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
