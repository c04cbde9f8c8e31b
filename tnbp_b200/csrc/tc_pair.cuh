// Both messages of a pair of legs on tcgen05 (sm_100a), for the complex64 and
// mixed sweeps.  A site's legs are taken as a plane (x, y) and an outer index
// o (every other leg and the physical one); with W the site tensor after the
// two other bond legs' messages were absorbed and V the site tensor,
//   N_x[x, x'] = sum_{o, y}  (sum_y2 W[x, y2, o] E_y[y2, y]) conj(V[x', y, o])
//   N_y[y, y'] = sum_{o, x}  (sum_x2 W[x2, y, o] E_x[x2, x]) conj(V[x, y', o])
// -- the last absorption of bp.h:137-152 for both targets and their Grams
// (bp.h:157-166) -- in one pass over W and V: the absorbed tensors stay on
// chip.  Degree-4 sites with every dim <= 32 (the others keep the separate
// leg and Gram kernels).
//
// Why: level by level, these two absorptions and Grams read and write a site
// tensor 12 times per pair; here 2 reads remain, and the bound moves from
// HBM and launch tails to what lies between the hand-overs of a tile: shared
// memory (operand stores and MMA reads, about 6000 cycles per tile at D =
// 32), conversions, FP64 additions and waits.  So two groups of warps, one
// per target, share the tiles but nothing else and fill each other's gaps (5 %
// of the tile's cycles at D = 32, 16 % at 16, against one group that takes the
// targets in turn).  One sweep of an 8x8 lattice's loop at D = 32 (36 degree-4
// sites): 3.96 ms in the separate kernels, 1.85 ms here; 6x6 at D = 16: 0.17
// -> 0.11 ms, at D = 24 0.46 ms.
//
// A tile is P planes (P Dx, P Dy <= 128 rows): raw complex64 planes arrive by
// cp.async, two tiles in flight, placed as PairLayout says.  Per target (say
// x; for y the roles swap):
//   1. rows (o, x) of W, split hi/lo (3xTF32), go to tensor memory as the A
//      operand; D1 = A_re [E_re | E_im], D2 = A_im [E_re | E_im] (hi.hi +
//      hi.lo + lo.hi, A from TMEM, 24 MMAs of N = 64 at D = 32), so only the
//      two 64-column halves of E are kept in shared memory;
//      P_re = D1_re - D2_im, P_im = D1_im + D2_re
//   2. P and the matching rows of V become the Gram's operands, eight columns
//      y at a time: rows [re_hi; im_hi; re_lo; im_lo] x 32 of 8 P contraction
//      columns (o, y); one M = 128, N = 128 MMA per 8 columns gives all four
//      hi/lo products
//   3. after 64 columns the FP32 Gram is added to FP64 registers, the cross
//      products apart from the main ones.
// Step 3 costs a fifth of the kernel (1.50 ms at D = 32, 0.089 at 16, 0.34 at
// 24 with one FP32 sum per tile, cross products added to it in FP32), but so
// these sums are no coarser than k_gram_tc's: the tensor core truncates as it
// accumulates, so that the error grows with the run and is of one sign.
// Messages of a degree-4 site against 64 bits, root mean square over 12 seeds
// with decaying bonds, leg by leg / one sum per tile / like this, in 1e-8:
// 18.1 / 13.2 / 11.5 at D = 32, 12.6 / 14.7 / 11.0 at 16, 10.1 / 11.0 / 9.9 at
// 12; the mixed 16x16 chi 16 solve takes 62 sweeps instead of 67 and its |dE|
// is 7e-8 instead of 8.9e-7.
// A chunk of tiles ends in one FP64 partial per target, reduced by
// k_msg_finalize in a fixed order.
//
// Every wait is bounded: on timeout the CTA records g_tc_error, waits once
// more (bounded) for its MMAs, frees its TMEM and returns without writing
// its partials.
#pragma once
#include <cstdint>
#include <type_traits>

#include "tc_gram.cuh"

namespace tnbp {

namespace tc {
constexpr int kPairWarps = 16;                               // converting warps
constexpr int kPairGroup = kPairWarps / 2;                   // those of one target
constexpr int kPairLoaders = 2;                              // loading warps, beside two that issue the MMAs
constexpr int kPairThreads = 32 * (kPairWarps + 2 + kPairLoaders);
// Registers per thread after the split: 512 x 112 + 128 x 32 = 640 x 96, what
// the launch gives the CTA (64 of the 112 are the FP64 sums).
constexpr int kPairRegsWork = 112, kPairRegsFeed = 32;
static_assert(kPairWarps * kPairRegsWork + (2 + kPairLoaders) * kPairRegsFeed <= 96 * (kPairWarps + 2 + kPairLoaders),
              "register split");
constexpr int kPairRawElems = 32 * 128;                      // one tensor's planes of a tile
constexpr int kPairWaitLimit = 1 << 22;
constexpr uint32_t kPairE = 64 * 32 * 4;                     // one of E's operands (N = 64, K = 32)
// One Gram operand of a stage: 128 rows, 2 P groups of four columns, these 32
// or 16 bytes further apart than they are large, so that the planes of one
// row of PairLayout's second form land in distinct banks.
__host__ __device__ constexpr uint32_t pair_group(uint32_t P) { return 128 * 16 + (P == 4 ? 32 : 16); }
__host__ __device__ constexpr uint32_t pair_op(uint32_t P) { return 2 * P * pair_group(P); }
// One tensor's planes of a tile: 32 x 32 x 4 or 16 x 16 x 8
__host__ __device__ constexpr uint32_t pair_raw(uint32_t P) { return P == 4 ? 32 * 128 : 16 * 128; }
__host__ __device__ constexpr size_t pair_ring(uint32_t P) { return 4 * ((size_t)pair_op(P) + pair_raw(P) * 8); }
__host__ __device__ constexpr size_t pair_smem_bytes() {
  return 128 + 4 * (size_t)kPairE + (pair_ring(4) > pair_ring(8) ? pair_ring(4) : pair_ring(8)) + 128;
}
// Planes per tile: 4 (8 up to dimension 16): the padded rows of
// either target stay within 128.
__host__ __device__ inline int pair_planes(int Dx, int Dy) { return (Dx > Dy ? Dx : Dy) <= 16 ? 8 : 4; }
// Where a tile's element (o, x, y) lies: y PE + (e ^ swz(y)), PE = P Xp, with
// e running as memory does: e = o Xp + x when planes are contiguous (L1 = 1),
// e = x P + o when consecutive o are.  So 16-byte copies, two elements each,
// fit both forms when Dx (L1) is even and the tensors are 16-byte aligned;
// with one form for both, memory that runs along o took 8-byte copies in
// 32-byte pieces (D = 32: 15100 -> 12500 cycles per tile in pair_gram, 10700 -> 8000
// in k_pair_absorb_tc).  A tile's rows are numbered as e, (o, x),
// or likewise with y for x, (o, y).  The swizzle makes reads of both kinds
// free of bank conflicts: rows (o, x) read eight bytes at one y, consecutive
// lanes consecutive e; rows (o, y) read a pair (x, x + 1) in the first form,
// whose eight lanes differ in y, and eight bytes in the second, whose sixteen
// lanes are P planes of 16 / P different y.
template <uint32_t P>
struct PairLayout {
  uint32_t along_x, Xp, Yp, PE;  // along_x: the first form
  __device__ __forceinline__ void set(bool first_form, uint32_t Dx, uint32_t Dy) {
    along_x = first_form;
    Xp = (Dx + 7u) & ~7u;
    Yp = (Dy + 7u) & ~7u;
    PE = P * Xp;
  }
  __device__ __forceinline__ uint32_t swz(uint32_t y) const { return along_x ? 2u * (y & 7u) : P * (y & (16u / P - 1u)); }
  // (o, i) of row r, i = x or y padded to N
  __device__ __forceinline__ void row(uint32_t r, uint32_t N, uint32_t& o, uint32_t& i) const {
    o = along_x ? r / N : r % P;
    i = along_x ? r - o * N : r / P;
  }
};
// A thread's row of a tile, and reads and writes of its groups of four
// columns j (j % 2 the same for every one of a thread).
template <uint32_t P>
struct PairRow {
  uint32_t ex, ey, base_y, swz_y, PE;  // ex: swizzled for y = 4 j
  uint32_t along_x, step_k, mask_k;
  __device__ __forceinline__ void set(const PairLayout<P>& l, uint32_t row, uint32_t odd) {
    const uint32_t rx = row < P * l.Xp ? row : 0, ry = row < P * l.Yp ? row : 0;
    uint32_t o, y;
    l.row(ry, l.Yp, o, y);
    along_x = l.along_x;
    PE = l.PE;
    ex = rx ^ l.swz(4 * odd);
    step_k = along_x ? 2 : P;
    mask_k = along_x ? 3 : 16 / P - 1;
    base_y = y * PE;
    ey = along_x ? o * l.Xp : o;
    swz_y = l.swz(y);
  }
  // (o, x) at y = 4 j + k
  __device__ __forceinline__ uint32_t at_x(uint32_t j, uint32_t k) const {
    return (ex ^ (step_k * (k & mask_k))) + (4 * j + k) * PE;
  }
  // (o, y) at x = 4 j; the three after it are this ^ 1, 2, 3 (^ P, 2 P, 3 P in the second form)
  template <bool Form>
  __device__ __forceinline__ uint32_t at_y(uint32_t j) const {
    return base_y + ((ey + (Form ? 4 : 4 * P) * j) ^ swz_y);
  }
  // Form: along_x, known to the caller so that a loop's reads need not wait
  // for each other's branches
  template <bool Form>
  __device__ __forceinline__ void read(const float2* t, bool target_y, uint32_t j, float4& re, float4& im) const {
    float2 a, b, c, d;
    if (!target_y) {
      a = t[at_x(j, 0)];
      b = t[at_x(j, 1)];
      c = t[at_x(j, 2)];
      d = t[at_x(j, 3)];
    } else if constexpr (Form) {
      const uint32_t i = at_y<Form>(j);
      const float4 u = *reinterpret_cast<const float4*>(t + i), v = *reinterpret_cast<const float4*>(t + (i ^ 2));
      re = make_float4(u.x, u.z, v.x, v.z);
      im = make_float4(u.y, u.w, v.y, v.w);
      return;
    } else {
      const uint32_t i = at_y<Form>(j);
      a = t[i];
      b = t[i ^ P];
      c = t[i ^ (2 * P)];
      d = t[i ^ (3 * P)];
    }
    re = make_float4(a.x, b.x, c.x, d.x);
    im = make_float4(a.y, b.y, c.y, d.y);
  }
  template <bool Form>
  __device__ __forceinline__ void write(float2* t, bool target_y, uint32_t j, float4 re, float4 im) const {
    const uint32_t i = at_y<Form>(j);
    if (target_y && Form) {
      *reinterpret_cast<float4*>(t + i) = make_float4(re.x, im.x, re.y, im.y);
      *reinterpret_cast<float4*>(t + (i ^ 2)) = make_float4(re.z, im.z, re.w, im.w);
      return;
    }
    t[target_y ? i : at_x(j, 0)] = make_float2(re.x, im.x);
    t[target_y ? i ^ P : at_x(j, 1)] = make_float2(re.y, im.y);
    t[target_y ? i ^ (2 * P) : at_x(j, 2)] = make_float2(re.z, im.z);
    t[target_y ? i ^ (3 * P) : at_x(j, 3)] = make_float2(re.w, im.w);
  }
};

// The sites that take it: degree 4, every bond dimension at most 32.
__host__ __device__ inline bool pair_ok(const int* D, int g) {
  return g == 4 && D[0] <= 32 && D[1] <= 32 && D[2] <= 32 && D[3] <= 32;
}

__device__ __forceinline__ void mma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
  const uint32_t z = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(z), "r"(z), "r"(z), "r"(z));
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, float4 v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(__float_as_uint(v.x)),
               "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w))
               : "memory");
}
// Four columns of this warp's lanes; the caller waits (tmem_ld_wait) before
// it uses them.
__device__ __forceinline__ void tmem_ld4_async(uint32_t addr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(addr));
}
// Waits for the loads; the values pass through it, so that no use of them can
// be moved before it.
__device__ __forceinline__ void tmem_ld_wait16(float* a, float* b, float* c, float* d) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(a[3]), "+f"(b[0]), "+f"(b[1]), "+f"(b[2]), "+f"(b[3]),
                 "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]), "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               :
               : "memory");
}

// x = hi + lo with hi = x rounded to 11 significant bits (half away, as
// cvt.rna.tf32 does) and lo = x - hi exact, of which the tensor core reads the
// upper 11 bits: lo has at most 12 below its sign, so that is off by at most
// one unit of x's last place, as far as rounding lo would be.  Three
// instructions per value; the conversion instruction expands to four and
// both roundings by it bound the kernel.  A NaN reaches the product in lo.
__device__ __forceinline__ void split1(float x, float& h, float& l) {
  h = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
  l = x - h;
}
__device__ __forceinline__ void split4(float4 v, float4& h, float4& l) {
  split1(v.x, h.x, l.x);
  split1(v.y, h.y, l.y);
  split1(v.z, h.z, l.z);
  split1(v.w, h.w, l.w);
}
__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t phase) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(addr), "r"(phase)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t addr) {
  asm volatile("{\n\t.reg .b64 s;\n\tmbarrier.arrive.shared::cta.b64 s, [%0];\n\t}\n" ::"r"(addr) : "memory");
}
// The chunks of one CTA: those whose first tile lies in [lo, hi) of all tasks'
// tiles (begins: exclusive prefix of tiles), so CTAs get equal shares of
// uneven tasks while a task's chunks depend on the task alone.
struct PairChunks {
  const LegPairTask* tasks;
  const long long* begins;
  int ntask, ti, chunk;
  long long hi;
  __device__ PairChunks(const LegPairTask* t, const long long* b, int n, long long lo, long long h)
      : tasks(t), begins(b), ntask(n), ti(find_task(b, n, lo)), chunk(0), hi(h) {
    chunk = (int)((lo - begins[ti] + tasks[ti].chunk_tiles - 1) / tasks[ti].chunk_tiles);
  }
  __device__ bool valid() {
    while (ti < ntask && chunk >= tasks[ti].nchunk) {
      ++ti;
      chunk = 0;
    }
    return ti < ntask && begins[ti] + (long long)chunk * tasks[ti].chunk_tiles < hi;
  }
};
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cp16(float2* dst, const float2* src, bool valid) {
  const uint32_t d = smem_u32(dst);
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp8(float2* dst, const float2* src, bool valid) {
  const uint32_t d = smem_u32(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
}  // namespace tc

// Whether two neighbouring elements e of a tile are always 16 aligned bytes
// of both tensors, and both or neither within them.
__device__ __forceinline__ bool pair_wide(const LegPairTask& tk) {
  const int run = tk.L1 == 1 ? tk.Dx : (int)tk.L1;
  return (run & 1) == 0 && ((reinterpret_cast<uintptr_t>(tk.W) | reinterpret_cast<uintptr_t>(tk.V)) & 15) == 0;
}

// The messages' operands, E_y then E_x, hi then lo each: element (n, k) of
// N = 2 Np rows (re, im), K = Np columns; legs leg0 .. leg1 - 1, by `nwarp` warps.
template <typename MR>
__device__ __forceinline__ void build_pair_e(const LegPairTask& tk, unsigned char* e_op, uint32_t Xp, uint32_t Yp, int leg0, int leg1,
                                             int warp, int lane, int nwarp) {
  using namespace tc;
  for (int leg = leg0; leg < leg1; ++leg) {
    const int D = leg == 0 ? tk.Dy : tk.Dx, Np = leg == 0 ? (int)Yp : (int)Xp, N2 = 2 * Np;
    const typename cvec<MR>::type* E = static_cast<const typename cvec<MR>::type*>(leg == 0 ? tk.Ey : tk.Ex);
    unsigned char* hi_op = e_op + (size_t)leg * 2 * kPairE;
    if (lane < Np) {
      for (int n = warp; n < N2; n += nwarp) {
        const int c = n < Np ? n : n - Np;
        double v = 0.0;
        if (lane < D && c < D) {
          const double2 m = to_d2(E[lane + (long long)D * c]);
          v = n < Np ? m.x : m.y;
        }
        // the remainder in FP64, so that complex128 messages keep their low bits
        const float h = to_tf32((float)v), l = to_tf32((float)(v - (double)h));
        *reinterpret_cast<float*>(hi_op + kmajor_off(n, lane, N2)) = h;
        *reinterpret_cast<float*>(hi_op + kPairE + kmajor_off(n, lane, N2)) = l;
      }
    }
    __syncwarp();
  }
}

// CTA `block` of `nblock`, all tasks of P planes per tile.
template <typename MR, uint32_t P>
__device__ __forceinline__ void pair_gram(const LegPairTask* __restrict__ tasks, const long long* __restrict__ begins, int ntask,
                                          long long ntile_all, uint32_t block, uint32_t nblock) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char pr_smem_raw[];
  unsigned char* smem = pr_smem_raw + ((128 - (smem_u32(pr_smem_raw) & 127)) & 127);
  unsigned char* e_op = smem;                       // E_y hi, lo, E_x hi, lo
  unsigned char* g_op = e_op + 4 * kPairE;          // per target: Gram operands of P and of V
  constexpr uint32_t kOp = pair_op(P), kRaw = pair_raw(P);
  float2* raw = reinterpret_cast<float2*>(g_op + 4 * kOp);  // [tile parity][W, V]
  // mbarriers, per target: leg operands ready, done; Gram operands ready,
  // done; per tile parity: tile arrived, used; per target: its warps met
  uint64_t* bars = reinterpret_cast<uint64_t*>(raw + 4 * kRaw);
  const uint32_t bar_leg = smem_u32(bars), bar_leg_done = bar_leg + 16, bar_ready = bar_leg + 32, bar_done = bar_leg + 48,
                 bar_full = bar_leg + 64, bar_free = bar_leg + 80, bar_group = bar_leg + 96;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  volatile int* fail = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;

  // persistent: an equal share of the tiles
  const long long share = (ntile_all + nblock - 1) / nblock, first_tile = block * share;
  const long long last_tile = min(ntile_all, first_tile + share);
  if (first_tile >= last_tile) return;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int i = 0; i < 14; ++i) {
      const int k = i / 2;  // as listed above
      const uint32_t count = k == 1 || k == 3 ? 1u : k == 4 ? 32u * kPairLoaders : k == 5 ? (uint32_t)kPairWarps : (uint32_t)kPairGroup;
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bars + i)), "r"(count));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *fail = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // Tensor memory per target: A's four blocks of kBlk columns at 0, D1 and D2
  // (2 kBlk each) after them, N's 128 columns over A when its MMAs are done
  // (four planes: no room) or after D (eight: the next tile's A and its MMAs
  // do not wait for this tile's N).
  constexpr uint32_t kBlk = P == 4 ? 32 : 16, kColP = 4 * kBlk, kColN = P == 4 ? 0 : 8 * kBlk;
  constexpr bool kAhead = P != 4;
  constexpr uint32_t kStages = P == 4 ? 2 : 1;  // of 8 P contraction columns: N starts afresh after 64

  // A bounded wait by a whole warp; false (for the whole warp) when it or
  // any other thread of the CTA gave up.
  auto wait = [&](uint32_t bar, uint32_t phase) -> bool {
    bool ok = __all_sync(0xffffffffu, mbar_try(bar, phase));
    for (int i = 0; i < kPairWaitLimit && !ok; ++i) {
      ok = __all_sync(0xffffffffu, mbar_try(bar, phase));
      if (!ok && (i & 1023) == 1023 && __any_sync(0xffffffffu, *fail)) break;
    }
    if (!ok) *fail = 1;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ok;
  };

  // The register split is made inside each role's branch, so that no path
  // leads from the smaller share into the converting warps' code.
  if (warp < kPairWarps) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPairRegsWork));
    // two groups of warps, one per target, each at its own pace; this
    // thread's row of a tile, (o, x) for target x, (o, y) for y; of its
    // groups of four columns, j, those with j % 2 == g
    const uint32_t target = (uint32_t)warp / kPairGroup, w8 = (uint32_t)warp % kPairGroup;
    const int row = 32 * (int)(w8 & 3) + lane;
    const uint32_t g = w8 >> 2;
    const uint32_t lanes = tmem + 256u * target + ((uint32_t)(32 * (w8 & 3)) << 16);
    unsigned char* const ops = g_op + target * 2 * kOp;
    double acc[32];
    // of the chunk's task: groups in a row, this thread's place in a tile and
    // in the operands
    uint32_t n = 0, op_row = 0, along_x = 1;
    bool in = false;  // this thread has a row
    PairRow<P> pr_row;

    // N of this row: columns 8 i + 4 g + k (those whose place this warp's
    // part of the next A takes), v against the hi rows of V, u against the lo
    // ones; of a hi row u is 2^-11 of v and they meet in FP64, a lo row's are
    // both that small
    auto drain = [&]() {
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        float v[8], u[8];
        const uint32_t c = lanes + kColN + 4u * g + 16u * h;
        tmem_ld4_async(c, v);
        tmem_ld4_async(c + 8, v + 4);
        tmem_ld4_async(c + 64, u);
        tmem_ld4_async(c + 72, u + 4);
        tmem_ld_wait16(v, v + 4, u, u + 4);
        if ((w8 & 3) < 2) {
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[8 * h + i] += (double)v[i] + (double)u[i];
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[8 * h + i] += (double)(v[i] + u[i]);
        }
      }
    };
    auto read4 = [&](const float2* t, uint32_t j, float4& re, float4& im) {
      if (target == 0 || along_x) pr_row.template read<true>(t, target != 0, j, re, im);
      else pr_row.template read<false>(t, true, j, re, im);
    };
    // rows of W as the A operand in tensor memory: [re_hi | im_hi | re_lo |
    // im_lo] of kBlk columns each
    auto put_a_form = [&](const float2* w, auto target_y, auto form) {
#pragma unroll
      for (uint32_t i = 0; i < kBlk / 8; ++i) {
        const uint32_t j = g + 2 * i;
        if (j < n) {
          float4 re, im, rh, rl, ih, il;
          const uint32_t c = lanes + 4 * j;
          pr_row.template read<decltype(form)::value>(w, decltype(target_y)::value, j, re, im);
          split4(re, rh, rl);
          split4(im, ih, il);
          tmem_st4(c, rh);
          tmem_st4(c + kBlk, ih);
          tmem_st4(c + 2 * kBlk, rl);
          tmem_st4(c + 3 * kBlk, il);
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    };
    auto put_a = [&](const float2* w) {
      if (target == 0) put_a_form(w, std::false_type{}, std::true_type{});
      else if (along_x) put_a_form(w, std::true_type{}, std::true_type{});
      else put_a_form(w, std::true_type{}, std::false_type{});
    };
    // P of this row, group j
    auto get_p = [&](uint32_t j, float4& re, float4& im) {
      float rr[4], ri[4], ir[4], ii[4];
      const uint32_t c = lanes + kColP + 4 * j, Np = 4 * n;
      tmem_ld4_async(c, rr);            // A_re E_re
      tmem_ld4_async(c + Np, ri);       // A_re E_im
      tmem_ld4_async(c + 2 * kBlk, ir);       // A_im E_re
      tmem_ld4_async(c + 2 * kBlk + Np, ii);  // A_im E_im
      tmem_ld_wait16(rr, ri, ir, ii);
      re = make_float4(rr[0] - ii[0], rr[1] - ii[1], rr[2] - ii[2], rr[3] - ii[3]);
      im = make_float4(ri[0] + ir[0], ri[1] + ir[1], ri[2] + ir[2], ri[3] + ir[3]);
    };
    // four consecutive contraction columns of one row (re and im) into an
    // operand: rows f (re_hi), 32 + f, 64 + f, 96 + f
    auto put_op = [&](unsigned char* p, float4 re, float4 im) {
      float4 rh, rl, ih, il;
      split4(re, rh, rl);
      split4(im, ih, il);
      *reinterpret_cast<float4*>(p) = rh;
      *reinterpret_cast<float4*>(p + 32 * 16) = ih;
      *reinterpret_cast<float4*>(p + 64 * 16) = rl;
      *reinterpret_cast<float4*>(p + 96 * 16) = il;
    };
    // operands written by this warp are visible to the MMAs issued after it
    auto publish = [&](uint32_t bar) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    uint32_t gram_ph = 0, leg_ph = 0, met_ph = 0;  // parities of the MMAs and meetings waited for
    auto gram_done = [&]() {
      const bool r = wait(bar_done + 8u * target, gram_ph);
      gram_ph ^= 1u;
      return r;
    };
    auto leg_done = [&]() {
      const bool r = wait(bar_leg_done + 8u * target, leg_ph);
      leg_ph ^= 1u;
      return r;
    };
    // One Gram stage, after the operands' last MMAs: this thread's groups
    // 2 s + g of P and of V
    auto stage = [&](const float2* v, uint32_t s) -> bool {
      float4 re, im, vr, vi;
      get_p(2 * s + g, re, im);
      read4(v, 2 * s + g, vr, vi);
      if (s > 0 && !gram_done()) return false;
      if (in) {
        unsigned char* op = ops + op_row + g * (P * pair_group(P));
        put_op(op, re, im);
        put_op(op + kOp, vr, vi);
      }
      if (s > 0 && s % kStages == 0) drain();
      publish(bar_ready + 8u * target);
      return true;
    };

    auto tile_ready = [&](uint32_t i) { return wait(bar_full + 8u * (i & 1u), (i >> 1) & 1u); };
    bool ok = true;
    uint32_t T = 0;  // tiles so far: tile T arrives in raw[T & 1]
    int cur = -1;
    for (PairChunks ch(tasks, begins, ntask, first_tile, last_tile); ok && ch.valid(); ++ch.chunk) {
    const LegPairTask& tk = tasks[ch.ti];
    const int ntile = min(tk.chunk_tiles, (int)((tk.n_outer + P - 1) / P) - ch.chunk * tk.chunk_tiles);
    if (ch.ti != cur) {  // no MMA is in flight between chunks
      cur = ch.ti;
      PairLayout<P> lay;
      lay.set(tk.L1 == 1, (uint32_t)tk.Dx, (uint32_t)tk.Dy);
      along_x = uniform(lay.along_x);
      n = uniform(target ? lay.Xp : lay.Yp) / 4;
      const uint32_t Np = target ? lay.Yp : lay.Xp;
      in = (uint32_t)row < P * Np;
      pr_row.set(lay, (uint32_t)row, g);
      uint32_t o, i;
      lay.row((uint32_t)row, Np, o, i);
      op_row = o * pair_group(P) + (i >> 3) * 128 + (i & 7) * 16;  // + P pair_group per group of four columns
      build_pair_e<MR>(tk, e_op, lay.Xp, lay.Yp, (int)target, (int)target + 1, (int)w8, lane, kPairGroup);
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[i] = 0.0;
    for (int t = 0; t < ntile && ok; ++t, ++T) {
      const float2* wr = raw + (size_t)(T & 1u) * 2 * kRaw;
      const float2* vr = wr + kRaw;
      if (!kAhead || t == 0) {
        if (!(ok = tile_ready(T))) break;
        put_a(wr);
        publish(bar_leg + 8u * target);
      }
      if (!(ok = leg_done())) break;
      for (uint32_t s = 0; s < n / 2 && ok; ++s) ok = stage(vr, s);
      if (!ok) break;
      if (lane == 0) mbar_arrive(bar_free + 8u * (T & 1u));
      if (kAhead && t + 1 < ntile) {
        if (!(ok = tile_ready(T + 1))) break;
        put_a(raw + (size_t)((T + 1) & 1u) * 2 * kRaw);
        publish(bar_leg + 8u * target);
      }
      if (!(ok = gram_done())) break;
      drain();
    }
    if (!ok) break;
    // rows r and 64 + r of D, then N, through shared memory (the target's Gram
    // operands are free)
    double* dsum = reinterpret_cast<double*>(ops);  // 64 x 64
    auto meet = [&]() {  // the target's warps
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_group + 8u * target);
      ok = wait(bar_group + 8u * target, met_ph);
      met_ph ^= 1u;
      return ok;
    };
    const int C = target == 0 ? tk.Dx : tk.Dy;
    double2* part = (target == 0 ? tk.part_x : tk.part_y) + (long long)ch.chunk * C * C;
    if (!meet()) break;
    auto spill = [&](int half) {
      if (row / 64 == half) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          double* d = dsum + (row & 63) + 65 * (8 * (i / 4) + 4 * (int)g + i % 4);
          *d = half ? acc[i] : *d + acc[i];
        }
      }
    };
    spill(1);
    if (!meet()) break;
    spill(0);
    if (!meet()) break;
    if (lane < C)
      for (int c2 = (int)w8; c2 < C; c2 += kPairGroup) {
        const double re = dsum[lane + 65 * c2] + dsum[32 + lane + 65 * (32 + c2)];
        const double im = dsum[32 + lane + 65 * c2] - dsum[lane + 65 * (32 + c2)];
        part[lane + (long long)C * c2] = make_double2(re, im);
      }
    if (!meet()) break;
    }  // chunks
    if (!ok && w8 == 0 && lane == 0) {
      // MMAs in flight get one more bounded wait before TMEM is freed
      atomicExch(&g_tc_error, 1);
      for (uint32_t ph = 0; ph < 2; ++ph) {
        mbar_wait(bar_leg_done + 8u * target, ph);
        mbar_wait(bar_done + 8u * target, ph);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPairRegsFeed));
    if (warp < kPairWarps + 2) {
      // ---- the issuing warps, one per target: MMAs in the order in which
      // its group publishes.  One elected thread issues; every value that
      // goes into an MMA is made warp-uniform first and the loops are
      // unrolled, so that operands sit in uniform registers (left to
      // per-thread registers each MMA took 170 cycles to issue, three times
      // its own time).
      const uint32_t target = uniform((uint32_t)(warp - kPairWarps)), base = uniform(tmem) + 256u * target;
      const uint32_t e0 = uniform(smem_u32(e_op)) + target * 2 * kPairE, g0 = uniform(smem_u32(g_op)) + target * 2 * kOp;
      uint32_t gram_ph = 0, leg_ph = 0;
      bool ok = true;
      const uint64_t da = smem_desc(g0, pair_group(P), 128), db = smem_desc(g0 + kOp, pair_group(P), 128);
      for (PairChunks ch(tasks, begins, ntask, first_tile, last_tile); ok && ch.valid(); ++ch.chunk) {
        const LegPairTask& tk = tasks[ch.ti];
        const int ntile = min(tk.chunk_tiles, (int)((tk.n_outer + P - 1) / P) - ch.chunk * tk.chunk_tiles);
        // target x absorbs E_y (K = Yp), y E_x
        const uint32_t k8 = uniform(((uint32_t)(target ? tk.Dx : tk.Dy) + 7u) >> 3), N2 = 16 * k8;
        for (int t = 0; t < ntile && ok; ++t) {
          if (!(ok = wait(bar_leg + 8u * target, leg_ph))) break;
          leg_ph ^= 1u;
          const uint32_t idesc = idesc_tf32(128, 0) | ((N2 >> 3) << 17);
          const uint64_t dh0 = smem_desc(e0, N2 * 16, 128), dl0 = smem_desc(e0 + kPairE, N2 * 16, 128);
          if (elect_one()) {
#pragma unroll
            for (uint32_t part = 0; part < 2; ++part)
#pragma unroll
              for (uint32_t s = 0; s < kBlk / 8; ++s)
                if (s < k8) {
                  const uint32_t d = base + kColP + 2 * kBlk * part, ah = base + kBlk * part + 8u * s;
                  const uint64_t dh = dh0 + s * 2 * N2, dl = dl0 + s * 2 * N2;  // two 16-byte K groups of N2 rows
                  mma_tf32_ts(d, ah, dh, idesc, s);
                  mma_tf32_ts(d, ah, dl, idesc, 1u);
                  mma_tf32_ts(d, ah + 2 * kBlk, dh, idesc, 1u);
                }
            mma_commit(bar_leg_done + 8u * target);
          }
          __syncwarp();
          for (uint32_t st = 0; st < k8; ++st) {
            if (!(ok = wait(bar_ready + 8u * target, gram_ph))) break;
            gram_ph ^= 1u;
            if (elect_one()) {
#pragma unroll
              for (uint32_t s = 0; s < P; ++s)
                mma_tf32(base + kColN, da + pair_group(P) / 8 * s, db + pair_group(P) / 8 * s, idesc_tf32(128, 128), st % kStages + s);
              mma_commit(bar_done + 8u * target);
            }
            __syncwarp();
          }
        }
      }
    } else {
      // ---- the loading warps: of each y the elements e of a tile, lanes along
      // memory, one or two elements per copy; padding is written as zeros
      uint32_t T = 0;
      bool ok = true;
      const uint32_t y0 = (uint32_t)(warp - kPairWarps - 2);
      for (PairChunks ch(tasks, begins, ntask, first_tile, last_tile); ok && ch.valid(); ++ch.chunk) {
        const LegPairTask& tk = tasks[ch.ti];
        const int ntile = min(tk.chunk_tiles, (int)((tk.n_outer + P - 1) / P) - ch.chunk * tk.chunk_tiles);
        const uint32_t Dx = (uint32_t)tk.Dx, Dy = (uint32_t)tk.Dy, L1 = (uint32_t)tk.L1, O = (uint32_t)tk.n_outer;
        PairLayout<P> lay;
        lay.set(L1 == 1, Dx, Dy);
        const float2* __restrict__ Wg = static_cast<const float2*>(tk.W);
        const ptrdiff_t VmW = static_cast<const float2*>(tk.V) - Wg;
        auto copy = [&](auto width, float2* dst, uint32_t o0) {
          constexpr uint32_t w = decltype(width)::value;
#pragma unroll 1
          for (uint32_t e = w * (uint32_t)lane; e < lay.PE; e += 32 * w) {
            uint32_t o, x;
            lay.row(e, lay.Xp, o, x);
            const uint32_t oo = o0 + o, hi = fast_div(oo, tk.div_l), lo = oo - hi * L1;
            const bool ok_ox = oo < O && x < Dx;
            const float2* p = Wg + (ok_ox ? (size_t)lo + (size_t)L1 * (x + Dx * (y0 + Dy * (size_t)hi)) : 0);
            const size_t dy = ok_ox ? (size_t)kPairLoaders * L1 * Dx : 0;
            float2* d = dst + y0 * lay.PE;
#pragma unroll 2
            for (uint32_t y = y0; y < lay.Yp; y += kPairLoaders) {
              const bool in = ok_ox && y < Dy;
              float2* de = d + (e ^ lay.swz(y));
              if constexpr (w == 2) {
                cp16(de, in ? p : Wg, in);
                cp16(de + kRaw, in ? p + VmW : Wg, in);
              } else {
                cp8(de, in ? p : Wg, in);
                cp8(de + kRaw, in ? p + VmW : Wg, in);
              }
              p += dy;
              d += kPairLoaders * lay.PE;
            }
          }
        };
        const bool wide = pair_wide(tk);
        for (int t = 0; t < ntile && ok; ++t, ++T) {
          const uint32_t st = T & 1u;
          if (T >= 2 && !(ok = wait(bar_free + 8u * st, ((T >> 1) - 1) & 1u))) break;
          float2* dst = raw + (size_t)st * 2 * kRaw;
          const uint32_t o0 = (uint32_t)(ch.chunk * tk.chunk_tiles + t) * P;
          if (wide) copy(std::integral_constant<uint32_t, 2>{}, dst, o0);
          else copy(std::integral_constant<uint32_t, 1>{}, dst, o0);
          // this thread's arrival, when its copies have landed
          asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_full + 8u * st) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// n4 tasks of four planes per tile (tiles4 tiles) on the first blocks4 CTAs,
// then n8 of eight: one launch, so that neither kind waits for the other's
// last CTAs.
template <typename MR>
__global__ void __launch_bounds__(tc::kPairThreads, 1)
    k_pair_gram_tc(const LegPairTask* __restrict__ tasks, const long long* __restrict__ begins, int n4, long long tiles4, int n8,
                   long long tiles8, int blocks4) {
  if ((int)blockIdx.x < blocks4) pair_gram<MR, 4>(tasks, begins, n4, tiles4, blockIdx.x, (uint32_t)blocks4);
  else pair_gram<MR, 8>(tasks + n4, begins + n4, n8, tiles8, blockIdx.x - (uint32_t)blocks4, gridDim.x - (uint32_t)blocks4);
}

// ---------------------------------------------------------------------------
// Both legs of a pair absorbed in one pass, out[x', y', o] =
// sum_{x, y} in[x, y, o] E_x[x, x'] E_y[y, y']: the W of the site's other pair
// (two absorptions of bp.h:137-152).
//
// Why: two launches of the leg kernel read and wrote the tensor twice; here it
// is read and written once, which leaves HBM (64 KB per tile at D = 32, about
// 2800 cycles per SM) and the two products' MMAs (1700 cycles) as bounds.
// One sweep of an 8x8 lattice's loop at D = 32: 1.86 ms in the leg kernel, 0.88 ms here (5400
// cycles per tile when planes are contiguous, 8000 when memory runs along o
// and a tile is 32-byte pieces); 6x6 at D = 16: 0.09 -> 0.04 ms.
//
// Tiles, rows and tensor-memory operands are those of pair_gram.  The first
// product's rows (o, x) go back over the tile they came from, the second
// takes rows (o, y) from there, and its rows return to the same place, from
// which the tile is written out as memory runs.  512 threads, two CTAs per SM
// (98 KB of shared memory, 256 tensor-memory columns each): one converts
// while the other waits.
// ---------------------------------------------------------------------------
namespace tc {
constexpr int kAbsorbThreads = 512;
constexpr uint32_t kAbsorbG = kAbsorbThreads / 128;  // warps that share a row
__host__ __device__ constexpr size_t absorb_smem_bytes() {
  return 128 + 4 * (size_t)kPairE + 2 * (size_t)kPairRawElems * 8 + 64;
}
}  // namespace tc

template <typename MR, uint32_t P>
__device__ __forceinline__ void pair_absorb(const LegPairTask* __restrict__ tasks, const long long* __restrict__ begins, int ntask,
                                            long long ntile_all, uint32_t block, uint32_t nblock) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char pr_smem_raw[];
  unsigned char* e_op = pr_smem_raw + ((128 - (smem_u32(pr_smem_raw) & 127)) & 127);  // E_y hi, lo, E_x hi, lo
  float2* raw = reinterpret_cast<float2*>(e_op + 4 * kPairE);                             // two tiles
  uint64_t* bar = reinterpret_cast<uint64_t*>(raw + 2 * kPairRawElems);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const long long share = (ntile_all + nblock - 1) / nblock, first = block * share, last = min(ntile_all, first + share);
  if (first >= last) return;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(256u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(1u));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot, base = uniform(tmem);
  constexpr uint32_t kColP = 128;  // A operand at 0, D1 at 128, D2 at 192

  // rows: (o, x) or (o, y); of a row's groups of four columns, j, this warp
  // has those with j % 4 == g
  const int row = 32 * (warp & 3) + lane;
  const uint32_t g = (uint32_t)warp >> 2, lanes = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  // of the task: its layout, this thread's row
  PairLayout<P> lay{1, 8, 8, 8 * P};
  PairRow<P> my;
  my.set(lay, 0, 0);
  bool in_x = false, in_y = false;
  // and its copies: two elements of every eighth y from cp_y on or one of
  // every fourth, from cp_d of a tile (four y's flip the swizzle by cp_flip)
  // and cp_off in memory, there cp_step apart (cp_plane per unit of o / L1)
  uint32_t cp_o = 0, cp_d = 0, cp_y = 0, cp_flip = 0, L1 = 1, Dy = 0, n_outer = 0;
  bool cp_mine = false, cp_pad = false, wide = false;
  size_t cp_off = 0, cp_step = 0, cp_plane = 0;
  FastDiv div_l{1, 1, 0};
  const float2* src = nullptr;
  ptrdiff_t dst = 0;  // output minus input

  // offset at y = cp_y of this thread's element in tile lt; false if it has none
  auto place = [&](uint32_t lt, size_t& off) {
    const uint32_t oo = lt * P + cp_o, hi = fast_div(oo, div_l);
    off = cp_off + (oo - hi * L1) + cp_plane * hi;
    return cp_mine && oo < n_outer;
  };
  auto load_tile = [&](uint32_t lt, int stage) {
    if (cp_mine || cp_pad) {
      size_t off;
      const bool ok = place(lt, off);
      const float2* p = ok ? src + off : src;
      float2* t = raw + (size_t)stage * kPairRawElems;
      uint32_t d = cp_d;
      if (wide) {
#pragma unroll 4
        for (uint32_t y = cp_y; y < lay.Yp; y += kAbsorbThreads / 64) {
          const bool in = ok && y < Dy;
          cp16(t + d, in ? p : src, in);
          p += cp_step;
          d += kAbsorbThreads / 64 * lay.PE;
        }
      } else {
#pragma unroll 4
        for (uint32_t y = cp_y; y < lay.Yp; y += kAbsorbG) {
          const bool in = ok && y < Dy;
          cp8(t + d, in ? p : src, in);
          p += cp_step;
          d = (d ^ cp_flip) + kAbsorbG * lay.PE;
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // rows of the tile as the A operand: [re_hi | im_hi | re_lo | im_lo]
  auto put_a_form = [&](const float2* t, bool target_y, auto form) {
    const uint32_t n = (target_y ? lay.Xp : lay.Yp) / 4;
#pragma unroll
    for (uint32_t j = g; j < 8; j += kAbsorbG)
      if (j < n) {
        const uint32_t c = lanes + 4 * j;
        float4 re, im, rh, rl, ih, il;
        my.template read<decltype(form)::value>(t, target_y, j, re, im);
        split4(re, rh, rl);
        split4(im, ih, il);
        tmem_st4(c, rh);
        tmem_st4(c + 32u, ih);
        tmem_st4(c + 64u, rl);
        tmem_st4(c + 96u, il);
      }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  };
  // the product's rows back over the tile
  auto put_back_form = [&](float2* t, bool target_y, auto form) {
    const uint32_t Np = target_y ? lay.Xp : lay.Yp, n = Np / 4;
    const bool valid = target_y ? in_y : in_x;
#pragma unroll
    for (uint32_t j = g; j < 8; j += kAbsorbG)
      if (j < n) {
        const uint32_t c = lanes + kColP + 4 * j;
        float rr[4], ri[4], ir[4], ii[4];
        tmem_ld4_async(c, rr);            // A_re E_re
        tmem_ld4_async(c + Np, ri);       // A_re E_im
        tmem_ld4_async(c + 64, ir);       // A_im E_re
        tmem_ld4_async(c + 64 + Np, ii);  // A_im E_im
        tmem_ld_wait16(rr, ri, ir, ii);
        if (valid)
          my.template write<decltype(form)::value>(t, target_y, j, make_float4(rr[0] - ii[0], rr[1] - ii[1], rr[2] - ii[2], rr[3] - ii[3]),
                   make_float4(ri[0] + ir[0], ri[1] + ir[1], ri[2] + ir[2], ri[3] + ir[3]));
      }
  };
  auto put_a = [&](const float2* t, bool target_y) {
    if (!target_y || lay.along_x) put_a_form(t, target_y, std::true_type{});
    else put_a_form(t, target_y, std::false_type{});
  };
  auto put_back = [&](float2* t, bool target_y) {
    if (!target_y || lay.along_x) put_back_form(t, target_y, std::true_type{});
    else put_back_form(t, target_y, std::false_type{});
  };
  auto leg_mma = [&](uint32_t which) {  // by warp 0; 0: E_y (K = Yp), 1: E_x
    const uint32_t k8 = uniform(which ? lay.Xp : lay.Yp) / 8, N2 = 16 * k8, idesc = idesc_tf32(128, 0) | ((N2 >> 3) << 17);
    const uint32_t op = uniform(smem_u32(e_op)) + which * 2 * kPairE;
    const uint64_t dh0 = smem_desc(op, N2 * 16, 128), dl0 = smem_desc(op + kPairE, N2 * 16, 128);
    if (elect_one()) {
#pragma unroll
      for (uint32_t part = 0; part < 2; ++part)
#pragma unroll
        for (uint32_t s = 0; s < 4; ++s)
          if (s < k8) {
            const uint32_t d = base + kColP + 64u * part, ah = base + 32u * part + 8u * s;
            const uint64_t dh = dh0 + s * 2 * N2, dl = dl0 + s * 2 * N2;
            mma_tf32_ts(d, ah, dh, idesc, s);
            mma_tf32_ts(d, ah, dl, idesc, 1u);
            mma_tf32_ts(d, ah + 64u, dh, idesc, 1u);
          }
      mma_commit(smem_u32(bar));
    }
    __syncwarp();
  };
  auto sync = [&]() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  };
  uint32_t phase = 0;
  bool ok = true;
  auto done = [&]() {  // every thread; the same answer for all
    const bool r = mbar_wait(smem_u32(bar), phase);
    phase ^= 1u;
    ok = !__syncthreads_or(!r);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return ok;
  };

  long long task_end = first;  // tile at which the current task ends
  uint32_t lt = 0;
  int ti = find_task(begins, ntask, first) - 1;
  bool loaded = false;
  for (long long tile = first; tile < last; ++tile, ++lt) {
    const int stage = (int)(tile - first) & 1;
    float2* t = raw + (size_t)stage * kPairRawElems;
    if (tile == task_end) {  // the next task; its first tile is loaded below
      const LegPairTask& tk = tasks[++ti];
      const uint32_t Dx = (uint32_t)tk.Dx;
      Dy = (uint32_t)tk.Dy;
      L1 = (uint32_t)tk.L1;
      n_outer = (uint32_t)tk.n_outer;
      div_l = tk.div_l;
      task_end = begins[ti] + (n_outer + P - 1) / P;
      lt = (uint32_t)(tile - begins[ti]);
      lay.set(L1 == 1, Dx, Dy);
      lay.along_x = uniform(lay.along_x);
      my.set(lay, (uint32_t)row, g & 1u);
      in_x = (uint32_t)row < P * lay.Xp;
      in_y = (uint32_t)row < P * lay.Yp;
      wide = pair_wide(tk);
      const uint32_t e = wide ? 2 * ((uint32_t)tid & 63u) : (uint32_t)row;
      uint32_t x;
      lay.row(e, lay.Xp, cp_o, x);
      cp_y = wide ? (uint32_t)tid >> 6 : g;
      cp_d = (e ^ lay.swz(cp_y)) + cp_y * lay.PE;
      cp_flip = lay.swz(4);
      cp_mine = e < lay.PE && x < Dx;
      cp_pad = e < lay.PE && !cp_mine;
      cp_off = (size_t)L1 * (x + (size_t)Dx * cp_y);
      cp_step = (size_t)L1 * Dx * (wide ? kAbsorbThreads / 64 : kAbsorbG);
      cp_plane = (size_t)L1 * Dx * Dy;
      src = static_cast<const float2*>(tk.V);
      dst = static_cast<const float2*>(tk.W) - src;
      loaded = false;
      build_pair_e<MR>(tk, e_op, lay.Xp, lay.Yp, 0, 2, warp, lane, kAbsorbThreads / 32);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (!loaded) {
      __syncthreads();  // the stage has been written out
      load_tile(lt, stage);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the tile is here; the other stage has been written out
    loaded = tile + 1 < task_end && tile + 1 < last;
    if (loaded) load_tile(lt + 1, stage ^ 1);
    put_a(t, false);
    sync();
    if (warp == 0) leg_mma(0);
    if (!done()) break;
    put_back(t, false);
    __syncthreads();
    put_a(t, true);
    sync();
    if (warp == 0) leg_mma(1);
    if (!done()) break;
    put_back(t, true);
    sync();
    size_t off;
    if (place(lt, off)) {
      float2* out = const_cast<float2*>(src) + dst + off;
      uint32_t d = cp_d;
      if (wide) {
#pragma unroll 4
        for (uint32_t y = cp_y; y < Dy; y += kAbsorbThreads / 64) {
          *reinterpret_cast<float4*>(out) = *reinterpret_cast<const float4*>(t + d);
          out += cp_step;
          d += kAbsorbThreads / 64 * lay.PE;
        }
      } else {
#pragma unroll 4
        for (uint32_t y = cp_y; y < Dy; y += kAbsorbG) {
          *out = t[d];
          out += cp_step;
          d = (d ^ cp_flip) + kAbsorbG * lay.PE;
        }
      }
    }
  }
  if (!ok && tid == 0) {
    // MMAs in flight get one more bounded wait before TMEM is freed
    atomicExch(&g_tc_error, 1);
    mbar_wait(smem_u32(bar), phase ^ 1u);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u));
  }
}

// The tasks' `W` is the output.
template <typename MR>
__global__ void __launch_bounds__(tc::kAbsorbThreads, 2)
    k_pair_absorb_tc(const LegPairTask* __restrict__ tasks, const long long* __restrict__ begins, int n4, long long tiles4, int n8,
                     long long tiles8, int blocks4) {
  if ((int)blockIdx.x < blocks4) pair_absorb<MR, 4>(tasks, begins, n4, tiles4, blockIdx.x, (uint32_t)blocks4);
  else pair_absorb<MR, 8>(tasks + n4, begins + n4, n8, tiles8, blockIdx.x - (uint32_t)blocks4, gridDim.x - (uint32_t)blocks4);
}

}  // namespace tnbp
