// The outgoing BP messages of small sites, one CTA each, in shared memory.
//
// For a site of degree g with bond dims D_k and physical dim d (n = d prod D
// elements), each target leg t gets
//   T_t = V x_{k != t} E_k                   (bp.h:137-152, legs in order)
//   N_t[c, c'] = sum_{q} T_t[.., c, ..] conj(V[.., c', ..])   (bp.h:157-166)
// normalized by its Frobenius norm, with the distance to the stored message
// (the condition's per-message term, bp.h:286-354), exactly as
// k_msg_finalize forms them.  The site tensor, two ping-pong buffers for the
// absorptions, the incoming messages and the Gram's partial sums all stay
// in shared memory, in FP64 whatever the storage precision: nothing but V,
// the messages and the results crosses HBM, and one launch covers every
// small site of a sweep (or of a server batch of many jobs), whatever their
// degrees and dims.  Sites too large for this (site_sweep_smem_bytes above
// kSiteSmemMax) take the per-level path of the sweep plan.
//
// What bounds it: the latency of one CTA's chain (three absorptions and a Gram
// at degree 4) while most SMs idle, so every target has a CTA of its own,
// which repeats the others' loads and absorptions, and indices are 32-bit.
// With one CTA per site and 64-bit indices a launch of the 10x10 random
// circuit took 34 us, one of the ragged 7x6 lattice 77 us (complex128); now
// 14 and 23 us, and the 4x4 chi 4 step 3.32 -> 2.94 ms.
//
// The Gram's partial sums are formed by P = 256 / C^2 thread groups over
// strided rows and reduced in a fixed order, so results do not depend on
// anything but the site's own data.
#pragma once
#include <cstdint>

#include "kernels.cuh"

namespace tnbp {

// SiteTask and site_sweep_smem_bytes are declared in kernels.cuh.

// grid: (sites, largest degree); CTAs beyond a site's degree leave at once.
template <typename R, typename MR>
__global__ void __launch_bounds__(kThreads) k_site_sweep(const SiteTask* __restrict__ tasks) {
  using CR = typename cvec<R>::type;
  using CM = typename cvec<MR>::type;
  extern __shared__ __align__(16) unsigned char site_smem[];
  __shared__ double red[32];
  const SiteTask* tk = tasks + blockIdx.x;
  const int g = tk->g, t = blockIdx.y;
  if (t >= g) return;
  const uint32_t n = (uint32_t)tk->n, tid = threadIdx.x;
  double2* Vs = reinterpret_cast<double2*>(site_smem);
  double2* buf[2] = {Vs + n, Vs + 2 * n};
  double2* Es = Vs + 3 * n;
  double2* part = Es;
  {
    const CR* V = static_cast<const CR*>(tk->V);
    for (uint32_t i = tid; i < n; i += kThreads) Vs[i] = to_d2(V[i]);
    for (int k = 0; k < g; ++k) {
      const uint32_t m = (uint32_t)(tk->D[k] * tk->D[k]);
      if (k != t) {
        const CM* E = static_cast<const CM*>(tk->E[k]);
        for (uint32_t i = tid; i < m; i += kThreads) part[i] = to_d2(E[i]);
      }
      part += m;
    }
  }
  __syncthreads();
  {
    // T_t: absorb the message of every other leg, in leg order
    const double2* src = Vs;
    const double2* e = Es;
    int which = 0;
    uint32_t L = 1, Lt = 1;
    for (int k = 0; k < g; ++k) {
      const uint32_t Dk = (uint32_t)tk->D[k];
      if (k == t) {
        Lt = L;
      } else {
        double2* dst = buf[which];
        which ^= 1;
        for (uint32_t i = tid; i < n; i += kThreads) {
          const uint32_t rest = i / L, l = i - rest * L, r = rest / Dk, kp = rest - r * Dk;
          const double2* a = src + l + L * Dk * r;
          const double2* ek = e + Dk * kp;
          double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
          for (uint32_t j = 0; j < Dk; ++j) cfma(acc, a[L * j], ek[j]);
          dst[i] = acc;
        }
        __syncthreads();
        src = dst;
      }
      L *= Dk;
      e += Dk * Dk;
    }
    // Gram over every index but leg t: C^2 outputs, P row groups each
    const uint32_t C = (uint32_t)tk->D[t], C2 = C * C;
    const uint32_t LC = Lt * C, Q = n / C;
    const uint32_t P = C2 >= kThreads ? 1 : kThreads / C2;
    for (uint32_t w = tid; w < C2 * P; w += kThreads) {
      const uint32_t p = w / C2, o = w - p * C2;
      const uint32_t c2 = o / C, c = o - c2 * C;
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
      for (uint32_t q = p; q < Q; q += P) {
        const uint32_t m = q / Lt, l = q - m * Lt;
        cfma_conj(acc, src[l + Lt * c + LC * m], Vs[l + Lt * c2 + LC * m]);
      }
      part[w] = acc;
    }
    __syncthreads();
    // fixed-order reduction of the groups, in place into part[0 .. C^2)
    double s_new = 0.0, s_old = 0.0;
    const CM* old = static_cast<const CM*>(tk->old[t]);
    for (uint32_t o = tid; o < C2; o += kThreads) {
      double2 v = part[o];
      for (uint32_t p = 1; p < P; ++p) v = v + part[p * C2 + o];
      part[o] = v;
      s_new += abs2(v);
      if (old) s_old += abs2(to_d2(old[o]));
    }
    const double nn = sqrt(block_sum(s_new, red));
    const double no = old ? sqrt(block_sum(s_old, red)) : 0.0;
    const double inv_n = nn > 0.0 ? 1.0 / nn : 1.0;
    const double inv_o = no > 0.0 ? 1.0 / no : 1.0;
    double d2 = 0.0;
    CM* out = static_cast<CM*>(tk->out[t]);
    for (uint32_t o = tid; o < C2; o += kThreads) {
      const double2 v = inv_n * part[o];
      if (old) d2 += abs2(v - inv_o * to_d2(old[o]));
      out[o] = from_d2<CM>(v);
    }
    d2 = block_sum(d2, red);
    if (tid == 0 && tk->dist[t]) *tk->dist[t] = sqrt(d2);
  }
}

}  // namespace tnbp
