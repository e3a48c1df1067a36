// hj_scan.cu -- the per-turn bins step on uniform bin centres: wake potential
// by a suffix scan, kick table, E0 update (sm_100a, FP64).
//
// Reference (MPI branch of apply_wakefield_inplace!, src/wakefield.jl:186-327):
//   g[i]   = delta(c_i, 0.15) * counts[i] / Σcounts                 :207-221, :238
//   pot[i] = current Σ_{j<=i} W[j] g[i-j]                           :231-243, :286-319
// with W[j] = F e^{c_j/cτ} (cos s c_j + a sin s c_j) where c_j <= 0, else 0
// (src/wakefield.jl:115-118).  On centres a step Δ apart W is a truncated
// geometric sequence: with J the last index with c_J <= 0,
//   W[J-d] = Re(A σ^d), 0 <= d <= J,  σ = e^{-Δ (1/cτ + i s)},  |σ| < 1,
// so with the suffix sums T[m] = Σ_{k>=m} σ^{k-m} g[k] = g[m] + σ T[m+1]
//   pot[i] = current Re A (T[i-J] - σ^{J+1} T[i+1]),   T[m] = σ^{-m} T[0] for m < 0
// (for i < J the factor on T[0] is σ^{J-i}).  The scan runs from the high bins
// down, where its factor contracts, so a rounding error is never amplified; the
// error is a few ulps of the largest |A| Σg, as an FFT convolution's is.  This
// takes O(B) operations per turn instead of the four length-B/2 complex FFTs
// of hj_wake.cu, which remain for centres that are not uniform.
//
// One cluster of C CTAs per bunch, NT threads each, E consecutive bins per
// thread: the thread's suffix sum, a weighted shuffle scan over the warp, over
// the warps, and (one cluster barrier) over the CTAs.  T[i-J], half a grid
// away, is read from the CTA that holds it through distributed shared memory.
// What bounds it is the chain of barriers and FP64 latencies, not bytes (80 B
// per bin and turn: 24 read, 24 cleared, 32 written) or operations (about 60 per
// bin).  16384 bins, serialised: 13.9 us against 42.7 for the FFT step and 10.1
// for the merge of block partials that it needed.  A whole turn of 1e5 particles at
// 4096 bins takes 15.5 us (30.5 with those two).
#include <cooperative_groups.h>

#include "hj_internal.h"

namespace hj {
namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// a + b c
__device__ __forceinline__ double2 cfma(double2 b, double2 c, double2 a) {
  return make_double2(fma(b.x, c.x, fma(-b.y, c.y, a.x)), fma(b.x, c.y, fma(b.y, c.x, a.y)));
}
__device__ __forceinline__ double2 shfl_down2(double2 v, int o) {
  return make_double2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o));
}

// x / n rounded as a division rounds it, from inv = 1/n rounded: the remainder of the
// product corrects it (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990).  x times inv alone is not exact for
// x = n m, so that particles at one z would have a length; a division is 0.3 us a turn.
__device__ __forceinline__ double quotient(double x, double n, double inv) {
  const double q = x * inv;
  return fma(fma(-q, n, x), inv, q);
}

constexpr int kPowLo = 128;                          // σ^0 .. σ^127
constexpr int kPowHi = (int)kMaxBins / kPowLo + 1;   // σ^{128 q}, q <= 128

constexpr int ilog2c(int v) { return v <= 1 ? 0 : 1 + ilog2c(v / 2); }

template <int NT, int E>
constexpr size_t scan_smem() {
  return sizeof(double2) * (size_t)(NT * E + kPowLo + kPowHi) + sizeof(double) * (size_t)(NT * E + 2);
}

// The turn's scalars past L1, which may hold the line as it was before the previous
// bins step wrote it: only a kernel's own wait makes plain loads see what other
// kernels wrote, and this one comes before it.
__device__ __forceinline__ TurnScalars load_scalars(const TurnScalars* p) {
  static_assert(sizeof(TurnScalars) % sizeof(long long) == 0, "whole words");
  TurnScalars s;
#pragma unroll
  for (int k = 0; k < (int)(sizeof(TurnScalars) / sizeof(long long)); ++k)
    reinterpret_cast<long long*>(&s)[k] = __ldcg(reinterpret_cast<const long long*>(p) + k);
  return s;
}

// All threads of the block, or of the cluster.
template <int C>
__device__ __forceinline__ void block_or_cluster_sync() {
  if constexpr (C > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// NT scanning threads and one more warp, which forms the turn's scalars (σ_z, the
// current, the E0 update) beside the scan.
template <int C, int NT, int E>
__device__ __forceinline__ void scan_body(const ScanArgs& a) {
  constexpr int L = NT * E, NW = NT / 32;
  static_assert(NT >= 256 && NW <= 31 && (L & (L - 1)) == 0 && C * L <= kMaxBins, "layout");
  constexpr int kLogE = ilog2c(E), kLogL = ilog2c(L);
  const int t = (int)threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool scalar = warp == NW;
  int rank = 0;
  if constexpr (C > 1) rank = (int)cg::this_cluster().block_rank();
  extern __shared__ __align__(16) double2 s_dyn[];
  double2* const s_T = s_dyn;               // [L] suffix sums within this CTA
  double2* const s_lo = s_T + L;            // [128] σ^r
  double2* const s_hi = s_lo + kPowLo;      // [129] σ^{128 q}
  double* const s_g = reinterpret_cast<double*>(s_hi + kPowHi);   // [L + 1] density, then pot
  __shared__ double2 s_agg[NW];             // warps' sums
  __shared__ double2 s_cagg;                // the CTA's
  __shared__ double2 s_K[NW][C];            // carries into the CTAs, a copy per warp
  __shared__ double s_sc[2];                // potential scale (NaN allowed), particles in range
  __shared__ double s_kick[C * NW];         // rank 0: Σ kick of every warp of the cluster
  const int B = a.use_wake ? a.B : 0, nc = B + 1;
  const int base = rank * L;
  TurnState* ts = a.ts;

  // before the pass has finished: the powers of σ and the smoothing weights
  // delta(c_i) (src/utils.jl:58-66) of this thread's bins base + t + k NT; the
  // scalar warp reads the turn's scalars, which the previous bins step wrote: every
  // block of this turn's pass had waited for it before it let this kernel start
  double lam[E];
  TurnScalars cur;
  double coef = 0.0;
  const double nd = (double)a.n, inv_n = 1.0 / nd;
  if (scalar) {
    cur = load_scalars(&ts->cur);
    // the wake current over σ_z (src/evolution.jl:373-386)
    coef = a.particle_factor / cur.E0 / (kTwoPi * a.params.radius) /
           (cur.eta0 * (a.sigma_E0_initial * a.sigma_E0_initial));
  } else if (B > 0) {
    if (t < kPowLo + kPowHi - 1) {
      const int n = t < kPowLo ? t : (t - kPowLo) * kPowLo;
      double2 p = make_double2(1.0, 0.0);
#pragma unroll
      for (int b = 0; b < kScanPowers; ++b)
        if ((n >> b) & 1) p = cmul(p, a.pw[b]);
      s_lo[t] = p;
    }
    if (t == 0) s_hi[kPowHi - 1] = a.pw[kScanPowers - 1];
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int i = base + t + k * NT;
      const double c = fma((double)(i - a.J), a.cstep, a.cJ);
      lam[k] = i < B ? a.lam_pref * exp(c * c * a.lam_f) : 0.0;
    }
  }
  grid_dependency_wait();
  grid_launch_dependents();

  // 1. this turn's counts and cell sums (the accumulators the pass added to, left
  //    zero for the next one), and the pass's per-block sums in a fixed order
  unsigned long long cn[E], cw[E], xn = 0ull, xw = 0ull;
  // cell B of a grid that fills the cluster's C L bins: the last CTA's thread 0
  const bool extra = B > 0 && B == C * L && rank == C - 1 && t == 0;
  double sum[kNumSums] = {0.0, 0.0, 0.0, 0.0};   // Σz, Σz², Σ(ΔE - ΔE_start), particles in range
  double sigma_z = 0.0, current = 0.0;
  if (scalar) {
    const double2* part = reinterpret_cast<const double2*>(a.part_sum);
    constexpr int U = 5;   // a wave of 148 blocks in one round of loads
    for (int b0 = lane; b0 < a.nblk; b0 += 32 * U) {
      double2 u[U], w[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int b = b0 + 32 * q;
        u[q] = b < a.nblk ? __ldcg(part + 2 * (size_t)b) : make_double2(0.0, 0.0);
        w[q] = b < a.nblk ? __ldcg(part + 2 * (size_t)b + 1) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        sum[0] += u[q].x;
        sum[1] += u[q].y;
        sum[2] += w[q].x;
        sum[3] += w[q].y;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < kNumSums; ++k) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
    double scale = 0.0;
    if (B > 0) {
      // src/utils.jl:593-605, src/evolution.jl:357
      if (a.n > 1) {
        const double mean = quotient(sum[0], nd, inv_n);
        double v = fma(-mean, mean, quotient(sum[1], nd, inv_n)) * a.n_over_n1;
        if (!(v > 0.0)) v = v != v ? v : 0.0;
        sigma_z = sqrt(v);
      }
      current = coef * sigma_z;
      if (sum[3] > 0.0) scale = current / sum[3];                // src/wakefield.jl:207, :305
    }
    if (lane == 0) {
      s_sc[0] = scale;
      s_sc[1] = sum[3];
    }
  } else if (B > 0) {
    unsigned long long n[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int i = base + t + k * NT;
      n[k] = i < B ? __ldcg(a.acc + i) : 0ull;
      cn[k] = i < nc ? __ldcg(a.acc + B + i) : 0ull;
      cw[k] = i < nc ? __ldcg(a.acc + B + nc + i) : 0ull;
    }
    if (extra) {
      xn = __ldcg(a.acc + B + B);
      xw = __ldcg(a.acc + B + nc + B);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) s_g[t + k * NT] = lam[k] * (double)n[k];
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int i = base + t + k * NT;
      if (i < B) a.counts[i] = n[k];
      if (a.clear) {
        if (i < B) a.acc[i] = 0ull;
        if (i < nc) a.acc[B + i] = a.acc[B + nc + i] = 0ull;
      }
    }
    if (extra && a.clear) a.acc[B + B] = a.acc[B + nc + B] = 0ull;
  }
  if (B > 0) {
    __syncthreads();
    // 2. suffix sums: thread (E bins), warp, CTA
    double2 v = make_double2(0.0, 0.0);
    double g[E];
    if (!scalar) {
#pragma unroll
      for (int k = E - 1; k >= 0; --k) {
        g[k] = s_g[t * E + k];
        v = cfma(v, a.pw[0], make_double2(g[k], 0.0));
      }
#pragma unroll
      for (int s = 0; s < 5; ++s) {
        const double2 u = shfl_down2(v, 1 << s);
        if (lane + (1 << s) < 32) v = cfma(u, a.pw[kLogE + s], v);
      }
      if (lane == 0) s_agg[warp] = v;
    }
    __syncthreads();
    if (!scalar) {
      double2 x = shfl_down2(v, 1);                   // the warp's sum above this thread
      if (lane == 31) x = make_double2(0.0, 0.0);
      double2 w = lane < NW ? s_agg[lane] : make_double2(0.0, 0.0);
#pragma unroll
      for (int s = 0; (1 << s) < NW; ++s) {
        const double2 u = shfl_down2(w, 1 << s);
        if (lane + (1 << s) < NW) w = cfma(u, a.pw[kLogE + 5 + s], w);
      }
      if (t == 0) s_cagg = w;
      const double2 wc = make_double2(__shfl_sync(0xffffffffu, w.x, (warp + 1) & 31),
                                      __shfl_sync(0xffffffffu, w.y, (warp + 1) & 31));
      if (warp < NW - 1) {
        const int d = E * (31 - lane);
        x = cfma(cmul(s_lo[d & (kPowLo - 1)], s_hi[d / kPowLo]), wc, x);
      }
#pragma unroll
      for (int k = E - 1; k >= 0; --k) {
        x = cfma(x, a.pw[0], make_double2(g[k], 0.0));
        s_T[t * E + k] = x;
      }
    }
    block_or_cluster_sync<C>();
    // 3. carries into the CTAs: K_c = T[(c+1) L]
    if (!scalar) {
      if constexpr (C > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        if (lane < C) {
          double2 K = make_double2(0.0, 0.0);
#pragma unroll
          for (int c = C - 1; c > 0; --c) {
            const double2 u = *cluster.map_shared_rank(&s_cagg, c);
            if (c > lane) K = cfma(K, a.pw[kLogL], u);
          }
          s_K[warp][lane] = K;
        }
        __syncwarp();
      }
    }
    auto pw = [&](int n) { return cmul(s_lo[n & (kPowLo - 1)], s_hi[n / kPowLo]); };
    auto T_at = [&](int m) {                          // 0 <= m < B
      const int r = m & (L - 1);
      if constexpr (C == 1) {
        return s_T[r];
      } else {
        const int c = m >> kLogL;
        return cfma(pw(L - r), s_K[warp][c], *cg::this_cluster().map_shared_rank(s_T + r, c));
      }
    };
    const double scale = s_sc[0];
    const bool conv = s_sc[1] > 0.0;                  // src/wakefield.jl:305-311
    double2 T0;
    auto pot_at = [&](int i) {
      double2 f = i >= a.J ? T_at(i - a.J) : cmul(pw(a.J - i), T0);
      if (i + 1 < B) {
        const double2 u = T_at(i + 1);
        f = cfma(make_double2(-u.x, -u.y), a.tau, f);
      }
      const double p = scale * fma(a.A.x, f.x, -(a.A.y * f.y));
      return conv ? p : 0.0;
    };
    // 4. the potential at this CTA's bins and the one below them (s_g[1 + r] =
    //    pot[base + r])
    if (!scalar) {
      T0 = T_at(0);
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const int i = base + t + k * NT;
        if (i < B) {
          const double p = pot_at(i);
          s_g[1 + t + k * NT] = p;
          a.pot[i] = p;
          if (i == 0) a.pot[-1] = p;
        }
      }
      if (t == NT - 1 && base > 0 && base - 1 < B) s_g[0] = pot_at(base - 1);
    }
    __syncthreads();
    // 5. kick table of the next pass, B + 1 cells: cell j in 1..B-1 spans centres
    // c[j-1]..c[j] and holds (pot[j-1], pot[j] - pot[j-1]); cells 0 and B are
    // flat: pot[0] below c1, and above cB the value the reference's clamped
    // interpolation takes there, pot[hi] (1 - w) + pot[hi+1] w with u =
    // (cB - c1)/Δc rounded as it rounds it (pot[B-2] when u is exactly B-1,
    // src/wakefield.jl:80-102).  With C[j] particles deposited in cell j and
    // S[j] = Σ w·2^24 over them, the same table gives
    //   Σ_i lerp(pot, z_i) = Σ_j C[j] pot_j + 2^-24 Σ_j S[j] step_j.
    if (!scalar) {
      double kick = 0.0;
      auto cell = [&](int j, unsigned long long n, unsigned long long sw) {
        double p0, d = 0.0;
        if (j < B) {
          p0 = s_g[j - base + (j > 0 ? 0 : 1)];
          if (j > 0) d = s_g[j - base + 1] - p0;
        } else if (B >= 2) {
          p0 = __dadd_rn(__dmul_rn(pot_at(a.hi_idx), __dsub_rn(1.0, a.hi_w)),
                         __dmul_rn(pot_at(a.hi_idx + 1), a.hi_w));
        } else {
          p0 = pot_at(0);
        }
        a.potd[j] = make_double2(p0, d);
        kick += (double)n * p0 + (double)sw * 5.9604644775390625e-08 * d;
      };
#pragma unroll
      for (int k = 0; k < E; ++k) {
        const int j = base + t + k * NT;
        if (j < nc) cell(j, cn[k], cw[k]);
      }
      if (extra) cell(B, xn, xw);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) kick += __shfl_down_sync(0xffffffffu, kick, o);
      if (lane == 0) {
        double* p = s_kick + rank * NW + warp;
        if constexpr (C > 1) p = cg::this_cluster().map_shared_rank(p, 0);
        *p = kick;
      }
    }
    block_or_cluster_sync<C>();
  }
  // 6. E0 update and next-turn scalars (src/evolution.jl:401-451, :300-304)
  if (scalar && rank == 0) {
    double kick = 0.0;
    if (B > 0) {
#pragma unroll
      for (int q = 0; q < (C * NW + 31) / 32; ++q)
        if (q * 32 + lane < C * NW) kick += s_kick[q * 32 + lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) kick += __shfl_down_sync(0xffffffffu, kick, o);
    }
    if (lane == 0) {
      const TurnSums u{sum[0], sum[2], sum[3], sigma_z, current, kick, B > 0 && sum[3] > 0.0};
      finish_turn(ts, cur, a.params, a.n, a.sigma_E0_initial, B > 0, u);
    }
  }
}

template <int C, int NT, int E>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(NT + 32, 1) k_scan(ScanArgs a) {
  scan_body<C, NT, E>(a);
}

// The step of a batch: cluster i (CTAs C i .. C i + C - 1) runs bunch i; slots
// past the live count and bunches with no turns left return at once (the CTAs
// of a cluster read the same state before any writes it, so they agree).
template <int C, int NT, int E>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(NT + 32, 1)
    k_batch_scan(const ScanArgs* __restrict__ bunches, const int32_t* __restrict__ n_bunches) {
  const int i = (int)(blockIdx.x / C);
  if (i >= *n_bunches) {
    grid_dependency_wait();   // every block completes after the kernels before it
    return;
  }
  __shared__ ScanArgs s_a;
  const int* src = reinterpret_cast<const int*>(bunches + i);
  for (int k = threadIdx.x; k < (int)(sizeof(ScanArgs) / sizeof(int)); k += NT + 32)
    reinterpret_cast<int*>(&s_a)[k] = __ldg(src + k);
  __syncthreads();
  // written by the previous bins step, which every block of this turn's pass has
  // waited for before it let this kernel start
  if (__ldcg(&s_a.ts->turns_left) <= 0) {
    grid_dependency_wait();
    return;
  }
  scan_body<C, NT, E>(s_a);
}

struct ScanForm {
  int C, NT, E;
  const void* fn;
  size_t smem;
};
template <int C, int NT, int E>
ScanForm plain_form() {
  return {C, NT, E, (const void*)k_scan<C, NT, E>, scan_smem<NT, E>()};
}
template <int C, int NT, int E>
ScanForm batch_form() {
  return {C, NT, E, (const void*)k_batch_scan<C, NT, E>, scan_smem<NT, E>()};
}

// Up to 1024 bins a CTA alone is faster than a cluster's barriers; above, one
// bin per thread while 8 CTAs hold them (1e5 particles, us a turn: 2048 bins 15.0 as
// 8 x 256 x 1 against 15.5 as 2 x 512 x 2 and 15.7 as 1 x 512 x 4; 4096 bins 16.2 as
// 8 x 512 x 1 against 16.9 as 4 x 512 x 2 and 18.9 as 2 x 512 x 4; 1000 bins 13.6
// as 1 x 512 x 2 against 14.5 as 4 x 512 x 1; 16384 bins 30.2 as 8 x 512 x 4 against
// 33.7 as 8 x 256 x 8).
ScanForm plain_scan_form(int B) {
  if (B <= 512) return plain_form<1, 256, 2>();
  if (B <= 1024) return plain_form<1, 512, 2>();
  if (B <= 2048) return plain_form<8, 256, 1>();
  if (B <= 4096) return plain_form<8, 512, 1>();
  if (B <= 8192) return plain_form<8, 512, 2>();
  return plain_form<8, 512, 4>();
}

// A batch of bunches of up to max_B bins with `room` SMs for each of its slots: the most
// CTAs per bunch that fit the SMs at once for all slots, beyond that the fewest that hold
// the bins (us a turn: 32 bunches of 8192 bins 268 -> 259 with 4 x 512 x 4 instead of 4 x
// 256 x 8, 64 of 2048 37 -> 31, 16 of up to 8192 48 -> 44; 256 of 4096 877 -> 869 with
// 1 x 512 x 8 instead of 2 x 256 x 8, 886 with 4 x 256 x 4).
ScanForm batch_scan_form(int max_B, int room) {
  if (max_B <= 512) return batch_form<1, 256, 2>();
  if (max_B <= 1024) return batch_form<1, 512, 2>();
  if (max_B <= 2048) {
    if (room >= 4) return batch_form<4, 512, 1>();
    if (room >= 2) return batch_form<2, 512, 2>();
    return batch_form<1, 512, 4>();
  }
  if (max_B <= 4096) {
    if (room >= 8) return batch_form<8, 512, 1>();
    if (room >= 4) return batch_form<4, 512, 2>();
    if (room >= 2) return batch_form<2, 512, 4>();
    return batch_form<1, 512, 8>();
  }
  if (max_B <= 8192) {
    if (room >= 8) return batch_form<8, 512, 2>();
    if (room >= 4) return batch_form<4, 512, 4>();
    return batch_form<2, 512, 8>();
  }
  if (room >= 8) return batch_form<8, 512, 4>();
  return batch_form<4, 512, 8>();
}

}  // namespace

cudaError_t prepare_scan_kernels(int max_smem) {
  for (int B = 256; B <= (int)kMaxBins; B *= 2) {
    cudaError_t e = allow_dynamic_smem(plain_scan_form(B).fn, max_smem);
    for (int room = 1; room <= 8 && e == cudaSuccess; room *= 2)
      e = allow_dynamic_smem(batch_scan_form(B, room).fn, max_smem);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_scan(const ScanArgs& a, cudaStream_t st) {
  const ScanForm f = plain_scan_form(a.use_wake ? a.B : 0);
  void* args[] = {const_cast<ScanArgs*>(&a)};
  PdlConfig l(dim3(f.C), dim3(f.NT + 32), f.smem, st);
  return cudaLaunchKernelExC(&l.cfg, f.fn, args);
}

cudaError_t launch_batch_scan(const ScanArgs* d_bunches, const int32_t* d_n_bunches,
                              int max_bunches, int max_B, int room, cudaStream_t st) {
  const ScanForm f = batch_scan_form(max_B, room);
  void* args[] = {const_cast<ScanArgs**>(&d_bunches), const_cast<int32_t**>(&d_n_bunches)};
  PdlConfig l(dim3(f.C * (max_bunches > 0 ? max_bunches : 1)), dim3(f.NT + 32), f.smem, st);
  return cudaLaunchKernelExC(&l.cfg, f.fn, args);
}

}  // namespace hj
