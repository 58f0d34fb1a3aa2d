// phl_eos_batch.cuh -- batched Helmholtz (rho, e) -> T inversion (helm_rhoe_given,
// source/source.F90:24982-25019) on independent samples, with three initial guesses:
//   PHL_GUESS_WARM     caller-provided T (the reference's warm start, source.F90:13649)
//   PHL_GUESS_MLP      learned guess (phl_mlp.cuh), judged by <= 3 Newton iterations
//   PHL_GUESS_BRACKET  cold guess: bisection over the table's T nodes for E(rho,T_j) <= e,
//                      then linear interpolation of E between the bracketing nodes
// Newton always finishes to the reference tolerance (helm_tol = 1e-11), so only the iteration
// count depends on the guess.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdlib>
#include <string>
#include "phl_device.cuh"
#include "phl_mlp.cuh"

#define PHL_GUESS_BRACKET 2
#ifndef PHL_GUESS_MLP
#define PHL_GUESS_MLP 1
#endif

namespace phl {

// Resident blocks of 128 threads per SM the inversion kernels are compiled for: 3 (168 registers).
// 2^22 samples on B200, learned guess (guess in the same kernel) 2.62 ms against 2.84 at 4 (128 registers, 850 B of spills) and
// 2.91 at 2 (unbounded); 10^6 samples, bracket guess 0.49 ms against 0.55 and 0.55.  The 36
// coefficients kept in shared memory between the evaluations of a solve ran 3 to 5% slower.
constexpr int EOS_MINB = 3;
// Without p and cs the warm start's kernel holds no full evaluation and fits 4 blocks (128 registers, no
// spills): 2^20 samples from a guess 0.1% off 202 us against 220 at 3 and 268 at 5 (with p and cs 320 at
// 3, 335 at 4).
constexpr int EOS_MINB_WARM = 4;
// single energies: 2^20 88 us with blocks of 128, 5 per SM, against 96 with 2 blocks of 256
constexpr int ENERGY_THREADS = 128, ENERGY_MINB = 5;

// cold guess; returns the number of EoS evaluations the search used
__device__ __forceinline__ int bracket_guess(const HelmTable &h, const HelmRho &r, HelmTemp &t, double e, double &Tg) {
  int lo = 0, hi = h.nT - 1;
  double r0[3], r1[3], elo, ehi, dd;
  helm_rho_bases(r, r0, r1);
  elo = helm_energy_at_node(h, r, r0, r1, lo + 1);
  if (e <= elo) { Tg = __ldg(h.T + lo); return 1; }
  helm_energy<false>(h, r, r0, r1, t, __ldg(h.T + hi) * 0.999999, ehi, dd);
  if (e >= ehi) { Tg = __ldg(h.T + hi) * 0.999999; return 2; }
  int evals = 2;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    const double em = helm_energy_at_node(h, r, r0, r1, mid + 1);
    ++evals;
    if (em <= e) { lo = mid; elo = em; } else { hi = mid; ehi = em; }
  }
  double t0 = __ldg(h.T + lo), t1 = __ldg(h.T + hi);
  double w = (e - elo) / (ehi - elo);
  Tg = t0 + w * (t1 - t0);
  return evals;
}

__global__ void __launch_bounds__(ENERGY_THREADS, ENERGY_MINB) k_eos_energy(HelmTable h, long long n,
                                                                            const double *rho, const double *T,
                                                                            const double *abar, const double *zbar,
                                                                            double *e) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  e[t] = helm_given2_energy(h, rho[t], T[t], abar[t], zbar[t]);
}

// per-warp sums of the batch statistics into the context's counters
// (slots: calls, iterations, non-converged, clamped, mlp accepted, mlp rejected, guess evaluations)
struct EosStat {
  unsigned long long v[7] = {0, 0, 0, 0, 0, 0, 0};
  __device__ __forceinline__ void flush(unsigned long long *stat) const {
    const int slot[7] = {STAT_NEWTON_CALLS, STAT_NEWTON_ITERS, STAT_NEWTON_NONCONV, STAT_NEWTON_CLAMP,
                         STAT_MLP_ACC,      STAT_MLP_REJ,      STAT_GUESS_EVALS};
#pragma unroll
    for (int q = 0; q < 7; ++q) {
      unsigned long long x = v[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if ((threadIdx.x & 31) == 0 && x) atomicAdd(stat + slot[q], x);
    }
  }
};

// outputs of one finished inversion (OUT: p or cs among them)
template <bool OUT>
__device__ __forceinline__ void eos_finish(const HelmTable &h, long long t, const HelmRho &r, HelmTemp &ht,
                                           double Tg, int used, double *T, double *p, double *cs, int *iters) {
  T[t] = Tg;
  if (OUT && (p || cs)) {
    double P, E, snd, cv;
    helm_full(h, r, ht, Tg, P, E, snd, cv);
    if (p) p[t] = P;
    if (cs) cs[t] = snd;
  }
  if (iters) iters[t] = used;
}

// Learned guess, phase 0: the network's log10 T of every sample, left in `guess` for phase 1.  A block
// takes 128 samples: features (the cold energy from 12 table coefficients), one tensor-core product,
// the FP32 layers as constant-bank operands.  A kernel of its own, so that the waits of the product and
// the block's barriers are hidden by 8 blocks an SM instead of the 3 that the Newton's registers leave
// (in one kernel, and with the FP32 layers read from memory, 2^22 samples took 2.62 ms, now 2.07).
static __global__ void __launch_bounds__(128, 8) k_eos_guess(HelmTable h, const __grid_constant__ MlpSmall w,
                                                             const __nv_bfloat16 *w2bf, long long n, const double *rho,
                                                             const double *e, const double *abar, const double *zbar,
                                                             float *guess, unsigned long long *stat) {
  extern __shared__ __align__(128) unsigned char sm[];
  MlpUmmaSmem &S = *reinterpret_cast<MlpUmmaSmem *>(sm);
  mlp_cta_setup(w2bf, S);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float feat[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (t < n) mlp_features(rho[t], e[t] - mlp_cold_energy(h, rho[t], abar[t], zbar[t]), abar[t], zbar[t], feat);
  bool ok = true, have = false;
  const float lT = mlp_forward_tile(w, feat, S, 0u, ok, have, stat + STAT_TC_STALLED);
  mlp_cta_teardown(S);
  if (t < n) guess[t] = lT;
}

// Phase 1.  Warm or bracket guess: the full Newton.  Learned guess: the one that phase 0 left in `lT`,
// judged by at most 3 reference Newton iterations; a sample whose guess did not converge within them
// without a reset is appended to `queue` (queue[0] = count, then index | judged iterations << 56) for
// phase 2, so that the fallback runs in converged warps instead of stalling the accepted lanes.
template <int GUESS, bool OUT>
__global__ void __launch_bounds__(128, GUESS == PHL_GUESS_WARM && !OUT ? EOS_MINB_WARM : EOS_MINB)
k_eos_invert(HelmTable h, long long n, const double *rho, const double *e, const double *abar, const double *zbar,
             double *T, double *p, double *cs, int *iters, const float *lT, unsigned long long *stat,
             unsigned long long *queue) {
  constexpr bool LEARNED = GUESS == PHL_GUESS_MLP;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  EosStat st;
  bool reject = false;
  int judged = 0;
  if (t < n) {
    const double ee = e[t];
    const HelmRho r = helm_rho_part(h, rho[t], abar[t], zbar[t]);
    HelmTemp ht;
    double Tg;
    int used = 0, clamped = 0;
    bool conv = false;
    if constexpr (LEARNED) {
      Tg = fmin(fmax(exp10((double)lT[t]), h.Tl * 1.000001), h.Th * 0.999999);
      st.v[6] = 1;  // the cold energy of phase 0
      used = helm_rhoe_newton(h, r, ht, ee, Tg, 3, clamped, &conv);
      st.v[3] = clamped;
      if (conv && clamped == 0) {
        st.v[0] = 1;
        st.v[1] = used;
        st.v[4] = 1;
        eos_finish<OUT>(h, t, r, ht, Tg, used, T, p, cs, iters);
      } else {
        reject = true;
        judged = used;
        st.v[5] = 1;
      }
    } else {
      if constexpr (GUESS == PHL_GUESS_BRACKET) st.v[6] = bracket_guess(h, r, ht, ee, Tg);
      else Tg = T[t];
      used = helm_rhoe_newton(h, r, ht, ee, Tg, 100, clamped, &conv);
      st.v[0] = 1;
      st.v[1] = used;
      st.v[2] = !conv;
      st.v[3] = clamped;
      eos_finish<OUT>(h, t, r, ht, Tg, used, T, p, cs, iters);
    }
  }
  if constexpr (LEARNED) {
    // warp-aggregated append of the rejected samples
    const unsigned mask = __ballot_sync(0xffffffffu, reject);
    if (mask) {
      const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
      unsigned long long base = 0;
      if (lane == leader) base = atomicAdd(queue, (unsigned long long)__popc(mask));
      base = __shfl_sync(0xffffffffu, base, leader);
      if (reject)
        queue[1 + base + __popc(mask & ((1u << lane) - 1u))] =
            (unsigned long long)t | ((unsigned long long)judged << 56);
    }
  }
  st.flush(stat);
}

// Phase 2 of the learned guess: the reference Newton from the bracket guess for the rejected
// samples (grid-stride over the queue written by phase 1)
__global__ void __launch_bounds__(128, EOS_MINB) k_eos_fallback(HelmTable h, const unsigned long long *queue,
                                                      const double *rho, const double *e, const double *abar,
                                                      const double *zbar, double *T, double *p, double *cs,
                                                      int *iters, unsigned long long *stat) {
  const long long count = (long long)queue[0];
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  // every lane runs the same number of trips so the warp-level flush stays converged
  const long long trips = (count + stride - 1) / stride;
  EosStat st;
  for (long long k = 0; k < trips; ++k) {
    const long long q = first + k * stride;
    if (q < count) {
      const unsigned long long ent = queue[1 + q];
      const long long t = (long long)(ent & ((1ull << 56) - 1));
      const int judged = (int)(ent >> 56);
      const double ee = e[t];
      const HelmRho r = helm_rho_part(h, rho[t], abar[t], zbar[t]);
      HelmTemp ht;
      double Tg;
      st.v[6] += bracket_guess(h, r, ht, ee, Tg);
      int clamped = 0;
      bool conv = false;
      const int used = helm_rhoe_newton(h, r, ht, ee, Tg, 100, clamped, &conv);
      st.v[0] += 1;
      st.v[1] += judged + used;
      st.v[2] += !conv;
      st.v[3] += clamped;
      eos_finish<true>(h, t, r, ht, Tg, judged + used, T, p, cs, iters);
    }
  }
  st.flush(stat);
}

// Launch the inversion on stream s (no synchronisation).  `queue` (n + 1 entries) and `lT` (n) are
// needed for the learned guess only.  Returns 0 or a cudaError_t.
inline int eos_launch(const HelmTable &h, cudaStream_t s, long long n, const double *rho, const double *e,
                      const double *abar, const double *zbar, double *T, double *p, double *cs, int *iters,
                      int guess, const Mlp &mlp, unsigned long long *stat, unsigned long long *queue, float *lT, int nsm) {
  const unsigned blocks = (unsigned)((n + 127) / 128);
  if (guess != PHL_GUESS_MLP) {
    auto k = guess == PHL_GUESS_BRACKET ? k_eos_invert<PHL_GUESS_BRACKET, true>
                                        : (p || cs ? k_eos_invert<PHL_GUESS_WARM, true> : k_eos_invert<PHL_GUESS_WARM, false>);
    k<<<blocks, 128, 0, s>>>(h, n, rho, e, abar, zbar, T, p, cs, iters, nullptr, stat, nullptr);
    return (int)cudaGetLastError();
  }
  const size_t sm = sizeof(MlpUmmaSmem);
  const cudaError_t err = cudaMemsetAsync(queue, 0, sizeof(unsigned long long), s);
  if (err != cudaSuccess) return (int)err;
  k_eos_guess<<<blocks, 128, sm, s>>>(h, mlp.small, mlp.w2bf, n, rho, e, abar, zbar, lT, stat);
  k_eos_invert<PHL_GUESS_MLP, true><<<blocks, 128, 0, s>>>(h, n, rho, e, abar, zbar, T, p, cs, iters, lT, stat, queue);
  // enough resident blocks to cover every SM several times; the loop covers any queue length
  const unsigned fb = (unsigned)std::min<long long>((long long)nsm * 8, (long long)blocks);
  k_eos_fallback<<<fb, 128, 0, s>>>(h, queue, rho, e, abar, zbar, T, p, cs, iters, stat);
  return (int)cudaGetLastError();
}

struct EosBatch {
  Mlp mlp;
  double *hbuf = nullptr;  // staging for the host-pointer variant
  int *ibuf = nullptr;
  unsigned long long *queue = nullptr;  // rejected learned guesses (count + entries)
  float *lT = nullptr;                  // the network's guesses
  int nsm = 0;
  DeviceMemory *mem = nullptr;

  void use(DeviceMemory *m) { mem = mlp.mem = m; }
  int sm_count() {
    if (!nsm) {
      int dev = 0;
      if (cudaGetDevice(&dev) != cudaSuccess ||
          cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        nsm = 148;
    }
    return nsm;
  }
  int energy(const HelmTable &h, cudaStream_t s, long long n, const double *rho, const double *T,
             const double *abar, const double *zbar, double *e) {
    if (n == 0) return 0;
    k_eos_energy<<<(unsigned)((n + ENERGY_THREADS - 1) / ENERGY_THREADS), ENERGY_THREADS, 0, s>>>(h, n, rho, T, abar, zbar, e);
    if (cudaGetLastError() != cudaSuccess) return -2;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -2;
    return 0;
  }
  int invert(const HelmTable &h, cudaStream_t s, long long n, const double *rho, const double *e,
             const double *abar, const double *zbar, double *T, double *p, double *cs, int *iters, int guess,
             unsigned long long *stat) {
    if (guess < 0 || guess > 2) return -1;
    if (guess == PHL_GUESS_MLP && !mlp.ready) return -4;
    if (n == 0) return 0;
    if (guess == PHL_GUESS_MLP && mlp.refresh(s)) return -2;
    if (guess == PHL_GUESS_MLP && !(mem->grow(&queue, (size_t)n + 1) && mem->grow(&lT, (size_t)n))) return -2;
    if (eos_launch(h, s, n, rho, e, abar, zbar, T, p, cs, iters, guess, mlp, stat, queue, lT, sm_count()))
      return -2;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -2;
    return 0;
  }
  int invert_host(const HelmTable &h, cudaStream_t s, long long n, const double *rho, const double *e,
                  const double *abar, const double *zbar, double *T, double *p, double *cs, int *iters, int guess,
                  unsigned long long *stat) {
    if (n == 0) return 0;
    if (!mem->grow(&hbuf, (size_t)n * 7) || (iters && !mem->grow(&ibuf, (size_t)n))) return -2;
    double *d_rho = hbuf, *d_e = hbuf + n, *d_a = hbuf + 2 * n, *d_z = hbuf + 3 * n, *d_T = hbuf + 4 * n;
    double *d_p = hbuf + 5 * n, *d_c = hbuf + 6 * n;
    size_t b = sizeof(double) * (size_t)n;
    if (cudaMemcpyAsync(d_rho, rho, b, cudaMemcpyHostToDevice, s) || cudaMemcpyAsync(d_e, e, b, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(d_a, abar, b, cudaMemcpyHostToDevice, s) || cudaMemcpyAsync(d_z, zbar, b, cudaMemcpyHostToDevice, s) ||
        cudaMemcpyAsync(d_T, T, b, cudaMemcpyHostToDevice, s))
      return -2;
    int rc = invert(h, s, n, d_rho, d_e, d_a, d_z, d_T, p ? d_p : nullptr, cs ? d_c : nullptr,
                    iters ? ibuf : nullptr, guess, stat);
    if (rc) return rc;
    if (cudaMemcpyAsync(T, d_T, b, cudaMemcpyDeviceToHost, s)) return -2;
    if (p && cudaMemcpyAsync(p, d_p, b, cudaMemcpyDeviceToHost, s)) return -2;
    if (cs && cudaMemcpyAsync(cs, d_c, b, cudaMemcpyDeviceToHost, s)) return -2;
    if (iters && cudaMemcpyAsync(iters, ibuf, sizeof(int) * (size_t)n, cudaMemcpyDeviceToHost, s)) return -2;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -2;
    return 0;
  }
  int mlp_train(const HelmTable &h, cudaStream_t s, long long n, unsigned long long seed, int epochs, int batch,
                double lr, double *final_loss) {
    return mlp.train(h, s, n, seed, epochs, batch, lr, final_loss);
  }
  int mlp_gradient(cudaStream_t s, long long n, const float *f, const float *t, float *g, double *loss) {
    return mlp.gradient_host(s, n, f, t, g, loss);
  }
  int mlp_get(cudaStream_t s, float *p) { return mlp.get(s, p); }
  int mlp_set(cudaStream_t s, const float *p) { return mlp.set(s, p); }
  int mlp_infer(cudaStream_t s, long long n, const float *f, float *o, unsigned long long *stalled) {
    return mlp.infer(s, n, f, o, stalled);
  }
};

}  // namespace phl
