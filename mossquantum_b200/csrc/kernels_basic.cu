// Plain per-gate sweeps, reductions, readout and parameter binding (sm_100a).
//
// These are the direct B200 equivalents of the reference's CPU kernels:
//   dense gate sweep       src/backends/cpu/gates/serial_short_range.jl:2-71,
//                          threaded_long_range.jl:3-132      -> k_dense<K>
//   diagonal / permutation src/backends/cpu/gates/specific/*.jl -> k_diag, k_monomial
//   expectation            src/backends/cpu/expectations/threaded*.jl -> k_cross_dense<K>
//   density expectation    src/backends/cpu/expectations/density_matrix_serial.jl -> k_dm_trace<K>
//   observable action      src/backends/cpu/operators/generic.jl:12-24 -> k_obs_apply<K>
//   probabilities          src/execution/probabilities.jl:42-105 -> k_marginal
// One thread owns one block of 2^K amplitudes that share all non-gate bits; consecutive
// threads own consecutive blocks, so the loads of a warp are coalesced double2 (16 B)
// accesses whenever the gate bits are not the lowest ones.
#include <algorithm>
#include <cstdarg>
#include <type_traits>

#include "family.cuh"
#include "kernels.h"

namespace mb {

namespace {

constexpr int kBlock = 256;

template <int D>
__device__ __forceinline__ void load_matrix(double2* sm, const double2* m, int mode) {
  for (int e = threadIdx.x; e < D * D; e += blockDim.x) sm[e] = mat_at(m, D, e % D, e / D, mode);
}

template <int K>
__device__ __forceinline__ void load_offsets(int64_t* soff, const Pos& pos) {
  constexpr int D = 1 << K;
  for (int a = threadIdx.x; a < D; a += blockDim.x) {
    int64_t o = 0;
#pragma unroll
    for (int j = 0; j < K; ++j)
      if ((a >> j) & 1) o |= int64_t(1) << pos.p[j];
    soff[a] = o;
  }
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_dense(double2* __restrict__ v, int64_t elems, Pos pos,
                                                   const double2* __restrict__ mats, int64_t mstride, int mode) {
  constexpr int D = 1 << K;
  __shared__ double2 sm[D * D];
  __shared__ int64_t soff[D];
  const int b = blockIdx.y;
  load_matrix<D>(sm, mats + b * mstride, mode);
  load_offsets<K>(soff, pos);
  __syncthreads();
  double2* vs = v + int64_t(b) * elems;
  const int64_t nblk = elems >> K;
  for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < nblk; j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = insert_zeros(j, K, pos.p);
    double2 in[D];
#pragma unroll
    for (int a = 0; a < D; ++a) in[a] = vs[base + soff[a]];
#pragma unroll
    for (int r = 0; r < D; ++r) {
      double2 acc = cmul(sm[r], in[0]);
#pragma unroll
      for (int c = 1; c < D; ++c) acc = cfma(sm[r + c * D], in[c], acc);
      vs[base + soff[r]] = acc;
    }
  }
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_diag(double2* __restrict__ v, int64_t elems, Pos pos,
                                                  const double2* __restrict__ mats, int64_t mstride, int mode,
                                                  uint32_t active) {
  constexpr int D = 1 << K;
  __shared__ double2 sd[D];
  __shared__ int64_t soff[D];
  const int b = blockIdx.y;
  for (int a = threadIdx.x; a < D; a += blockDim.x) sd[a] = mat_at(mats + b * mstride, D, a, a, mode);
  load_offsets<K>(soff, pos);
  __syncthreads();
  double2* vs = v + int64_t(b) * elems;
  const int64_t nblk = elems >> K;
  for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < nblk; j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = insert_zeros(j, K, pos.p);
#pragma unroll
    for (int a = 0; a < D; ++a)
      if ((active >> a) & 1) {
        double2 x = vs[base + soff[a]];
        vs[base + soff[a]] = cmul(sd[a], x);
      }
  }
}

struct Sigma {
  int n;          // active entries
  int from[32];   // local index read
  int to[32];     // local index written
};

template <int K>
__global__ void __launch_bounds__(kBlock) k_monomial(double2* __restrict__ v, int64_t elems, Pos pos,
                                                      const double2* __restrict__ mats, int64_t mstride,
                                                      int mode, Sigma sg) {
  constexpr int D = 1 << K;
  __shared__ double2 sph[D];
  __shared__ int64_t soff[D];
  const int b = blockIdx.y;
  for (int e = threadIdx.x; e < sg.n; e += blockDim.x)
    sph[e] = mat_at(mats + b * mstride, D, sg.to[e], sg.from[e], mode);
  load_offsets<K>(soff, pos);
  __syncthreads();
  double2* vs = v + int64_t(b) * elems;
  const int64_t nblk = elems >> K;
  for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < nblk; j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = insert_zeros(j, K, pos.p);
    double2 x[D];
#pragma unroll
    for (int e = 0; e < D; ++e)
      if (e < sg.n) x[e] = vs[base + soff[sg.from[e]]];
#pragma unroll
    for (int e = 0; e < D; ++e)
      if (e < sg.n) vs[base + soff[sg.to[e]]] = cmul(sph[e], x[e]);
  }
}

__global__ void k_set_basis(double2* v, int64_t elems, int64_t index) {
  const int b = blockIdx.y;
  double2* vs = v + int64_t(b) * elems;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < elems; i += int64_t(gridDim.x) * blockDim.x)
    vs[i] = make_double2(i == index ? 1.0 : 0.0, 0.0);
}

// rho[r + dim*c] = psi[r] conj(psi[c])
__global__ void k_to_density(const double2* __restrict__ psi, double2* __restrict__ rho, int n) {
  const int b = blockIdx.y;
  const int64_t dim = int64_t(1) << n, elems = dim * dim;
  const double2* p = psi + int64_t(b) * dim;
  double2* r = rho + int64_t(b) * elems;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < elems; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t row = i & (dim - 1), col = i >> n;
    r[i] = cmul(p[row], cconj(p[col]));
  }
}

// Weighted sum of B density matrices: one thread per element reads it in every sample, so the
// whole batch is read once at HBM rate (64 samples of 10 qubits: 1.07 GB). A gradient then reverses
// one matrix in place of B (64 samples of 10 qubits, 4 noisy layers: 49.9 -> 3.4 ms per call).
__global__ void __launch_bounds__(kBlock) k_weighted_density(const double2* __restrict__ in,
                                                              const double* __restrict__ w, int B, int64_t elems,
                                                              double2* __restrict__ out) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < elems; i += int64_t(gridDim.x) * blockDim.x) {
    double2 acc = cz();
    int b = 0;
    for (; b + 8 <= B; b += 8) {
      double2 x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) x[k] = in[int64_t(b + k) * elems + i];
#pragma unroll
      for (int k = 0; k < 8; ++k) acc = make_double2(fma(w[b + k], x[k].x, acc.x), fma(w[b + k], x[k].y, acc.y));
    }
    for (; b < B; ++b) {
      const double2 x = in[int64_t(b) * elems + i];
      acc = make_double2(fma(w[b], x.x, acc.x), fma(w[b], x.y, acc.y));
    }
    out[i] = acc;
  }
}

// sum_b w_b |psi_b><psi_b|
__global__ void __launch_bounds__(kBlock) k_weighted_outer(const double2* __restrict__ psi,
                                                            const double* __restrict__ w, int B, int n,
                                                            double2* __restrict__ out) {
  const int64_t dim = int64_t(1) << n, elems = dim * dim;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < elems; i += int64_t(gridDim.x) * blockDim.x) {
    const double2 *r = psi + (i & (dim - 1)), *c = psi + (i >> n);
    double2 acc = cz();
    for (int b = 0; b < B; ++b) acc = cfma_conj(cscale(c[int64_t(b) * dim], w[b]), r[int64_t(b) * dim], acc);
    out[i] = acc;
  }
}

__global__ void k_identity_density(double2* rho, int n) {
  const int b = blockIdx.y;
  const int64_t dim = int64_t(1) << n, elems = dim * dim;
  double2* r = rho + int64_t(b) * elems;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < elems; i += int64_t(gridDim.x) * blockDim.x)
    r[i] = make_double2((i & (dim - 1)) == (i >> n) ? 1.0 : 0.0, 0.0);
}

__global__ void k_scale(double2* v, int64_t count, double s) {
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += int64_t(gridDim.x) * blockDim.x)
    v[i] = cscale(v[i], s);
}

// ---- block reduction + last-block completion ---------------------------------------------
__device__ __forceinline__ double2 warp_sum(double2 x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x.x += __shfl_down_sync(0xffffffffu, x.x, o);
    x.y += __shfl_down_sync(0xffffffffu, x.y, o);
  }
  return x;
}

// Reduces `acc` over the block, stores the block partial, and lets the last block of the
// sample (then the last sample) finish the reduction in a fixed order.
__device__ void finish_reduction(double2 acc, double2* partials, unsigned* counters, const ReduceOut& ro) {
  __shared__ double2 warp_part[32];
  __shared__ bool last_block, last_sample;
  const int b = blockIdx.y, nb = gridDim.y, G = gridDim.x;
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) warp_part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double2 s = cz();
    for (int w = 0; w < int(blockDim.x >> 5); ++w) s = cadd(s, warp_part[w]);
    partials[int64_t(b) * G + blockIdx.x] = s;
    __threadfence();
    unsigned ticket = atomicAdd(&counters[b], 1u);
    last_block = ticket == unsigned(G - 1);
  }
  __syncthreads();
  if (!last_block) return;
  if (threadIdx.x == 0) {
    double2 s = cz();
    for (int g = 0; g < G; ++g) s = cadd(s, __ldcg(&partials[int64_t(b) * G + g]));
    counters[b] = 0;
    if (ro.out) ro.out[b] = ro.accumulate ? cadd(__ldcg(&ro.out[b]), s) : s;
    // Per-sample results also land in partials[nb * G + b] for the weighted total.
    partials[int64_t(nb) * G + b] = s;
    __threadfence();
    unsigned ticket = atomicAdd(&counters[nb], 1u);
    last_sample = ticket == unsigned(nb - 1);
    if (last_sample) {
      counters[nb] = 0;
      if (ro.grad) {
        double t = 0.0;
        for (int q = 0; q < nb; ++q) {
          double w = ro.weights ? ro.weights[q] : 1.0;
          t += w * __ldcg(&partials[int64_t(nb) * G + q]).x;
        }
        ro.grad[0] += t;
      }
    }
  }
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_cross_dense(const double2* __restrict__ c, const double2* __restrict__ v,
                                                         int64_t elems, Pos pos, const double2* __restrict__ mats,
                                                         int64_t mstride, int mode, double2* partials,
                                                         unsigned* counters, ReduceOut ro) {
  constexpr int D = 1 << K;
  __shared__ double2 sm[D * D];
  __shared__ int64_t soff[D];
  const int b = blockIdx.y;
  load_matrix<D>(sm, mats + b * mstride, mode);
  load_offsets<K>(soff, pos);
  __syncthreads();
  const double2* cs = c + int64_t(b) * elems;
  const double2* vs = v + int64_t(b) * elems;
  const int64_t nblk = elems >> K;
  double2 acc = cz();
  for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < nblk; j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = insert_zeros(j, K, pos.p);
    double2 in[D];
#pragma unroll
    for (int a = 0; a < D; ++a) in[a] = vs[base + soff[a]];
#pragma unroll
    for (int r = 0; r < D; ++r) {
      double2 mv = cmul(sm[r], in[0]);
#pragma unroll
      for (int q = 1; q < D; ++q) mv = cfma(sm[r + q * D], in[q], mv);
      acc = cfma_conj(cs[base + soff[r]], mv, acc);
    }
  }
  finish_reduction(acc, partials, counters, ro);
}

// Scalar (zero-qubit) cross product sum conj(c) v.
__global__ void __launch_bounds__(kBlock) k_cross_scalar(const double2* __restrict__ c, const double2* __restrict__ v,
                                                          int64_t elems, const double2* __restrict__ m,
                                                          double2* partials, unsigned* counters, ReduceOut ro) {
  const int b = blockIdx.y;
  const double2 scale = m[0];
  const double2* cs = c + int64_t(b) * elems;
  const double2* vs = v + int64_t(b) * elems;
  double2 acc = cz();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < elems; i += int64_t(gridDim.x) * blockDim.x)
    acc = cfma_conj(cs[i], vs[i], acc);
  acc = cmul(scale, acc);
  finish_reduction(acc, partials, counters, ro);
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_dm_trace(const double2* __restrict__ rho, int n, Pos pos,
                                                      const double2* __restrict__ m, double2* partials,
                                                      unsigned* counters, ReduceOut ro) {
  constexpr int D = 1 << K;
  __shared__ double2 sm[D * D];
  __shared__ int64_t soff[D];
  const int b = blockIdx.y;
  load_matrix<D>(sm, m, MAT_PLAIN);
  load_offsets<K>(soff, pos);
  __syncthreads();
  const int64_t dim = int64_t(1) << n;
  const double2* r = rho + int64_t(b) * dim * dim;
  const int64_t nblk = dim >> K;
  double2 acc = cz();
  for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < nblk; j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = insert_zeros(j, K, pos.p);
#pragma unroll
    for (int a = 0; a < D; ++a)
#pragma unroll
      for (int q = 0; q < D; ++q)  // M[a,q] * rho[base|q, base|a]
        acc = cfma(sm[a + q * D], r[(base + soff[q]) + dim * (base + soff[a])], acc);
  }
  finish_reduction(acc, partials, counters, ro);
}

// s * tr(rho) (the identity key of an observable on a density matrix).
__global__ void __launch_bounds__(kBlock) k_dm_trace0(const double2* __restrict__ rho, int n,
                                                       const double2* __restrict__ m, double2* partials,
                                                       unsigned* counters, ReduceOut ro) {
  const int b = blockIdx.y;
  const int64_t dim = int64_t(1) << n;
  const double2* r = rho + int64_t(b) * dim * dim;
  double2 acc = cz();
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < dim; i += int64_t(gridDim.x) * blockDim.x)
    acc = cadd(acc, r[i + dim * i]);
  acc = cmul(m[0], acc);
  finish_reduction(acc, partials, counters, ro);
}

template <int K>
__global__ void __launch_bounds__(kBlock) k_obs_apply(const double2* __restrict__ in, double2* __restrict__ out,
                                                       int64_t elems, Pos pos, const double2* __restrict__ m,
                                                       int first) {
  constexpr int D = 1 << K;
  __shared__ double2 sm[D * D];
  __shared__ int64_t soff[D];
  const int b = blockIdx.y;
  load_matrix<D>(sm, m, MAT_PLAIN);
  load_offsets<K>(soff, pos);
  __syncthreads();
  const double2* is = in + int64_t(b) * elems;
  double2* os = out + int64_t(b) * elems;
  const int64_t nblk = elems >> K;
  for (int64_t j = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; j < nblk; j += int64_t(gridDim.x) * blockDim.x) {
    const int64_t base = insert_zeros(j, K, pos.p);
    double2 x[D];
#pragma unroll
    for (int a = 0; a < D; ++a) x[a] = is[base + soff[a]];
#pragma unroll
    for (int r = 0; r < D; ++r) {
      double2 acc = first ? cz() : os[base + soff[r]];
#pragma unroll
      for (int q = 0; q < D; ++q) acc = cfma(sm[r + q * D], x[q], acc);
      os[base + soff[r]] = acc;
    }
  }
}

__global__ void k_obs_scalar(const double2* __restrict__ in, double2* __restrict__ out, int64_t count,
                             const double2* __restrict__ m, int first) {
  const double2 s = m[0];
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += int64_t(gridDim.x) * blockDim.x)
    out[i] = first ? cmul(s, in[i]) : cfma(s, in[i], out[i]);
}

// Marginal probabilities without atomics. The five lowest address bits are the lanes of a warp
// (32 consecutive amplitudes, 512 B); a work unit is one value of the readout bits above them
// and one of `splits` parts of the sum over the other high bits, which its warp runs through
// with a masked increment, each lane in a register. Only then are the lanes whose index differs
// in unread bits added (shuffles) and the bins written, each by one lane: no contention however
// few the bins, and the same sum on every run. With splits > 1 the units write partial
// histograms that k_marginal_sum adds in order.
// Bound: one read of the state (HBM, or L2 up to about 2^22 amplitudes). Ten of 22 qubits: 12.7 us
// and 6.6 us for the sum, against 70 us with a shared-memory histogram and double atomics.
struct Readout {
  int nq;
  int nh;                 // readout bits above the lanes
  int hpos[32], hbin[32]; // their address bits (ascending) and bins' bits
  int lbin[5];            // bin bit of lane bit l, or -1
  uint64_t inner;         // high address bits that are summed over
  int ninner;
};

__device__ __forceinline__ uint64_t deposit_mask(uint64_t x, uint64_t mask) {
  uint64_t r = 0;
  for (uint64_t m = mask; m && x; m &= m - 1, x >>= 1)
    if (x & 1) r |= m & (~m + 1);
  return r;
}

constexpr int kMarginalTerms = 16;   // loads in flight per lane
template <bool DM>
__global__ void __launch_bounds__(kBlock) k_marginal(const double2* __restrict__ v, int n, const Readout ro, int splits,
                                                      int nsamples, double* out, unsigned* flags, double tol) {
  const int lane = threadIdx.x & 31;
  const int64_t dim = int64_t(1) << n, elems = DM ? dim * dim : dim;
  const int64_t stride = DM ? dim + 1 : 1;
  const int64_t M = int64_t(1) << ro.nq, units = (int64_t(nsamples) * splits) << ro.nh;
  const int64_t nwarps = int64_t(gridDim.x) * (kBlock / 32);
  const int64_t per = (int64_t(1) << ro.ninner) / splits;   // both powers of two
  unsigned bad = 0;
  for (int64_t u = int64_t(blockIdx.x) * (kBlock / 32) + (threadIdx.x >> 5); u < units; u += nwarps) {
    const int64_t h = u & ((int64_t(1) << ro.nh) - 1);
    const int64_t rest = u >> ro.nh;
    const int s = int(rest % splits), b = int(rest / splits);
    uint64_t base = uint64_t(lane), bin = 0;
    for (int k = 0; k < ro.nh; ++k) {
      const uint64_t bit = (uint64_t(h) >> k) & 1;
      base |= bit << ro.hpos[k];
      bin |= bit << ro.hbin[k];
    }
    const double2* vs = v + int64_t(b) * elems;
    double p = 0.0;
    if (lane < dim) {
      uint64_t x = deposit_mask(uint64_t(s) * per, ro.inner);
      auto terms = [&](auto width) {   // so many loads in flight
        constexpr int W = decltype(width)::value;
        double2 a[W];
#pragma unroll
        for (int k = 0; k < W; ++k) {
          a[k] = vs[int64_t(base | x) * stride];
          x = ((x | ~ro.inner) + 1) & ro.inner;
        }
#pragma unroll
        for (int k = 0; k < W; ++k) {
          if (DM) {
            bad |= (fabs(a[k].y) > tol ? 1u : 0u) | (a[k].x < -tol ? 2u : 0u);
            p += a[k].x;
          } else {
            p += a[k].x * a[k].x + a[k].y * a[k].y;
          }
        }
      };
      int64_t i = 0;
      for (; i + kMarginalTerms <= per; i += kMarginalTerms) terms(std::integral_constant<int, kMarginalTerms>());
      for (; i < per; ++i) terms(std::integral_constant<int, 1>());
    }
    bool mine = lane < dim;
#pragma unroll
    for (int l = 0; l < 5; ++l) {
      const uint64_t bit = (lane >> l) & 1;
      if (ro.lbin[l] < 0) {
        p += __shfl_xor_sync(0xffffffffu, p, 1 << l);
        mine = mine && bit == 0;
      } else {
        bin |= bit << ro.lbin[l];
      }
    }
    if (mine) out[(int64_t(s) * nsamples + b) * M + int64_t(bin)] = p;
  }
  if (DM && bad) {
    if (bad & 1u) atomicOr(&flags[0], 1u);
    if (bad & 2u) atomicOr(&flags[1], 1u);
  }
}

// The whole register in its own order: a copy of squares (24 qubits: 78 us, 301 through the units above, whose
// warps then have one load each).
template <bool DM>
__global__ void __launch_bounds__(kBlock) k_probabilities(const double2* __restrict__ v, int n, int nsamples,
                                                          double* __restrict__ out, unsigned* flags, double tol) {
  const int64_t dim = int64_t(1) << n, total = int64_t(nsamples) << n;
  unsigned bad = 0;
  for (int64_t g = int64_t(blockIdx.x) * kBlock + threadIdx.x; g < total; g += int64_t(gridDim.x) * kBlock) {
    if (DM) {
      const double2 a = v[((g >> n) << (2 * n)) + (g & (dim - 1)) * (dim + 1)];
      bad |= (fabs(a.y) > tol ? 1u : 0u) | (a.x < -tol ? 2u : 0u);
      out[g] = a.x;
    } else {
      const double2 a = v[g];
      out[g] = a.x * a.x + a.y * a.y;
    }
  }
  if (DM && bad) {
    if (bad & 1u) atomicOr(&flags[0], 1u);
    if (bad & 2u) atomicOr(&flags[1], 1u);
  }
}

// Adds the parts of every bin in a fixed order: L threads (a warp, or a block where bins are few and
// parts many) stride over them, then a butterfly and the warps in order.
template <int L>
__global__ void __launch_bounds__(kBlock) k_marginal_sum(const double* __restrict__ part, int splits, int64_t count,
                                                          double* __restrict__ out) {
  __shared__ double warp_sum[kBlock / 32];
  const int sub = threadIdx.x & (L - 1);
  for (int64_t i = (int64_t(blockIdx.x) * kBlock + threadIdx.x) / L; i < count; i += int64_t(gridDim.x) * kBlock / L) {
    double p = 0.0;
#pragma unroll 8
    for (int s = sub; s < splits; s += L) p += part[int64_t(s) * count + i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
    if (L > 32) {
      if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = p;
      __syncthreads();
      if (sub == 0)
        for (int w = 1; w < L / 32; ++w) p += warp_sum[w];
      __syncthreads();
    }
    if (sub == 0) out[i] = p;
  }
}

// ---- parameter binding --------------------------------------------------------------------
// (family_matrix and bind_record: family.cuh, shared with the host-side lowering check)
__global__ void k_bind(const BindRec* __restrict__ recs, int nrecs, const double* __restrict__ theta, int nslots,
                       int rows, double2* table, int64_t stride) {
  const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= int64_t(nrecs) * rows) return;
  const int row = int(idx / nrecs), q = int(idx % nrecs);
  const BindRec rc = recs[q];
  const double t = rc.slot >= 0 ? theta[int64_t(row) * nslots + rc.slot] : rc.value;
  bind_record(rc, t, table, table + int64_t(row) * stride);
}

}  // namespace

// ---------------------------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------------------------
#define MB_DISPATCH_K(K, CALL) \
  switch (K) {                 \
    case 1: { constexpr int KK = 1; CALL; } break; \
    case 2: { constexpr int KK = 2; CALL; } break; \
    case 3: { constexpr int KK = 3; CALL; } break; \
    case 4: { constexpr int KK = 4; CALL; } break; \
    case 5: { constexpr int KK = 5; CALL; } break; \
    default: set_error("unsupported local operator size %d", K); return MB_EUNSUPPORTED; \
  }

static dim3 sample_grid(int64_t work, int nsamples) {
  int64_t per = (int64_t(148) * 8 + nsamples - 1) / nsamples;
  if (per < 1) per = 1;
  return dim3(grid_for(work, kBlock, per), nsamples);
}

int launch_dense(double2* v, int64_t elems, int nsamples, const Pos& pos, const double2* mats, int64_t mstride,
                 int mode, cudaStream_t st) {
  if (nsamples <= 0 || elems == 0) return MB_OK;
  dim3 g = sample_grid(elems >> pos.k, nsamples);
  {
    ProfScope ps("k_dense", 32.0 * elems * nsamples, st, 8.0 * (1 << pos.k) * elems * nsamples);
    MB_DISPATCH_K(pos.k, (k_dense<KK><<<g, kBlock, 0, st>>>(v, elems, pos, mats, mstride, mode)));
  }
  MB_LAUNCHED();
  return MB_OK;
}

int launch_diag(double2* v, int64_t elems, int nsamples, const Pos& pos, const double2* mats, int64_t mstride,
                int mode, uint32_t active, cudaStream_t st) {
  if (nsamples <= 0 || elems == 0 || active == 0) return MB_OK;
  dim3 g = sample_grid(elems >> pos.k, nsamples);
  {
    ProfScope ps("k_diag", 32.0 * elems * nsamples * __builtin_popcount(active) / (1 << pos.k), st);
    MB_DISPATCH_K(pos.k, (k_diag<KK><<<g, kBlock, 0, st>>>(v, elems, pos, mats, mstride, mode, active)));
  }
  MB_LAUNCHED();
  return MB_OK;
}

int launch_monomial(double2* v, int64_t elems, int nsamples, const Pos& pos, const double2* mats, int64_t mstride,
                    int mode, const int* sigma, int d, cudaStream_t st) {
  if (nsamples <= 0 || elems == 0) return MB_OK;
  Sigma sg{};
  // sigma[a] < 0 marks an entry the caller found unchanged (fixed point with phase 1).
  for (int a = 0; a < d; ++a)
    if (sigma[a] >= 0) { sg.from[sg.n] = a; sg.to[sg.n] = sigma[a]; ++sg.n; }
  if (sg.n == 0) return MB_OK;
  dim3 g = sample_grid(elems >> pos.k, nsamples);
  {
    ProfScope ps("k_monomial", 32.0 * elems * nsamples * sg.n / (1 << pos.k), st);
    MB_DISPATCH_K(pos.k, (k_monomial<KK><<<g, kBlock, 0, st>>>(v, elems, pos, mats, mstride, mode, sg)));
  }
  MB_LAUNCHED();
  return MB_OK;
}

int launch_set_basis(double2* v, int64_t elems, int nsamples, int64_t index, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  k_set_basis<<<sample_grid(elems, nsamples), kBlock, 0, st>>>(v, elems, index);
  MB_LAUNCHED();
  return MB_OK;
}

int launch_to_density(const double2* psi, double2* rho, int n, int nsamples, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  k_to_density<<<sample_grid(int64_t(1) << (2 * n), nsamples), kBlock, 0, st>>>(psi, rho, n);
  MB_LAUNCHED();
  return MB_OK;
}

int launch_weighted_density(const double2* in, bool pure, const double* w, int B, int n, double2* out, cudaStream_t st) {
  const int64_t elems = int64_t(1) << (2 * n);
  const int grid = grid_for(elems, kBlock, int64_t(148) * 32);
  {
    ProfScope ps("k_weighted_density", 16.0 * double(elems) * (pure ? 1 : B + 1), st);
    if (pure) k_weighted_outer<<<grid, kBlock, 0, st>>>(in, w, B, n, out);
    else k_weighted_density<<<grid, kBlock, 0, st>>>(in, w, B, elems, out);
  }
  MB_LAUNCHED();
  return MB_OK;
}

int launch_identity_density(double2* rho, int n, int nsamples, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  k_identity_density<<<sample_grid(int64_t(1) << (2 * n), nsamples), kBlock, 0, st>>>(rho, n);
  MB_LAUNCHED();
  return MB_OK;
}

int launch_scale(double2* v, int64_t count, double s, cudaStream_t st) {
  if (count <= 0) return MB_OK;
  k_scale<<<grid_for(count, kBlock), kBlock, 0, st>>>(v, count, s);
  MB_LAUNCHED();
  return MB_OK;
}

static int reduce_grid(int64_t work, int nsamples, const ReduceWs& ws, int slot, dim3* g) {
  int64_t cap_per = (ws.capacity / (nsamples + 1)) - 1;
  int64_t per = std::min<int64_t>((int64_t(148) * 4 + nsamples - 1) / nsamples, cap_per);
  if (per < 1 || nsamples + 1 > ws.ncounters) {
    set_error("reduction workspace too small for %d samples", nsamples);
    return MB_EUNSUPPORTED;
  }
  (void)slot;
  *g = dim3(grid_for(work, kBlock, per), nsamples);
  return MB_OK;
}

int launch_cross_dense(const double2* c, const double2* v, int64_t elems, int nsamples, const Pos& pos,
                       const double2* m, int64_t mstride, int mode, const ReduceWs& ws, int slot,
                       const ReduceOut& ro, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  dim3 g;
  int rc = reduce_grid(elems >> pos.k, nsamples, ws, slot, &g);
  if (rc) return rc;
  if (pos.k == 0) {
    k_cross_scalar<<<g, kBlock, 0, st>>>(c, v, elems, m, ws.partials, ws.counters, ro);
  } else {
    ProfScope ps("k_cross_dense", (c == v ? 16.0 : 32.0) * elems * nsamples, st);
    MB_DISPATCH_K(pos.k, (k_cross_dense<KK><<<g, kBlock, 0, st>>>(c, v, elems, pos, m, mstride, mode, ws.partials,
                                                                  ws.counters, ro)));
  }
  MB_LAUNCHED();
  return MB_OK;
}

int launch_dm_trace(const double2* rho, int n, int nsamples, const Pos& pos, const double2* m, const ReduceWs& ws,
                    int slot, const ReduceOut& ro, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  dim3 g;
  int rc = reduce_grid((int64_t(1) << n) >> pos.k, nsamples, ws, slot, &g);
  if (rc) return rc;
  MB_DISPATCH_K(pos.k, (k_dm_trace<KK><<<g, kBlock, 0, st>>>(rho, n, pos, m, ws.partials, ws.counters, ro)));
  MB_LAUNCHED();
  return MB_OK;
}

int launch_dm_trace0(const double2* rho, int n, int nsamples, const double2* m, const ReduceWs& ws,
                     const ReduceOut& ro, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  dim3 g;
  int rc = reduce_grid(int64_t(1) << n, nsamples, ws, 0, &g);
  if (rc) return rc;
  k_dm_trace0<<<g, kBlock, 0, st>>>(rho, n, m, ws.partials, ws.counters, ro);
  MB_LAUNCHED();
  return MB_OK;
}

int launch_obs_apply(const double2* in, double2* out, int64_t elems, int nsamples, const Pos& pos, const double2* m,
                     int first, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  if (pos.k == 0) {
    k_obs_scalar<<<grid_for(elems * nsamples, kBlock), kBlock, 0, st>>>(in, out, elems * nsamples, m, first);
  } else {
    dim3 g = sample_grid(elems >> pos.k, nsamples);
    MB_DISPATCH_K(pos.k, (k_obs_apply<KK><<<g, kBlock, 0, st>>>(in, out, elems, pos, m, first)));
  }
  MB_LAUNCHED();
  return MB_OK;
}

int launch_marginal(const double2* v, int n, int is_dm, int nsamples, const int* qubits, int nq, double* out,
                    unsigned* flags, double tol, double* scratch, int64_t scratch_cap, cudaStream_t st) {
  if (nsamples <= 0) return MB_OK;
  bool identity = nq == n;
  for (int j = 0; j < nq; ++j) identity = identity && qubits[j] == j;
  if (identity) {
    const int64_t total = int64_t(nsamples) << n;
    // A pure state is read whole and a density matrix only on its diagonal: 16 B per entry read.
    ProfScope ps("k_probabilities", 16.0 * double(total), st);
    if (is_dm) k_probabilities<true><<<grid_for(total, kBlock), kBlock, 0, st>>>(v, n, nsamples, out, flags, tol);
    else k_probabilities<false><<<grid_for(total, kBlock), kBlock, 0, st>>>(v, n, nsamples, out, flags, tol);
    MB_LAUNCHED();
    return MB_OK;
  }
  Readout ro{};
  ro.nq = nq;
  for (int l = 0; l < 5; ++l) ro.lbin[l] = -1;
  uint64_t read = 0;
  for (int j = 0; j < nq; ++j) read |= uint64_t(1) << qubits[j];
  for (int q = 0; q < n; ++q) {
    if (!((read >> q) & 1)) {
      if (q >= 5) ro.inner |= uint64_t(1) << q, ++ro.ninner;
      continue;
    }
    const int j = int(std::find(qubits, qubits + nq, q) - qubits);
    if (q < 5) ro.lbin[q] = j;
    else ro.hpos[ro.nh] = q, ro.hbin[ro.nh++] = j;
  }
  // Split the sums while the units leave warps idle (16 per SM are enough at 16 loads in flight; 64 with
  // 22 qubits, one read: 62 us a call against 50), a part keeps at least 4 terms per lane (16 qubits, one read:
  // 7.0 us of kernel, 8.1 with parts of 16), and the partial histograms fit the scratch.
  const int64_t count = (int64_t(1) << nq) * nsamples;
  int splits = 1;
  while ((int64_t(nsamples) * splits << ro.nh) < int64_t(148) * 16 && (int64_t(1) << ro.ninner) / splits >= 8 &&
         int64_t(splits) * 2 * count <= scratch_cap)
    splits *= 2;
  const int64_t units = (int64_t(nsamples) * splits) << ro.nh;
  const int grid = grid_for(units, kBlock / 32, int64_t(148) * 8);
  double* dst = splits > 1 ? scratch : out;
  {
    ProfScope ps("k_marginal", 16.0 * double(int64_t(1) << n) * nsamples, st);
    if (is_dm) k_marginal<true><<<grid, kBlock, 0, st>>>(v, n, ro, splits, nsamples, dst, flags, tol);
    else k_marginal<false><<<grid, kBlock, 0, st>>>(v, n, ro, splits, nsamples, dst, flags, tol);
  }
  MB_LAUNCHED();
  if (splits > 1) {
    const int64_t cap = int64_t(148) * 8;
    if (splits >= kBlock && count <= cap) k_marginal_sum<kBlock><<<grid_for(count, 1, cap), kBlock, 0, st>>>(scratch, splits, count, out);
    else k_marginal_sum<32><<<grid_for(count, kBlock / 32, cap), kBlock, 0, st>>>(scratch, splits, count, out);
    MB_LAUNCHED();
  }
  return MB_OK;
}

int launch_bind(const BindRec* recs, int nrecs, const double* theta, int nslots, int rows, double2* table,
                int64_t stride, cudaStream_t st) {
  if (nrecs <= 0 || rows <= 0) return MB_OK;
  int64_t work = int64_t(nrecs) * rows;
  k_bind<<<grid_for(work, 128, int64_t(1) << 30), 128, 0, st>>>(recs, nrecs, theta, nslots, rows, table, stride);
  MB_LAUNCHED();
  return MB_OK;
}

}  // namespace mb
