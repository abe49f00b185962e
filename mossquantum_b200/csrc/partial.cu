// Partial trace, inner products and fidelities on the device
// (src/observables/partial_trace.jl:11-97, src/states/state_vector.jl:93,
// src/states/density_matrix.jl:129-130, src/states/batch_*.jl fidelity).
//
// partial_tr keeps the remaining qubits in their original order as the low bits of the result
// and sums over the traced ones (_partial_tr_impl): for a density matrix
//   r[a, c] = sum_t rho[(a, t), (c, t)],
// for a pure state r = V V' with V[a, t] = psi[(a, t)], a blocked product split over t. Every sum
// has a fixed order, so the results are deterministic. Inner products and <y|rho|y>
// reduce per sample in two deterministic stages (per-block partials, then one block per sample).
#include <algorithm>
#include <cmath>
#include <vector>

#include "internal.h"

namespace mb {
namespace {

constexpr int kRThreads = 256;

struct Split {
  int m, k;
  int keep[32];    // remaining qubits, ascending
  int trace[32];   // traced qubits, ascending
};

__host__ __device__ __forceinline__ int64_t deposit(int64_t x, int nb, const int* bits) {
  int64_t r = 0;
  for (int j = 0; j < nb; ++j) r |= ((x >> j) & 1) << bits[j];
  return r;
}

// Density matrices: r[a, c] = sum_t rho[(a, t), (c, t)]. L threads of a block share one entry and
// stride over t (L = 1, 32 or 256, the fewest that give the GPU 2^18 threads; more threads per
// entry only shorten the serial sum). Bound by the 2^(2m + k) entries read.
template <int L>
__global__ void __launch_bounds__(256) k_partial_trace_dm(const double2* __restrict__ in, double2* __restrict__ out,
                                                          int n, const Split sp, int nsamples) {
  const int64_t dm_out = int64_t(1) << sp.m, total = int64_t(nsamples) << (2 * sp.m);
  const int64_t dim = int64_t(1) << n;
  const int nt = 1 << sp.k;
  __shared__ double2 part[8];
  const int sub = threadIdx.x & (L - 1);
  for (int64_t g = (int64_t(blockIdx.x) * 256 + threadIdx.x) / L; g < total; g += int64_t(gridDim.x) * 256 / L) {
    const double2* s = in + ((g >> (2 * sp.m)) << (2 * n)) +
                       (deposit(g & (dm_out - 1), sp.m, sp.keep) + deposit((g >> sp.m) & (dm_out - 1), sp.m, sp.keep) * dim);
    double re = 0.0, im = 0.0;
    for (int t = sub; t < nt; t += L) {
      const double2 x = s[deposit(t, sp.k, sp.trace) * (dim + 1)];
      re += x.x;
      im += x.y;
    }
    if (L > 1) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
      }
    }
    if (L > 32) {
      if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = make_double2(re, im);
      __syncthreads();
      if (sub == 0) {
        re = im = 0.0;
        for (int w = 0; w < L / 32; ++w) re += part[w].x, im += part[w].y;
      }
      __syncthreads();
    }
    if (sub == 0) out[g] = make_double2(re, im);
  }
}

// Pure states, few traced configurations and few products: one thread per entry of r. The staged product
// below takes 4 to 10 us more to start: 4 qubits, 2 kept 21 against 31 us a call, 8 qubits, 4 kept 26
// against 30, 12 qubits, 8 kept 28 against 34. Beyond 2^20 products (12 qubits, 10 kept: 44 against
// 30) or 2^4 terms per thread (2^5 from six kept qubits; 8 qubits, 2 kept, 2^6 terms: 42 against 32) it is faster.
constexpr int64_t kPTFewWork = int64_t(1) << 20;
__global__ void __launch_bounds__(256) k_partial_entries(const double2* __restrict__ in, double2* __restrict__ out, int n,
                                                         const Split sp, int nsamples) {
  const int64_t total = int64_t(nsamples) << (2 * sp.m), dm_out = int64_t(1) << sp.m;
  const int nt = 1 << sp.k;
  for (int64_t g = int64_t(blockIdx.x) * 256 + threadIdx.x; g < total; g += int64_t(gridDim.x) * 256) {
    const double2* s = in + ((g >> (2 * sp.m)) << n);
    const int64_t ra = deposit(g & (dm_out - 1), sp.m, sp.keep), rc = deposit((g >> sp.m) & (dm_out - 1), sp.m, sp.keep);
    double re = 0.0, im = 0.0;
#pragma unroll 4
    for (int t = 0; t < nt; ++t) {
      const int64_t rt = deposit(t, sp.k, sp.trace);
      const double2 u = s[ra | rt], v = s[rc | rt];   // u * conj(v)
      re += u.x * v.x + u.y * v.y;
      im += u.y * v.x - u.x * v.y;
    }
    out[g] = make_double2(re, im);
  }
}

// Pure states: r = V V', V[a, t] = psi[(a, t)], as a blocked product. A CTA owns one pair of
// 2^ma-row blocks (ma = min(m, 6)) of r and one chunk of t; per step it stages both blocks' tiles of
// 2^tb columns (2^(ma + tb) <= 2^11 amplitudes) with cp.async, double-buffered, the copy running
// in ascending address order whichever bits are kept so that it stays coalesced, and its threads
// accumulate BS x BS micro-tiles (rows a, a + nb, ...: consecutive threads read consecutive
// shared words). r is Hermitian: only block pairs ia <= ic and, on the diagonal pair, only
// micro-tiles i <= j are formed; spare threads take further columns (`groups`). Chunks of t keep
// every SM busy (one CTA each: a thread's 16 complex accumulators are 32 independent FP64 chains of two
// multiply-adds per column, enough for three warps per scheduler, and a second CTA would make them
// spill); k_partial_sum adds the chunks in order and writes both halves of r.
// 22 qubits, 6 kept: 85 us and 6 us for the sum, against 34.5 ms with one thread per entry of r
// looping over t; the floor is 31 us of FP64 (2^28 complex multiply-adds, half of them by symmetry).
constexpr int kPTBits = 11;        // log2 of a staged tile's amplitudes
// Threads: 256 micro-tiles of a block pair, or three times 136 of the one block there is up to six
// kept qubits (twice 136 leave nine warps on four schedulers: 93 us, thirteen 85; at 22 qubits, 6 kept). Pairs have the
// registers to run two columns at once (22 qubits, 8 kept: the call 558 -> 520 us); with 416 threads
// two measured the same as one.
constexpr int kPTThreads = 288, kPTThreadsOne = 416;

struct TraceArgs {
  int n, m, k, ma, tb;             // qubits, kept, traced; row and column bits of a tile
  int keep[32], trace[32];
  int nblocks;                     // 2^(m - ma) row blocks
  int chunks;                      // parts of the t range
  int npairs;
  int64_t entries;                 // partial entries per (sample, pair, chunk)
};

__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}

// Row-block pair q in the order (0,0), (0,1), (1,1), (0,2), ...: ia <= ic.
__device__ __forceinline__ void pair_of(int q, int* ia, int* ic) {
  int c = int((sqrtf(8.0f * q + 1.0f) - 1.0f) * 0.5f);
  while (c * (c + 1) / 2 > q) --c;
  while ((c + 1) * (c + 2) / 2 <= q) ++c;
  *ic = c;
  *ia = q - c * (c + 1) / 2;
}

// Entry (r, c) of micro-tile (i, j) of block pair (ia, ic), and its mirror image.
__device__ __forceinline__ void put_entry(double2* out, const TraceArgs& a, int ia, int ic, int i, int j, int nb, int r,
                                          int c, double2 v) {
  const int64_t row = (int64_t(ia) << a.ma) + i + r * nb, col = (int64_t(ic) << a.ma) + j + c * nb;
  if (row == col) v.y = 0.0;                        // a sum of |psi|^2
  out[row + (col << a.m)] = v;
  if (ia != ic || i != j) out[col + (row << a.m)] = cconj(v);
}

template <int BS, int NT>
__global__ void __launch_bounds__(NT, 1) k_partial_outer(const double2* __restrict__ in, const TraceArgs a,
                                                                double2* __restrict__ part,
                                                                double2* __restrict__ out) {
  extern __shared__ double2 sm[];
  const int A = 1 << a.ma, T = 1 << a.tb, E = A * T;
  const int q = blockIdx.x, ch = blockIdx.y, b = blockIdx.z;
  int ia, ic;
  pair_of(q, &ia, &ic);
  const bool diag = ia == ic;
  const int nbuf = diag ? 1 : 2;                    // row blocks staged per step
  double2* buf = sm;                                // [2 steps][nbuf][T][A]
  uint32_t* goff = reinterpret_cast<uint32_t*>(sm + size_t(a.nblocks > 1 ? 4 : 2) * E);
  uint16_t* slot = reinterpret_cast<uint16_t*>(goff + E);
  // Staging map: element e's bits, in ascending address order, are the tile's ma kept and tb
  // traced bits (the lowest of each kind).
  for (int e = threadIdx.x; e < E; e += NT) {
    uint64_t off = 0;
    int row = 0, col = 0;
    for (int x = 0, y = 0, j = 0; x < a.ma || y < a.tb; ++j) {
      const bool kept = y >= a.tb || (x < a.ma && a.keep[x] < a.trace[y]);
      const uint64_t bit = (e >> j) & 1;
      if (kept) off |= bit << a.keep[x], row |= int(bit) << x, ++x;
      else off |= bit << a.trace[y], col |= int(bit) << y, ++y;
    }
    goff[e] = uint32_t(off);
    slot[e] = uint16_t(col * A + row);
  }
  const double2* src = in + (int64_t(b) << a.n);
  int64_t hi_a = 0, hi_c = 0;                       // the row blocks' fixed kept bits
  for (int j = a.ma; j < a.m; ++j) {
    hi_a |= int64_t((ia >> (j - a.ma)) & 1) << a.keep[j];
    hi_c |= int64_t((ic >> (j - a.ma)) & 1) << a.keep[j];
  }
  const int64_t all = int64_t(1) << (a.k - a.tb), s0 = all * ch / a.chunks, steps = all * (ch + 1) / a.chunks - s0;
  auto base_t = [&](int64_t s) {
    int64_t r = 0;
    for (int j = a.tb; j < a.k; ++j) r |= ((s >> (j - a.tb)) & 1) << a.trace[j];
    return r;
  };
  auto stage = [&](int64_t s, int which) {
    const int64_t t = base_t(s);
    double2* d = buf + size_t(which) * nbuf * E;
    for (int e = threadIdx.x; e < E; e += NT) {
      cp16(d + slot[e], src + (hi_a | t | goff[e]));
      if (!diag) cp16(d + E + slot[e], src + (hi_c | t | goff[e]));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int nb = A / BS;                            // micro-tile rows
  const int P = diag ? nb * (nb + 1) / 2 : nb * nb; // micro-tiles
  const int groups = NT / P;
  const int g = threadIdx.x / P, p = threadIdx.x - g * P;
  const bool on = g < groups;
  int i = 0, j = 0;
  if (diag) {
    pair_of(p, &i, &j);
  } else {
    i = p / nb;
    j = p - i * nb;
  }
  double2 acc[BS][BS];
#pragma unroll
  for (int r = 0; r < BS; ++r)
#pragma unroll
    for (int s = 0; s < BS; ++s) acc[r][s] = make_double2(0.0, 0.0);
  __syncthreads();
  stage(s0, 0);
  for (int64_t s = 0; s < steps; ++s) {
    if (s + 1 < steps) {
      stage(s0 + s + 1, int((s + 1) & 1));
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const double2* ra = buf + size_t(s & 1) * nbuf * E;
    const double2* rc = diag ? ra : ra + E;
    if (on) {
#pragma unroll NT == kPTThreads ? 2 : 1
      for (int t = g; t < T; t += groups) {
        double2 x[BS];
#pragma unroll
        for (int r = 0; r < BS; ++r) x[r] = ra[t * A + i + r * nb];
#pragma unroll
        for (int c = 0; c < BS; ++c) {
          const double2 y = rc[t * A + j + c * nb];
#pragma unroll
          for (int r = 0; r < BS; ++r) acc[r][c] = cfma_conj(y, x[r], acc[r][c]);
        }
      }
    }
    __syncthreads();
  }
  // Column groups add up in shared memory (halving), four entries at a time; with one chunk the
  // entries go straight to r, else to the CTA's partial tile of P * BS * BS.
  double2* red = sm;
  double2* dst = part + ((int64_t(b) * a.npairs + q) * a.chunks + ch) * a.entries;
#pragma unroll
  for (int r = 0; r < BS; ++r) {
    if (groups > 1) {
#pragma unroll
      for (int c = 0; c < BS; ++c)
        if (on) red[c * NT + threadIdx.x] = acc[r][c];
      __syncthreads();
      for (int n = groups; n > 1;) {
        const int half = (n + 1) / 2;
        if (g < n - half)
#pragma unroll
          for (int c = 0; c < BS; ++c) {
            double2* x = red + c * NT + threadIdx.x;
            *x = cadd(*x, x[half * P]);
          }
        __syncthreads();
        n = half;
      }
      if (g == 0)
#pragma unroll
        for (int c = 0; c < BS; ++c) acc[r][c] = red[c * NT + threadIdx.x];
      __syncthreads();
    }
    if (on && g == 0)
#pragma unroll
      for (int c = 0; c < BS; ++c) {
        if (a.chunks > 1) dst[int64_t(r * BS + c) * P + p] = acc[r][c];
        else put_entry(out + (int64_t(b) << (2 * a.m)), a, ia, ic, i, j, nb, r, c, acc[r][c]);
      }
  }
}

// Adds the chunks of every partial entry in order and writes the entry and its mirror image. Lanes of a
// warp share an entry when there are many chunks.
template <int BS, int L>
__global__ void __launch_bounds__(256) k_partial_sum(const double2* __restrict__ part, const TraceArgs a,
                                                     double2* __restrict__ out, int nsamples) {
  const int64_t total = int64_t(nsamples) * a.npairs * a.entries;
  const int nb = (1 << a.ma) / BS;
  const int sub = threadIdx.x & (L - 1);
  for (int64_t w = (int64_t(blockIdx.x) * 256 + threadIdx.x) / L; w < total; w += int64_t(gridDim.x) * 256 / L) {
    const int64_t bq = w / a.entries, e = w - bq * a.entries;
    const int q = int(bq % a.npairs), b = int(bq / a.npairs);
    int ia, ic, i, j;
    pair_of(q, &ia, &ic);
    const int P = ia == ic ? nb * (nb + 1) / 2 : nb * nb;
    const int p = int(e % P), x = int(e / P);
    if (x >= BS * BS) continue;                     // a diagonal pair has fewer entries (whole warps agree)
    double2 v = make_double2(0.0, 0.0);
    for (int c = sub; c < a.chunks; c += L) v = cadd(v, part[(bq * a.chunks + c) * a.entries + e]);
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if (sub) continue;
    if (ia == ic) {
      pair_of(p, &i, &j);
    } else {
      i = p / nb;
      j = p - i * nb;
    }
    put_entry(out + (int64_t(b) << (2 * a.m)), a, ia, ic, i, j, nb, x / BS, x % BS, v);
  }
}

// Stage 1 of <x|y> (conj on x) or <y|rho|y>: block g of sample b sums a strided range.
__global__ void __launch_bounds__(kRThreads) k_pair_partials(const double2* __restrict__ x, const double2* __restrict__ y,
                                                             int n, int sandwich, int G, double2* __restrict__ part) {
  const int b = blockIdx.y;
  const int64_t dim = int64_t(1) << n;
  const int64_t count = sandwich ? dim * dim : dim;
  const double2* xs = x + int64_t(b) * count;
  const double2* ys = y + int64_t(b) * dim;
  double re = 0.0, im = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * kRThreads + threadIdx.x; i < count; i += int64_t(G) * kRThreads) {
    if (sandwich) {
      // rho[r, c] at r + c*dim contributes conj(y_r) rho[r, c] y_c
      const int64_t r = i & (dim - 1), c = i >> n;
      const double2 rho = xs[i], yr = ys[r], yc = ys[c];
      const double2 t = make_double2(rho.x * yc.x - rho.y * yc.y, rho.x * yc.y + rho.y * yc.x);
      re += yr.x * t.x + yr.y * t.y;
      im += yr.x * t.y - yr.y * t.x;
    } else {
      const double2 u = xs[i], v = ys[i];
      re += u.x * v.x + u.y * v.y;
      im += u.x * v.y - u.y * v.x;
    }
  }
  __shared__ double sre[kRThreads], sim[kRThreads];
  sre[threadIdx.x] = re;
  sim[threadIdx.x] = im;
  __syncthreads();
  for (int w = kRThreads / 2; w > 0; w >>= 1) {
    if (int(threadIdx.x) < w) {
      sre[threadIdx.x] += sre[threadIdx.x + w];
      sim[threadIdx.x] += sim[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) part[int64_t(b) * G + blockIdx.x] = make_double2(sre[0], sim[0]);
}

__global__ void k_pair_finish(const double2* __restrict__ part, int G, double2* __restrict__ out) {
  if (threadIdx.x != 0) return;
  double re = 0.0, im = 0.0;
  for (int g = 0; g < G; ++g) {
    re += part[int64_t(blockIdx.x) * G + g].x;
    im += part[int64_t(blockIdx.x) * G + g].y;
  }
  out[blockIdx.x] = make_double2(re, im);
}

bool is_dm_kind(int kind) { return kind == MB_DENSITY || kind == MB_BATCH_DENSITY; }

int trace_density(mb_state in, const Split& sp, mb_state out) {
  const int64_t work = (int64_t(1) << (2 * sp.m)) * in->batch, nt = int64_t(1) << sp.k;
  const int64_t want = int64_t(1) << 18, cap = int64_t(g_ctx.sm_count) * 32;
  if (work >= want || nt < 32)
    k_partial_trace_dm<1><<<grid_for(work, 256, cap), 256, 0, g_ctx.stream>>>(in->d, out->d, in->n, sp, in->batch);
  else if (work * 32 >= want || nt < 256)
    k_partial_trace_dm<32><<<grid_for(work * 32, 256, cap), 256, 0, g_ctx.stream>>>(in->d, out->d, in->n, sp, in->batch);
  else
    k_partial_trace_dm<256><<<grid_for(work * 256, 256, cap), 256, 0, g_ctx.stream>>>(in->d, out->d, in->n, sp, in->batch);
  MB_LAUNCHED();
  return MB_OK;
}

template <int BS>
int trace_pure_bs(mb_state in, TraceArgs a, mb_state out) {
  const int B = in->batch, A = 1 << a.ma, nb = A / BS;
  a.nblocks = 1 << (a.m - a.ma);
  a.npairs = a.nblocks * (a.nblocks + 1) / 2;
  const int P = a.nblocks > 1 ? nb * nb : nb * (nb + 1) / 2;
  a.entries = int64_t(P) * BS * BS;
  const int64_t steps = int64_t(1) << (a.k - a.tb);
  // Chunks of t until every SM has a CTA, while a chunk keeps at least four steps (a step is
  // one staged tile; shorter chunks spend their time on the pipeline's start and on partial tiles).
  a.chunks = int(std::max<int64_t>(1, std::min<int64_t>(steps / 4, g_ctx.sm_count / (int64_t(a.npairs) * B))));
  const size_t E = size_t(1) << (a.ma + a.tb);
  const int nt = a.nblocks > 1 ? kPTThreads : kPTThreadsOne;
  auto* outer = a.nblocks > 1 ? k_partial_outer<BS, kPTThreads> : k_partial_outer<BS, kPTThreadsOne>;
  const size_t shm = std::max(E * ((a.nblocks > 1 ? 4 : 2) * sizeof(double2) + sizeof(uint32_t) + sizeof(uint16_t)),
                              sizeof(double2) * size_t(BS * nt));
  const int64_t per = int64_t(a.npairs) * a.chunks * a.entries;
  double2* part = nullptr;
  if (a.chunks > 1 && dev_alloc((void**)&part, sizeof(double2) * size_t(per) * B)) a.chunks = 1;  // no room: unsplit
  cudaFuncSetAttribute(outer, cudaFuncAttributeMaxDynamicSharedMemorySize, int(shm));
  int rc = MB_OK;
  for (int b0 = 0; b0 < B && !rc; b0 += 65535) {    // grid.z limit
    const int nbat = std::min(65535, B - b0);
    const double2* src = in->d + (int64_t(b0) << a.n);
    double2* dst = out->d + (int64_t(b0) << (2 * a.m));
    double2* pt = part ? part + per * b0 : nullptr;
    ProfScope ps("k_partial_outer", 16.0 * double(int64_t(1) << a.n) * nbat, g_ctx.stream);
    outer<<<dim3(a.npairs, a.chunks, nbat), nt, shm, g_ctx.stream>>>(src, a, pt, dst);
    ++launch_counter();
    if (a.chunks > 1) {
      const int64_t work = int64_t(nbat) * a.npairs * a.entries, cap = int64_t(g_ctx.sm_count) * 32;
      if (a.chunks >= 32)
        k_partial_sum<BS, 32><<<grid_for(work * 32, 256, cap), 256, 0, g_ctx.stream>>>(pt, a, dst, nbat);
      else
        k_partial_sum<BS, 1><<<grid_for(work, 256, cap), 256, 0, g_ctx.stream>>>(pt, a, dst, nbat);
      ++launch_counter();
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      set_error("partial trace: %s", cudaGetErrorString(e));
      rc = MB_EDEVICE;
    }
  }
  dev_free(part);
  return rc;
}

int trace_pure(mb_state in, const Split& sp, mb_state out) {
  const int64_t entries = int64_t(in->batch) << (2 * sp.m);
  if (sp.k <= (sp.m >= 6 ? 5 : 4) && entries <= (kPTFewWork >> sp.k)) {
    ProfScope ps("k_partial_entries", 16.0 * double(in->elems) * in->batch, g_ctx.stream);
    k_partial_entries<<<grid_for(entries, 256), 256, 0, g_ctx.stream>>>(in->d, out->d, in->n, sp, in->batch);
    MB_LAUNCHED();
    return MB_OK;
  }
  TraceArgs a{};
  a.n = in->n;
  a.m = sp.m;
  a.k = sp.k;
  std::copy(sp.keep, sp.keep + sp.m, a.keep);
  std::copy(sp.trace, sp.trace + sp.k, a.trace);
  a.ma = std::min(sp.m, 6);
  a.tb = std::min(sp.k, kPTBits - a.ma);
  // 2x2 micro-tiles below two kept qubits, else 4x4 (16 products per 8 shared-memory reads)
  return sp.m < 2 ? trace_pure_bs<2>(in, a, out) : trace_pure_bs<4>(in, a, out);
}

int pair_reduce(const double2* x, const double2* y, int n, int sandwich, int B, double* host_out) {
  const int64_t dim = int64_t(1) << n;
  const int64_t count = sandwich ? dim * dim : dim;
  const int G = int(std::max<int64_t>(1, std::min<int64_t>((count + kRThreads - 1) / kRThreads,
                                                          std::max<int64_t>(1, int64_t(g_ctx.sm_count) * 8 / B))));
  double2* part = nullptr;
  double2* res = nullptr;
  int rc = dev_alloc((void**)&part, sizeof(double2) * size_t(G) * B);
  if (!rc) rc = dev_alloc((void**)&res, sizeof(double2) * B);
  cudaStream_t st = g_ctx.stream;
  if (!rc) {
    k_pair_partials<<<dim3(G, B), kRThreads, 0, st>>>(x, y, n, sandwich, G, part);
    k_pair_finish<<<B, 32, 0, st>>>(part, G, res);
    launch_counter() += 2;
    cudaMemcpyAsync(host_out, res, sizeof(double2) * B, cudaMemcpyDeviceToHost, st);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
      set_error("reduction failed");
      rc = MB_EDEVICE;
    }
  }
  dev_free(part);
  dev_free(res);
  return rc;
}

}  // namespace
}  // namespace mb

using namespace mb;

extern "C" int mb_partial_trace(mb_state in, const int* sites, int k, mb_state out) {
  std::lock_guard<std::recursive_mutex> lk(g_mu);
  if (int rc = check_init()) return rc;
  if (int rc = check_not_capturing("mb_partial_trace")) return rc;
  if (!in || !out || in == out || k < 1 || (k && !sites)) return MB_EINVAL;
  const int n = in->n;
  if (k >= n) {
    set_error("trace out between 1 and n-1 qubits (the full trace is a scalar)");
    return MB_EINVAL;
  }
  Split sp{};
  sp.m = n - k;
  sp.k = k;
  bool traced[64] = {false};
  for (int j = 0; j < k; ++j) {
    if (sites[j] < 0 || sites[j] >= n) {
      set_error("site out of range.");
      return MB_EINVAL;
    }
    if (traced[sites[j]]) {
      set_error("duplicate sites not allowed.");
      return MB_EINVAL;
    }
    traced[sites[j]] = true;
  }
  for (int q = 0, a = 0, t = 0; q < n; ++q) {
    if (traced[q]) sp.trace[t++] = q;
    else sp.keep[a++] = q;
  }
  const bool batch_in = in->kind == MB_BATCH_PURE || in->kind == MB_BATCH_DENSITY;
  const int want_kind = batch_in ? MB_BATCH_DENSITY : MB_DENSITY;
  if (out->kind != want_kind || out->n != sp.m || out->batch != in->batch) {
    set_error("partial trace output must be a %s of %d qubits and the input's batch size",
              batch_in ? "BatchDensityMatrix" : "DensityMatrix", sp.m);
    return MB_EINVAL;
  }
  if (in->batch == 0) return MB_OK;
  const int rc = is_dm_kind(in->kind) ? trace_density(in, sp, out) : trace_pure(in, sp, out);
  if (rc) return rc;
  MB_CHECK_CUDA(cudaStreamSynchronize(g_ctx.stream));
  return MB_OK;
}

extern "C" int mb_inner(mb_state x, mb_state y, double* out) {
  std::lock_guard<std::recursive_mutex> lk(g_mu);
  if (int rc = check_init()) return rc;
  if (int rc = check_not_capturing("mb_inner")) return rc;
  if (!x || !y || !out) return MB_EINVAL;
  if (is_dm_kind(x->kind) || is_dm_kind(y->kind) || x->n != y->n || x->batch != y->batch) {
    set_error("inner products need two pure states of the same size and batch");
    return MB_EINVAL;
  }
  if (x->batch == 0) return MB_OK;
  return pair_reduce(x->d, y->d, x->n, 0, x->batch, out);
}

extern "C" int mb_sandwich(mb_state rho, mb_state y, double* out) {
  std::lock_guard<std::recursive_mutex> lk(g_mu);
  if (int rc = check_init()) return rc;
  if (int rc = check_not_capturing("mb_sandwich")) return rc;
  if (!rho || !y || !out) return MB_EINVAL;
  if (!is_dm_kind(rho->kind) || is_dm_kind(y->kind) || rho->n != y->n || rho->batch != y->batch) {
    set_error("<y|rho|y> needs a density matrix and a pure state of the same size and batch");
    return MB_EINVAL;
  }
  if (rho->batch == 0) return MB_OK;
  return pair_reduce(rho->d, y->d, rho->n, 1, rho->batch, out);
}

extern "C" int mb_state_extract(mb_state src, int index, mb_state dst) {
  std::lock_guard<std::recursive_mutex> lk(g_mu);
  if (int rc = check_init()) return rc;
  if (!src || !dst || index < 0 || index >= src->batch) return MB_EINVAL;
  const bool ok = ((src->kind == MB_BATCH_PURE && dst->kind == MB_PURE) ||
                   (src->kind == MB_BATCH_DENSITY && dst->kind == MB_DENSITY)) && dst->n == src->n;
  if (!ok) {
    set_error("extract needs a batch source and a single state of the same kind and size");
    return MB_EINVAL;
  }
  MB_CHECK_CUDA(cudaMemcpyAsync(dst->d, src->d + int64_t(index) * src->elems, sizeof(double2) * src->elems,
                                cudaMemcpyDeviceToDevice, g_ctx.stream));
  MB_CHECK_CUDA(cudaStreamSynchronize(g_ctx.stream));
  return MB_OK;
}

extern "C" int mb_state_broadcast(mb_state src, mb_state dst) {
  std::lock_guard<std::recursive_mutex> lk(g_mu);
  if (int rc = check_init()) return rc;
  if (!src || !dst) return MB_EINVAL;
  const bool ok = ((src->kind == MB_PURE && dst->kind == MB_BATCH_PURE) ||
                   (src->kind == MB_DENSITY && dst->kind == MB_BATCH_DENSITY)) && dst->n == src->n;
  if (!ok) {
    set_error("broadcast needs a single source and a batch destination of the same kind and size");
    return MB_EINVAL;
  }
  for (int b = 0; b < dst->batch; ++b)
    MB_CHECK_CUDA(cudaMemcpyAsync(dst->d + int64_t(b) * dst->elems, src->d, sizeof(double2) * src->elems,
                                  cudaMemcpyDeviceToDevice, g_ctx.stream));
  MB_CHECK_CUDA(cudaStreamSynchronize(g_ctx.stream));
  return MB_OK;
}

extern "C" int mb_state_tile(mb_state src, int copies, mb_state dst) {
  std::lock_guard<std::recursive_mutex> lk(g_mu);
  if (int rc = check_init()) return rc;
  if (!src || !dst || copies < 0) return MB_EINVAL;
  if (src->kind != dst->kind || src->kind < MB_BATCH_PURE || dst->n != src->n ||
      int64_t(dst->batch) != int64_t(src->batch) * copies) {
    set_error("tile needs batch states of one kind and size, the destination holding `copies` copies of the source");
    return MB_EINVAL;
  }
  const size_t bytes = sizeof(double2) * size_t(src->elems) * src->batch;
  for (int c = 0; c < copies; ++c)
    MB_CHECK_CUDA(cudaMemcpyAsync(reinterpret_cast<char*>(dst->d) + bytes * c, src->d, bytes, cudaMemcpyDeviceToDevice,
                                  g_ctx.stream));
  MB_CHECK_CUDA(cudaStreamSynchronize(g_ctx.stream));
  return MB_OK;
}
