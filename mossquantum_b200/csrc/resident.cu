// K8: whole objectives of small pure states in one launch.
//
// A state of up to 12 qubits (and, for gradients, its adjoint beside it) fits the shared memory of one
// SM, so a circuit, <H> and the reverse sweep need no pass over HBM and no launch per gate: one CTA
// per sample binds the angles, runs the gates, forms H psi and runs the reverse
// (src/differentiation/circuit.jl:77-229, objectives.jl:183-296). At these sizes the sweep is bound
// by latency: a barrier and a shared-memory round trip per step, so steps are what the layout saves.
//  - Linear frame. CNOT, SWAP and X permute basis states linearly over GF(2), so they move no
//    amplitudes: the host keeps, per qubit t, the parity mask row[t] (and a constant) that gives bit
//    t's value from a storage index, and the flip mask col[t] that toggles bit t alone. A gate on t
//    pairs storage indexes p and p ^ col[t]; controls and Pauli strings are parities.
//  - Runs. Consecutive gates on one qubit form a group, multiplied into one 2x2 when the angles are
//    bound.
//  - Stages. Groups whose targets share a frame run together, R qubits at a time: a thread holds the
//    2^R amplitudes (of both states) that the targets span, so R groups cost one barrier and one
//    round trip. The hardware-efficient ansatz takes n / R stages per layer.
//  - Gradients. All gradients of a group follow from four cross sums of its pairs (k_resident's
//    reverse); a step only stores each thread's part, and the parts are added a chunk at a time.
// Sums have a fixed order: the same bits on every run.
// Measured (8 qubits, 2 layers of the ansatz): value 10 us and gradient 17 us of SM time (47 and 60 us
// per call; the plain reverse took 266 launches and 2.0 ms); 48 samples of 12 qubits, 4 layers:
// 150 us (732 launches and 5.3 ms per call before). One qubit per stage took 226 us for the last: the
// stages are bound by barriers and shared-memory round trips, and three qubits' tuples of both
// states are what a thread's registers hold. Above 12 qubits the passes over HBM are the only form:
// two states no longer fit one SM.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "fusemat.cuh"
#include "internal.h"

namespace mb {
namespace {

constexpr int kResMaxBits = 12;    // 2 x 64 KiB of amplitudes
constexpr int kResMaxThreads = 512;
constexpr size_t kResMaxShared = 224 * 1024;

enum RType : uint16_t {
  RO_RX, RO_RY, RO_RZ, RO_PHASE,   // rotation families: (cos, sin) at cs[data]
  RO_U1,                           // fixed 2x2 (column-major at table[data], stride of the entries in e)
  RO_X,                            // exchange (controlled; the uncontrolled one is frame)
  RO_NEG,                          // sign flip of the target's 1 amplitude (CZ, Z)
};

// One gate of a pair group; read when the groups are bound and when gradients are formed.
struct __align__(8) ROp {
  uint16_t type, neg;   // neg: adjoint family gate (angle and generator negated)
  int16_t slot;         // parameter slot of a gradient, or -1
  uint16_t group;
  int32_t data;
  int32_t e[4];         // RO_U1: table offsets of m00, m10, m01, m11
};

enum RKind : uint16_t { RG_PAIRS, RG_U2, RG_DIAG };

// One run of gates of a stage, on its local bit `bit`.
struct __align__(8) RGroup {
  uint16_t bit, nctl;
  uint16_t ctl[4];      // parity masks of the controls
  uint16_t cbits;       // their constants
  uint16_t cm;          // four bits per control: which local flips toggle it
  uint16_t op0, nops;
  int16_t grad;         // row of the group's cross sums, or -1
  uint16_t pad;
};

// RG_PAIRS: groups [g0, g0 + ng) on R targets with flip masks v and parity masks r (constants rc).
// RG_U2 / RG_DIAG: one gate without gradients, its matrix at mat[g0..] (RG_U2 on targets 0 and 1;
// RG_DIAG with local bit 0 at r[0] and bits 1..4 at ctl).
struct __align__(8) RStage {
  uint16_t kind, g0, ng, rc;
  uint16_t v[3], r[3], pivot[3];  // pivots (ascending): storage bits left out when tuples are counted
  uint16_t ctl[4], nctl, cbits;
};

struct RAngle {
  int family, slot;
  double value;
};

}  // namespace

struct ResidentPlan {
  int n = 0;
  bool ok = false;
  bool unique = true;               // every slot has one gate
  int nstages = 0, ngroups = 0, nops = 0, ncs = 0, nmat = 0, ngrad = 0;   // ngrad: groups with gradients
  uint16_t row[kResMaxBits] = {0}, col[kResMaxBits] = {0}, rconst = 0;  // frame after the circuit
  void* d = nullptr;                // stages, groups, ops, angles, matrix offsets
  size_t off_groups = 0, off_ops = 0, off_ang = 0, off_mat = 0;
};

namespace {

// Parameters travel with the launch up to this many; more go up in a copy first.
constexpr int kResTheta = 384;
struct RTheta {
  double v[kResTheta];
};

struct RArgs {
  int n, grad, nstages, ngroups, nops, ncs, nmat, ngrad, nslots, unique, nflips, nstr, B, chunk;
  uint16_t row[kResMaxBits], col[kResMaxBits], rconst;
  const RStage* stages;
  const RGroup* groups;
  const ROp* ops;
  const RAngle* angles;
  const int* mat_off;
  const double2* table;
  const double* theta;              // null: in the launch's RTheta
  const double* weights;
  const double2* init;
  const PFlip* flips;
  const PString* strings;
  double2* values;                  // per sample
  double* gout;                     // weighted gradient, nslots
  double* gsample;                  // per sample rows (more than one sample)
  unsigned* counter;
};

__device__ __forceinline__ int rswz(int i) { return i ^ ((i >> 3) & 7); }
__device__ __forceinline__ unsigned par(unsigned x) { return __popc(x) & 1u; }

struct M2 {
  double2 m00, m10, m01, m11;
};

__device__ __forceinline__ M2 op_matrix(const ROp& op, const double2* cs, const double2* __restrict__ table) {
  const double2 z = cz(), one = make_double2(1.0, 0.0);
  if (op.type == RO_X) return M2{z, one, one, z};
  if (op.type == RO_NEG) return M2{one, z, z, make_double2(-1.0, 0.0)};
  if (op.type == RO_U1) return M2{table[op.e[0]], table[op.e[1]], table[op.e[2]], table[op.e[3]]};
  const double c = cs[op.data].x, s = op.neg ? -cs[op.data].y : cs[op.data].y;
  if (op.type == RO_RX) return M2{make_double2(c, 0.0), make_double2(0.0, -s), make_double2(0.0, -s), make_double2(c, 0.0)};
  if (op.type == RO_RY) return M2{make_double2(c, 0.0), make_double2(s, 0.0), make_double2(-s, 0.0), make_double2(c, 0.0)};
  if (op.type == RO_RZ) return M2{make_double2(c, -s), z, z, make_double2(c, s)};
  return M2{one, z, z, make_double2(c, s)};
}

__device__ __forceinline__ M2 mul(const M2& a, const M2& b) {
  return M2{cfma(a.m01, b.m10, cmul(a.m00, b.m00)), cfma(a.m11, b.m10, cmul(a.m10, b.m00)),
            cfma(a.m01, b.m11, cmul(a.m00, b.m01)), cfma(a.m11, b.m11, cmul(a.m10, b.m01))};
}
__device__ __forceinline__ M2 dagger(const M2& a) { return M2{cconj(a.m00), cconj(a.m01), cconj(a.m10), cconj(a.m11)}; }

__device__ __forceinline__ void apply(const M2& m, double2& x, double2& y) {
  const double2 a = x, b = y;
  x = cfma(m.m01, b, cmul(m.m00, a));
  y = cfma(m.m11, b, cmul(m.m10, a));
}

// Storage index of pair q: a zero inserted at the pivot.
__device__ __forceinline__ int insert0(int q, int pivot) {
  return ((q >> pivot) << (pivot + 1)) | (q & ((1 << pivot) - 1));
}

// Element-wise diagonal and 4x4 gates (no gradients): one state.
__device__ __noinline__ void other_stage(const RStage& g, const double2* mat, double2* s, int n, bool adj) {
  if (g.kind == RG_DIAG) {
    for (int p = threadIdx.x; p < (1 << n); p += blockDim.x) {
      unsigned idx = par(g.r[0] & p) ^ (g.rc & 1u);
      for (int c = 0; c < g.nctl; ++c) idx |= (par(g.ctl[c] & p) ^ ((g.cbits >> c) & 1u)) << (c + 1);
      const double2 f = mat[g.g0 + idx];
      s[rswz(p)] = cmul(adj ? cconj(f) : f, s[rswz(p)]);
    }
    return;
  }
  for (int q = threadIdx.x; q < (1 << (n - 2)); q += blockDim.x) {
    const int p = insert0(insert0(q, g.pivot[0]), g.pivot[1]);
    const unsigned a0 = par(g.r[0] & p) ^ (g.rc & 1u), a1 = par(g.r[1] & p) ^ ((g.rc >> 1) & 1u);
    int at[4];
    double2 x[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      at[m] = rswz(p ^ (((m & 1) ^ a0) ? g.v[0] : 0) ^ (((m >> 1) ^ a1) ? g.v[1] : 0));
      x[m] = s[at[m]];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      double2 acc = cz();
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const double2 u = adj ? cconj(mat[g.g0 + m + 4 * r]) : mat[g.g0 + r + 4 * m];
        acc = cfma(u, x[m], acc);
      }
      s[at[r]] = acc;
    }
  }
}

// Which of a thread's pairs a group acts on: one bit per local index with the target bit clear.
template <int R>
__device__ __forceinline__ unsigned pairs_on(const RGroup& g, unsigned base) {
  unsigned on = (1u << (1 << R)) - 1u;
  for (int c = 0; c < g.nctl; ++c) {
    const unsigned p0 = par(g.ctl[c] & base) ^ ((g.cbits >> c) & 1u), cm = (g.cm >> (4 * c)) & 15u;
    unsigned ok = 0;
#pragma unroll
    for (int m = 0; m < (1 << R); ++m) ok |= (p0 ^ par(cm & unsigned(m))) << m;
    on &= ok;
  }
  return on;
}

// ALL: every pair, without a branch between the pairs' independent chains.
template <int R, int K, bool ALL>
__device__ __forceinline__ void apply_bit(double2 (&a)[1 << R], const M2& m, unsigned on) {
#pragma unroll
  for (int j = 0; j < (1 << R); ++j)
    if (!((j >> K) & 1) && (ALL || ((on >> j) & 1u))) apply(m, a[j], a[j | (1 << K)]);
}

// f(integral constant) for the run-time bit 0 .. R-1.
template <int R, typename F>
__device__ __forceinline__ void on_bit(int bit, F f) {
  if (bit == 0) f(std::integral_constant<int, 0>());
  if constexpr (R > 1) if (bit == 1) f(std::integral_constant<int, 1>());
  if constexpr (R > 2) if (bit == 2) f(std::integral_constant<int, 2>());
}

template <int R, int K, bool ALL>
__device__ __forceinline__ void cross_bit(const double2 (&y)[1 << R], const double2 (&d)[1 << R], unsigned on,
                                          double (&s)[4]) {
#pragma unroll
  for (int j = 0; j < (1 << R); ++j)
    if (!((j >> K) & 1) && (ALL || ((on >> j) & 1u))) {
      const double2 y0 = y[j], y1 = y[j | (1 << K)], d0 = d[j], d1 = d[j | (1 << K)];
      s[0] = fma(d0.y, y0.x, fma(-d0.x, y0.y, s[0]));
      s[1] = fma(d1.y, y1.x, fma(-d1.x, y1.y, s[1]));
      s[2] = fma(d0.y, y1.x, fma(-d0.x, y1.y, fma(d1.y, y0.x, fma(-d1.x, y0.y, s[2]))));
      s[3] = fma(d0.x, y1.x, fma(d0.y, y1.y, fma(-d1.x, y0.x, fma(-d1.y, y0.y, s[3]))));
    }
}

// A thread holds one tuple of 2^R amplitudes per state; the block has 2^(n-R) threads (at least a
// warp: threads past the last tuple load nothing and store nothing).
template <int R>
__global__ void __launch_bounds__(kResMaxThreads) k_resident(const __grid_constant__ RArgs a,
                                                             const __grid_constant__ RTheta th) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int n = a.n, dim = 1 << n, T = blockDim.x, tx = threadIdx.x, b = blockIdx.x;
  constexpr int A = 1 << R;
  double2* psi = reinterpret_cast<double2*>(raw);
  double2* del = psi + dim;
  M2* gm = reinterpret_cast<M2*>(del + (a.grad ? dim : 0));   // fused matrix of every group
  double2* cs = reinterpret_cast<double2*>(gm + a.ngroups);
  double2* mat = cs + a.ncs;
  double2* sc = mat + a.nmat;                              // string coefficients
  double* gbuf = reinterpret_cast<double*>(sc + a.nstr);   // chunk rows of T partial cross sums
  double* gsum = gbuf + (a.grad ? a.chunk * T : 0);        // four cross sums per group with gradients
  RGroup* groups = reinterpret_cast<RGroup*>(gsum + (a.grad ? 4 * a.ngrad : 0));
  RStage* stages = reinterpret_cast<RStage*>(groups + a.ngroups);
  ROp* ops = reinterpret_cast<ROp*>(stages + a.nstages);
  uint32_t* sz = reinterpret_cast<uint32_t*>(ops + a.nops);   // parity mask | constant << 31
  uint32_t* fv = sz + a.nstr;                              // flip masks, first strings
  int* fs = reinterpret_cast<int*>(fv + a.nflips);
  __shared__ double2 wsum[kResMaxThreads / 32];
  __shared__ bool last;

  const double2* init = a.init + (int64_t(b) << n);
  for (int p = tx; p < dim; p += T) psi[rswz(p)] = init[p];
  for (int i = tx; i < a.ncs; i += T) {
    const RAngle ang = a.angles[i];
    const double t = ang.slot < 0 ? ang.value : a.theta ? a.theta[ang.slot] : th.v[ang.slot];
    double s, c;
    sincos(ang.family == MB_FAM_PHASE ? t : 0.5 * t, &s, &c);
    cs[i] = make_double2(c, s);
  }
  for (int i = tx; i < a.nmat; i += T) mat[i] = a.table[a.mat_off[i]];
  for (int i = tx; i < a.nstages; i += T) stages[i] = a.stages[i];
  for (int i = tx; i < a.ngroups; i += T) groups[i] = a.groups[i];
  for (int i = tx; i < a.nops; i += T) ops[i] = a.ops[i];
  bool imag = false;                                       // some string coefficient is not real
  for (int i = tx; i < a.nstr; i += T) {
    const PString p = a.strings[i];
    uint32_t m = 0, k = 0;
    for (int t = 0; t < n; ++t)
      if ((p.z >> t) & 1) m ^= a.row[t], k ^= (a.rconst >> t) & 1u;
    sz[i] = m | (k << 31);
    sc[i] = p.c;
    imag |= p.c.y != 0.0;
  }
  for (int i = tx; i < a.nflips; i += T) {
    const PFlip f = a.flips[i];
    uint32_t m = 0;
    for (int t = 0; t < n; ++t)
      if ((f.x >> t) & 1) m ^= a.col[t];
    fv[i] = m;
    fs[i] = f.s0;
    if (i + 1 == a.nflips) fs[i + 1] = f.s0 + f.ns;
  }
  imag = __syncthreads_or(imag);
  // two threads per group, one column each
  for (int i = tx; i < 2 * a.ngroups; i += T) {
    const RGroup g = groups[i >> 1];
    const M2 first = op_matrix(ops[g.op0], cs, a.table);
    CDD x = wide(i & 1 ? first.m01 : first.m00), y = wide(i & 1 ? first.m11 : first.m10);
    for (int o = 1; o < g.nops; ++o) {
      const M2 m = op_matrix(ops[g.op0 + o], cs, a.table);
      const CDD u = x;
      x = cdot(m.m00, u, m.m01, y);
      y = cdot(m.m10, u, m.m11, y);
    }
    double2* out = reinterpret_cast<double2*>(gm + (i >> 1)) + 2 * (i & 1);   // m00, m10, m01, m11
    out[0] = narrow(x);
    out[1] = narrow(y);
  }
  __syncthreads();

  const int nt = dim >> R;
  const bool mine = tx < nt;
  // Storage slots of this thread's tuple: local index m at at ^ (the flips of m's bits).
  auto slots = [&](const RStage& g, int* sv, unsigned* base) {
    int p = tx;
#pragma unroll
    for (int i = 0; i < R; ++i) p = insert0(p, g.pivot[i]);
    int at = rswz(p);
    unsigned q = unsigned(p);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      sv[i] = rswz(g.v[i]);
      if (par(g.r[i] & unsigned(p)) ^ ((g.rc >> i) & 1u)) at ^= sv[i], q ^= g.v[i];
    }
    *base = q;
    return at;
  };
  auto slot = [](int at, const int* sv, int m) {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if ((m >> i) & 1) at ^= sv[i];
    return at;
  };

  // Forward.
  for (int si = 0; si < a.nstages; ++si) {
    const RStage st = stages[si];
    if (st.kind != RG_PAIRS) {
      other_stage(st, mat, psi, n, false);
      __syncthreads();
      continue;
    }
    if (mine) {
      int sv[R];
      unsigned base;
      const int at = slots(st, sv, &base);
      double2 x[A];
#pragma unroll
      for (int m = 0; m < A; ++m) x[m] = psi[slot(at, sv, m)];
      for (int gi = st.g0; gi < st.g0 + st.ng; ++gi) {
        const RGroup& g = groups[gi];
        const M2 m = gm[gi];
        if (g.nctl == 0) {
          on_bit<R>(g.bit, [&](auto k) { apply_bit<R, decltype(k)::value, true>(x, m, 0u); });
        } else {
          const unsigned on = pairs_on<R>(g, base);
          on_bit<R>(g.bit, [&](auto k) { apply_bit<R, decltype(k)::value, false>(x, m, on); });
        }
      }
#pragma unroll
      for (int m = 0; m < A; ++m) psi[slot(at, sv, m)] = x[m];
    }
    __syncthreads();
  }

  // <H>, and delta = 2 H psi for the reverse (Hermitian H, expectation.jl:4-73).
  // A thread takes its 2^R amplitudes together, so a string is read once for all of them.
  double2 e = cz();
  if (mine) {
    double2 h[A];
#pragma unroll
    for (int k = 0; k < A; ++k) h[k] = cz();
    for (int f = 0; f < a.nflips; ++f) {
      const unsigned x = fv[f];
      double2 c[A];
#pragma unroll
      for (int k = 0; k < A; ++k) c[k] = cz();
      for (int s = fs[f]; s < fs[f + 1]; ++s) {
        const uint32_t z = sz[s];
        const double2 v = sc[s];
#pragma unroll
        for (int k = 0; k < A; ++k) {
          const unsigned src = unsigned(tx + k * nt) ^ x;
          const long long flip = (long long)(par(z & 0x7fffffffu & src) ^ (z >> 31)) << 63;
          c[k].x += __longlong_as_double(__double_as_longlong(v.x) ^ flip);
          if (imag) c[k].y += __longlong_as_double(__double_as_longlong(v.y) ^ flip);
        }
      }
#pragma unroll
      for (int k = 0; k < A; ++k) h[k] = cfma(c[k], psi[rswz((tx + k * nt) ^ int(x))], h[k]);
    }
#pragma unroll
    for (int k = 0; k < A; ++k) {
      const int i = rswz(tx + k * nt);
      e = cfma_conj(psi[i], h[k], e);
      if (a.grad) del[i] = make_double2(2.0 * h[k].x, 2.0 * h[k].y);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    e.x += __shfl_xor_sync(0xffffffffu, e.x, o);
    e.y += __shfl_xor_sync(0xffffffffu, e.y, o);
  }
  if ((tx & 31) == 0) wsum[tx >> 5] = e;
  __syncthreads();
  if (tx == 0) {
    for (int w = 1; w < (T >> 5); ++w) e = cadd(e, wsum[w]);
    a.values[b] = e;
  }
  if (!a.grad) return;

  // Reverse. A group's gradients all follow from the cross sums C = sum over its pairs of
  // delta y' after the group: with y_k = V y before gate k, Re<y_k|D|delta_k> = Re tr(V'DV C), and
  // V'DV is anti-Hermitian, so four real sums serve every gate of the group.
  int row = 0, done = 0;                                   // rows waiting in gbuf; rows already added
  auto add_rows = [&]() {
    // lane l of a row's threads holds sum l & 3
    for (int r = tx >> 5; r < row; r += T >> 5) {
      double s = 0.0;
      for (int i = tx & 31; i < T; i += 32) s += gbuf[r * T + i];
#pragma unroll
      for (int o = 16; o >= 4; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((tx & 31) < 4) gsum[4 * (done + r) + (tx & 3)] = s;
    }
    done += row;
    row = 0;
  };
  for (int si = a.nstages - 1; si >= 0; --si) {
    const RStage st = stages[si];
    if (st.kind != RG_PAIRS) {
      other_stage(st, mat, psi, n, true);
      other_stage(st, mat, del, n, true);
      __syncthreads();
      continue;
    }
    int sv[R], at = 0;
    unsigned base = 0;
    double2 y[A], d[A];
    if (mine) {
      at = slots(st, sv, &base);
#pragma unroll
      for (int m = 0; m < A; ++m) {
        const int i = slot(at, sv, m);
        y[m] = psi[i];
        d[m] = del[i];
      }
    }
    for (int gi = st.g0 + st.ng - 1; gi >= st.g0; --gi) {
      const RGroup& g = groups[gi];
      double s[4] = {0.0, 0.0, 0.0, 0.0};
      if (mine) {
        const M2 m = dagger(gm[gi]);
        if (g.nctl == 0) {
          on_bit<R>(g.bit, [&](auto k) {
            constexpr int K = decltype(k)::value;
            if (g.grad >= 0) cross_bit<R, K, true>(y, d, 0u, s);
            apply_bit<R, K, true>(y, m, 0u);
            apply_bit<R, K, true>(d, m, 0u);
          });
        } else {
          const unsigned on = pairs_on<R>(g, base);
          on_bit<R>(g.bit, [&](auto k) {
            constexpr int K = decltype(k)::value;
            if (g.grad >= 0) cross_bit<R, K, false>(y, d, on, s);
            apply_bit<R, K, false>(y, m, on);
            apply_bit<R, K, false>(d, m, on);
          });
        }
      }
      if (g.grad >= 0) {
        if (row == a.chunk) {
          __syncthreads();
          add_rows();
          __syncthreads();
        }
        // lane bits 0 and 1 choose the sum a lane keeps
        const bool b0 = tx & 1, b1 = tx & 2;
        const double u0 = (b0 ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, b0 ? s[0] : s[1], 1);
        const double u1 = (b0 ? s[3] : s[2]) + __shfl_xor_sync(0xffffffffu, b0 ? s[2] : s[3], 1);
        gbuf[row * T + tx] = (b1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2);
        ++row;
      }
    }
    if (mine)
#pragma unroll
      for (int m = 0; m < A; ++m) {
        const int i = slot(at, sv, m);
        psi[i] = y[m];
        del[i] = d[m];
      }
    __syncthreads();
  }
  add_rows();

  double* gs = a.B > 1 ? a.gsample + int64_t(b) * a.nslots : a.gout;
  for (int s = tx; s < a.nslots; s += T) gs[s] = 0.0;
  __syncthreads();
  const double scale = a.B > 1 ? 1.0 : a.weights[0];
  auto gate_gradient = [&](int o) {
    const ROp op = ops[o];
    const RGroup g = groups[op.group];
    M2 V = dagger(op_matrix(ops[g.op0 + g.nops - 1], cs, a.table));
    for (int k = g.op0 + g.nops - 2; k >= o; --k) V = mul(dagger(op_matrix(ops[k], cs, a.table)), V);
    // generators (i/2)X, (i/2)Y, (i/2)Z, diag(0, -i)
    const double2 z = cz();
    M2 D{z, z, z, z};
    if (op.type == RO_RX) D.m01 = D.m10 = make_double2(0.0, 0.5);
    else if (op.type == RO_RY) D.m01 = make_double2(0.5, 0.0), D.m10 = make_double2(-0.5, 0.0);
    else if (op.type == RO_RZ) D.m00 = make_double2(0.0, 0.5), D.m11 = make_double2(0.0, -0.5);
    else D.m11 = make_double2(0.0, -1.0);
    const M2 M = mul(dagger(V), mul(D, V));
    const double* C = gsum + 4 * g.grad;
    const double s = -(M.m00.y * C[0] + M.m11.y * C[1] + M.m01.x * C[3] + M.m01.y * C[2]);
    return scale * (op.neg ? -s : s);
  };
  if (a.unique) {
    for (int o = tx; o < a.nops; o += T) {
      const int slot = ops[o].slot;
      if (slot >= 0) gs[slot] = gate_gradient(o);
    }
  } else if (tx == 0) {
    for (int o = 0; o < a.nops; ++o) {
      const int slot = ops[o].slot;
      if (slot >= 0) gs[slot] += gate_gradient(o);
    }
  }
  if (a.B == 1) return;
  // The last sample to finish adds the weighted rows, samples in order.
  __threadfence();
  __syncthreads();
  if (tx == 0) last = atomicAdd(a.counter, 1u) == unsigned(a.B - 1);
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int s = tx; s < a.nslots; s += T) {
    double sum = 0.0;
#pragma unroll 8
    for (int q = 0; q < a.B; ++q) sum = fma(a.weights[q], __ldcg(a.gsample + int64_t(q) * a.nslots + s), sum);
    a.gout[s] = sum;
  }
  if (tx == 0) *a.counter = 0;
}

// ---- host: the plan of one circuit ------------------------------------------------------------
struct Builder {
  mb_circuit c;
  ResidentPlan* P;
  int R;
  std::vector<RStage> stages;
  std::vector<RGroup> groups;
  std::vector<ROp> ops;
  std::vector<RAngle> angles;
  std::vector<int> mats;
  struct Control {
    uint16_t n = 0, ctl[4] = {0, 0, 0, 0}, cbits = 0;
  };
  struct Held {
    ROp op;
    Control ctl;
  };
  std::vector<Held> open[kResMaxBits];
  uint16_t row[kResMaxBits], col[kResMaxBits], rconst = 0;
  // The stage being filled: its targets and the frame it runs in.
  bool filling = false;
  std::vector<int> targets;
  uint16_t srow[kResMaxBits], scol[kResMaxBits], sconst = 0;

  uint16_t bit(int t) const { return uint16_t((rconst >> t) & 1); }
  static uint16_t high_bit(unsigned v) { return uint16_t(31 - __builtin_clz(v)); }

  // Pivots of `count` independent flip masks: storage bits of which every tuple has exactly one
  // member with all of them clear.
  static void pivots(const uint16_t* v, int count, uint16_t* out) {
    uint16_t w[3];
    for (int i = 0; i < count; ++i) {
      w[i] = v[i];
      for (int j = 0; j < i; ++j)
        if ((w[i] >> out[j]) & 1) w[i] ^= w[j];
      out[i] = high_bit(w[i]);
      for (int j = 0; j < i; ++j)
        if ((w[j] >> out[i]) & 1) w[j] ^= w[i];
    }
    std::sort(out, out + count);
  }
  void finish_stage() {
    if (!filling) return;
    filling = false;
    RStage& s = stages.back();
    // free places hold other qubits of the frame
    for (int q = 0; q < c->n && int(targets.size()) < R; ++q)
      if (std::find(targets.begin(), targets.end(), q) == targets.end()) targets.push_back(q);
    for (int i = 0; i < R; ++i) {
      s.v[i] = scol[targets[i]];
      s.r[i] = srow[targets[i]];
      s.rc |= uint16_t(((sconst >> targets[i]) & 1) << i);
    }
    pivots(s.v, R, s.pivot);
    for (int g = s.g0; g < s.g0 + s.ng; ++g)
      for (int k = 0; k < groups[g].nctl; ++k)
        for (int i = 0; i < R; ++i)
          groups[g].cm |= uint16_t((__builtin_popcount(groups[g].ctl[k] & s.v[i]) & 1) << (4 * k + i));
  }
  // Local bit of qubit q in the stage being filled, starting another if q or its frame does not fit.
  int place(int q) {
    if (filling && (scol[q] != col[q] || srow[q] != row[q] || ((sconst >> q) & 1) != bit(q))) finish_stage();
    if (filling) {
      const auto it = std::find(targets.begin(), targets.end(), q);
      if (it != targets.end()) return int(it - targets.begin());
      if (int(targets.size()) == R) finish_stage();
    }
    if (!filling) {
      filling = true;
      targets.clear();
      std::copy(row, row + c->n, srow);
      std::copy(col, col + c->n, scol);
      sconst = rconst;
      RStage s{};
      s.kind = RG_PAIRS;
      s.g0 = uint16_t(groups.size());
      stages.push_back(s);
    }
    targets.push_back(q);
    return int(targets.size()) - 1;
  }
  void close(int q) {
    if (open[q].empty()) return;
    // a controlled gate is a group by itself: its predecessors on the target go before it
    const Control& last = open[q].back().ctl;
    const size_t count = open[q].size() - (last.n ? 1 : 0);
    if (count) emit(q, Control(), open[q].data(), count);
    if (last.n) emit(q, last, &open[q].back(), 1);
    open[q].clear();
  }
  void emit(int q, const Control& ctl, const Held* h, size_t count) {
    RGroup g{};
    g.bit = uint16_t(place(q));
    g.nctl = ctl.n;
    std::copy(ctl.ctl, ctl.ctl + 4, g.ctl);
    g.cbits = ctl.cbits;
    g.op0 = uint16_t(ops.size());
    g.nops = uint16_t(count);
    g.grad = -1;
    for (size_t i = 0; i < count; ++i) {
      ops.push_back(h[i].op);
      ops.back().group = uint16_t(groups.size());
      if (h[i].op.slot >= 0) g.grad = 0;
    }
    groups.push_back(g);
    stages.back().ng += 1;
  }
  Control controls(const int* q, int count) const {
    Control k;
    k.n = uint16_t(count);
    for (int j = 0; j < count; ++j) {
      k.ctl[j] = row[q[j]];
      k.cbits |= uint16_t(bit(q[j]) << j);
    }
    return k;
  }
  // A single-target gate: it joins the target's open group; with controls it also ends it, so that
  // later gates on a control cannot be emitted before it.
  void single(ROp op, int t, const int* ctl, int nctl) {
    for (int j = 0; j < nctl; ++j) close(ctl[j]);
    open[t].push_back(Held{op, controls(ctl, nctl)});
    if (nctl) close(t);
  }
  uint16_t matrix(const COp& o, int count, const int* elems) {
    const uint16_t at = uint16_t(mats.size());
    for (int e = 0; e < count; ++e) mats.push_back(o.mat_off + elems[e]);
    return at;
  }

  bool add(const COp& o) {
    if (o.kind != MB_OP_GATE || o.k < 1) return false;
    const int d = 1 << o.k;
    if (o.parametric) {
      int fam = o.family, tj = 0;
      if (fam == MB_FAM_SELECT) return false;
      if (o.k > 1) {
        const BindRec* br = nullptr;
        for (const BindRec& r : c->binds)
          if (r.mat_off == o.mat_off) br = &r;
        if (!br) return false;
        for (int j = 0; j < o.k; ++j)
          if (br->perm[1 << j] == d / 2) tj = j;   // own-order top bit: the target
        fam = fam == MB_FAM_CCPHASE ? int(MB_FAM_PHASE) : fam - MB_FAM_CRX + MB_FAM_RX;
      }
      ROp op{};
      op.type = uint16_t(fam == MB_FAM_RX ? RO_RX : fam == MB_FAM_RY ? RO_RY : fam == MB_FAM_RZ ? RO_RZ : RO_PHASE);
      op.data = int32_t(angles.size());
      angles.push_back(RAngle{fam, o.slot, o.value});
      op.neg = (o.flags & MB_OPF_ADJOINT) ? 1 : 0;
      op.slot = int16_t(o.gen_off >= 0 ? o.slot : -1);
      int ctl[4], nc = 0;
      for (int j = 0; j < o.k; ++j)
        if (j != tj) ctl[nc++] = o.pos[j];
      single(op, o.pos[tj], ctl, nc);
      return true;
    }
    const double2* M = c->fixed_table.data() + o.mat_off;
    auto is = [&](int r, int cc, double x) { return M[r + d * cc].x == x && M[r + d * cc].y == 0.0; };
    // SWAP
    if (o.k == 2 && is(0, 0, 1) && is(1, 2, 1) && is(2, 1, 1) && is(3, 3, 1) && o.cls == CLS_MONO) {
      close(o.pos[0]);
      close(o.pos[1]);
      std::swap(row[o.pos[0]], row[o.pos[1]]);
      std::swap(col[o.pos[0]], col[o.pos[1]]);
      const uint16_t b0 = bit(o.pos[0]), b1 = bit(o.pos[1]);
      if (b0 != b1) rconst ^= uint16_t((1 << o.pos[0]) | (1 << o.pos[1]));
      return true;
    }
    const int tj = o.k == 1 ? 0 : controlled_target(M, o.k);
    if (tj >= 0) {
      const int tb = 1 << tj, cm = (d - 1) & ~tb;
      const int e[4] = {cm + d * cm, (cm | tb) + d * cm, cm + d * (cm | tb), (cm | tb) + d * (cm | tb)};
      const bool x = is(cm, cm, 0) && is(cm | tb, cm, 1) && is(cm, cm | tb, 1) && is(cm | tb, cm | tb, 0);
      const bool neg = is(cm, cm, 1) && is(cm | tb, cm, 0) && is(cm, cm | tb, 0) && is(cm | tb, cm | tb, -1);
      int ctl[4], nc = 0;
      const int t = o.pos[tj];
      for (int j = 0; j < o.k; ++j)
        if (j != tj) ctl[nc++] = o.pos[j];
      if (x && nc == 0) {
        close(t);
        rconst ^= uint16_t(1 << t);
        return true;
      }
      if (x && nc == 1) {
        // CNOT: bit t becomes t ^ c; toggling c alone must now toggle t's old value too
        close(t);
        close(ctl[0]);
        row[t] ^= row[ctl[0]];
        if (bit(ctl[0])) rconst ^= uint16_t(1 << t);
        col[ctl[0]] ^= col[t];
        return true;
      }
      ROp op{};
      op.type = uint16_t(x ? RO_X : neg ? RO_NEG : RO_U1);
      op.slot = -1;
      for (int i = 0; i < 4; ++i) op.e[i] = o.mat_off + e[i];
      single(op, t, ctl, nc);
      return true;
    }
    for (int j = 0; j < o.k; ++j) close(o.pos[j]);
    RStage g{};
    g.v[0] = col[o.pos[0]];
    g.r[0] = row[o.pos[0]];
    g.rc = bit(o.pos[0]);
    if (o.cls == CLS_DIAG) {
      g.kind = RG_DIAG;
      int e[32];
      for (int i = 0; i < d; ++i) e[i] = i * (d + 1);
      g.g0 = matrix(o, d, e);
      const Control k = controls(o.pos + 1, o.k - 1);
      g.nctl = k.n;
      std::copy(k.ctl, k.ctl + 4, g.ctl);
      g.cbits = k.cbits;
    } else if (o.k == 2) {
      g.kind = RG_U2;
      int e[16];
      for (int i = 0; i < 16; ++i) e[i] = i;
      g.g0 = matrix(o, 16, e);
      g.v[1] = col[o.pos[1]];
      g.r[1] = row[o.pos[1]];
      g.rc |= uint16_t(bit(o.pos[1]) << 1);
      pivots(g.v, 2, g.pivot);
    } else {
      return false;
    }
    finish_stage();
    stages.push_back(g);
    return true;
  }
};

// Qubits per stage: three from 9 qubits; below, two keep more than one warp busy (8 qubits: 64 threads).
int resident_width(int n) { return n >= 9 ? 3 : n >= 4 ? 2 : 1; }
int resident_threads(int n) { return std::max(32, 1 << (n - resident_width(n))); }

size_t resident_shared(const ResidentPlan& P, int nflips, int nstr, bool grad, int T, int chunk) {
  size_t s = (sizeof(double2) << P.n) * (grad ? 2 : 1);
  s += sizeof(double2) * (size_t(P.ncs) + P.nmat + nstr) + sizeof(M2) * size_t(P.ngroups);
  if (grad) s += sizeof(double) * (size_t(chunk) * T + 4 * size_t(P.ngrad));
  s += sizeof(RGroup) * size_t(P.ngroups) + sizeof(RStage) * size_t(P.nstages) + sizeof(ROp) * size_t(P.nops);
  s += sizeof(uint32_t) * (size_t(nstr) + 2 * size_t(nflips) + 1);
  return (s + 15) & ~size_t(15);
}

int build_plan(mb_circuit c, ResidentPlan* P) {
  P->n = c->n;
  Builder B;
  B.c = c;
  B.P = P;
  B.R = resident_width(c->n);
  for (int t = 0; t < c->n; ++t) B.row[t] = B.col[t] = uint16_t(1 << t);
  for (const COp& o : c->ops) {
    // 16-bit indexes, and room left in shared memory in any case
    if (B.groups.size() > 4000 || B.ops.size() > 16000 || c->nslots > 32767 || B.angles.size() > 4000 || B.mats.size() > 8000) return MB_OK;
    if (!B.add(o)) return MB_OK;
  }
  for (int q = 0; q < c->n; ++q) B.close(q);
  B.finish_stage();
  // rows of the cross sums in the order the reverse meets the groups
  for (size_t g = B.groups.size(); g-- > 0;)
    if (B.groups[g].grad >= 0) {
      if (P->ngrad == 32767) return MB_OK;
      B.groups[g].grad = int16_t(P->ngrad++);
    }
  std::vector<char> seen(size_t(std::max(1, c->nslots)), 0);
  for (const ROp& op : B.ops)
    if (op.slot >= 0) {
      P->unique = P->unique && !seen[op.slot];
      seen[op.slot] = 1;
    }
  P->nstages = int(B.stages.size());
  P->ngroups = int(B.groups.size());
  P->nops = int(B.ops.size());
  P->ncs = int(B.angles.size());
  P->nmat = int(B.mats.size());
  std::memcpy(P->row, B.row, sizeof(P->row));
  std::memcpy(P->col, B.col, sizeof(P->col));
  P->rconst = B.rconst;
  std::vector<unsigned char> h;
  auto put = [&](const void* d, size_t bytes) {
    const size_t at = (h.size() + 15) & ~size_t(15);
    h.resize(at + bytes);
    if (bytes) std::memcpy(h.data() + at, d, bytes);
    return at;
  };
  put(B.stages.data(), sizeof(RStage) * B.stages.size());
  P->off_groups = put(B.groups.data(), sizeof(RGroup) * B.groups.size());
  P->off_ops = put(B.ops.data(), sizeof(ROp) * B.ops.size());
  P->off_ang = put(B.angles.data(), sizeof(RAngle) * B.angles.size());
  P->off_mat = put(B.mats.data(), sizeof(int) * B.mats.size());
  if (int rc = dev_alloc(&P->d, h.size())) return rc;
  MB_CHECK_CUDA(cudaMemcpyAsync(P->d, h.data(), h.size(), cudaMemcpyHostToDevice, g_ctx.stream));
  MB_CHECK_CUDA(cudaStreamSynchronize(g_ctx.stream));
  P->ok = true;
  return MB_OK;
}

}  // namespace

void resident_release(mb_circuit c) {
  if (!c->resident) return;
  dev_free(c->resident->d);
  delete c->resident;
  c->resident = nullptr;
}

int resident_run(mb_circuit c, mb_observable o, mb_state init, const double* theta, const double* weights,
                 double2* values, double* grad, bool* done) {
  *done = false;
  const int n = c->n, B = init->batch;
  const bool pure = init->kind == MB_PURE || init->kind == MB_BATCH_PURE;
  if (!pure || c->has_channel || n < 1 || n > kResMaxBits || B < 1 || g_ctx.capturing) return MB_OK;
  const char* on = getenv("MB_RESIDENT");   // 0: every objective through the general passes
  if (on && atoi(on) == 0) return MB_OK;
  ObsStrings os;
  if (!observable_strings(o, n, 1024, &os)) return MB_OK;
  if (!c->resident) {
    c->resident = new ResidentPlan();
    if (int rc = build_plan(c, c->resident)) {
      resident_release(c);
      return rc;
    }
  }
  const ResidentPlan& P = *c->resident;
  if (!P.ok) return MB_OK;
  const int T = resident_threads(n);
  // Rows per chunk: 32 KiB of partial cross sums.
  const int chunk = std::max(4, 4096 / T);
  const size_t shm = resident_shared(P, os.nflips, os.nstr, grad != nullptr, T, chunk);
  if (shm > kResMaxShared) return MB_OK;

  // Parameters travel with the launch and results are written to pinned memory: at these sizes each
  // copy on the stream costs more than it moves. Weights, which only the last of several samples
  // reads, and long parameter lists go up in a copy. The call waits for its results, so the buffers
  // are free again when it returns.
  const size_t ns = size_t(c->nslots), nw = grad ? size_t(B) : 0;
  const size_t down = 2 * size_t(B) + (grad ? ns : 0), rows = grad && B > 1 ? size_t(B) * ns : 0;
  SmallBufs bufs;
  if (bufs.take(ns + nw + down, ns + nw + rows)) return MB_OK;   // no room: the general form
  double* hp = bufs.h;
  double* dp = bufs.d;
  RTheta th;
  const bool direct = ns <= kResTheta;
  std::copy(theta, theta + ns, direct ? th.v : hp);
  if (grad) std::copy(weights, weights + B, hp + ns);
  cudaStream_t st = g_ctx.stream;
  const size_t first = direct ? ns : 0, up = B > 1 || !direct ? ns + nw - first : 0;
  if (up) MB_CHECK_CUDA(cudaMemcpyAsync(dp + first, hp + first, sizeof(double) * up, cudaMemcpyHostToDevice, st));

  RArgs a{};
  a.n = n;
  a.grad = grad ? 1 : 0;
  a.nstages = P.nstages;
  a.ngroups = P.ngroups;
  a.nops = P.nops;
  a.ncs = P.ncs;
  a.nmat = P.nmat;
  a.ngrad = P.ngrad;
  a.nslots = c->nslots;
  a.unique = P.unique;
  a.nflips = os.nflips;
  a.nstr = os.nstr;
  a.B = B;
  a.chunk = chunk;
  std::memcpy(a.row, P.row, sizeof(a.row));
  std::memcpy(a.col, P.col, sizeof(a.col));
  a.rconst = P.rconst;
  const unsigned char* d = static_cast<const unsigned char*>(P.d);
  a.stages = reinterpret_cast<const RStage*>(d);
  a.groups = reinterpret_cast<const RGroup*>(d + P.off_groups);
  a.ops = reinterpret_cast<const ROp*>(d + P.off_ops);
  a.angles = reinterpret_cast<const RAngle*>(d + P.off_ang);
  a.mat_off = reinterpret_cast<const int*>(d + P.off_mat);
  a.table = c->d_table;
  a.theta = direct ? nullptr : dp;
  a.weights = (B > 1 ? dp : hp) + ns;
  a.init = init->d;
  a.flips = os.flips;
  a.strings = os.strings;
  double* res = hp + ns + nw + ((ns + nw) & 1);   // 16-byte aligned; the buffer leaves room
  a.values = reinterpret_cast<double2*>(res);
  a.gout = res + 2 * size_t(B);
  a.gsample = dp + ns + nw;
  a.counter = g_ctx.counters;
  auto launch = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(shm));
    kern<<<B, T, shm, st>>>(a, th);
  };
  {
    ProfScope ps("k_resident", 16.0 * double(init->elems) * B, st);
    if (resident_width(n) == 3) launch(k_resident<3>);
    else if (resident_width(n) == 2) launch(k_resident<2>);
    else launch(k_resident<1>);
  }
  MB_LAUNCHED();
  MB_CHECK_CUDA(cudaStreamSynchronize(st));
  std::memcpy(values, res, sizeof(double2) * B);
  if (grad) std::copy(res + 2 * size_t(B), res + down, grad);
  *done = true;
  return MB_OK;
}

}  // namespace mb
