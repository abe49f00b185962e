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
//    bound: the hardware-efficient ansatz takes n steps per layer.
//  - Gradients. All gradients of a group follow from four cross sums of its pairs (k_resident's
//    reverse); a step only stores each thread's part, and the parts are added a chunk at a time.
// Sums have a fixed order: the same bits on every run.
// Measured (8 qubits, 2 layers of the ansatz): value 20 us and gradient 28 us, where the plain
// reverse took 266 launches (1.98 ms per call); 48 samples of 12 qubits, 4 layers: 220 us against
// 732 launches (5.3 ms). Above 12 qubits the passes over HBM are the only form: two states no longer
// fit one SM.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

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

enum RKind : uint16_t { RG_PAIR, RG_U2, RG_DIAG };

struct __align__(8) RGroup {
  uint16_t kind, nctl;
  uint16_t ctl[4];      // parity masks of the controls (RG_DIAG: of local bits 1..4)
  uint16_t cbits;       // their constants
  uint16_t v, r;        // flip mask and parity mask of the target
  uint16_t rc, pivot;   // parity constant; storage bit left out when pairs are counted
  uint16_t v2, r2;      // RG_U2: second bit
  uint16_t rc2, pivot2;
  uint16_t op0, nops;   // RG_PAIR: gates; others: first entry in mat
  int16_t grad;         // row of the group's cross sums, or -1
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
  int ngroups = 0, nops = 0, ncs = 0, nmat = 0, ngrad = 0;   // ngrad: groups with gradients
  uint16_t row[kResMaxBits] = {0}, col[kResMaxBits] = {0}, rconst = 0;  // frame after the circuit
  void* d = nullptr;                // groups, ops, angles, matrix offsets
  size_t off_ops = 0, off_ang = 0, off_mat = 0;
};

namespace {

struct RArgs {
  int n, grad, ngroups, nops, ncs, nmat, ngrad, nslots, unique, nflips, nstr, B, chunk;
  uint16_t row[kResMaxBits], col[kResMaxBits], rconst;
  const RGroup* groups;
  const ROp* ops;
  const RAngle* angles;
  const int* mat_off;
  const double2* table;
  const double* theta;
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

__device__ __forceinline__ bool controls_on(const RGroup& g, unsigned p) {
  bool on = true;
  for (int c = 0; c < g.nctl; ++c) on = on && (par(g.ctl[c] & p) ^ ((g.cbits >> c) & 1u));
  return on;
}

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

// A run's product is rounded once: its entries are carried as high and low parts, because an error
// of the matrix is the same for every amplitude and adds up over the steps, where roundings of
// amplitudes average out.
struct DD {
  double h, l;
};
__device__ __forceinline__ DD dd_fma(double a, DD b, DD c) {
  const double p = a * b.h, q = fma(a, b.h, -p) + a * b.l;     // a * b
  const double s = c.h + p, z = s - c.h;
  const double r = ((c.h - (s - z)) + (p - z)) + (c.l + q);    // two-sum of the high parts
  const double h = s + r;
  return DD{h, r - (h - s)};
}
struct CDD {
  DD x, y;
};
struct M2DD {
  CDD m00, m10, m01, m11;
};
__device__ __forceinline__ CDD wide(double2 a) { return CDD{DD{a.x, 0.0}, DD{a.y, 0.0}}; }
__device__ __forceinline__ double2 narrow(const CDD& a) { return make_double2(a.x.h, a.y.h); }
// a * b + c * d
__device__ __forceinline__ CDD cdot(double2 a, const CDD& b, double2 c, const CDD& d) {
  const DD z{0.0, 0.0};
  return CDD{dd_fma(-c.y, d.y, dd_fma(c.x, d.x, dd_fma(-a.y, b.y, dd_fma(a.x, b.x, z)))),
             dd_fma(c.y, d.x, dd_fma(c.x, d.y, dd_fma(a.y, b.x, dd_fma(a.x, b.y, z))))};
}
__device__ __forceinline__ M2DD mul(const M2& a, const M2DD& b) {
  return M2DD{cdot(a.m00, b.m00, a.m01, b.m10), cdot(a.m10, b.m00, a.m11, b.m10),
              cdot(a.m00, b.m01, a.m01, b.m11), cdot(a.m10, b.m01, a.m11, b.m11)};
}

// Storage index of pair q: a zero inserted at the pivot.
__device__ __forceinline__ int insert0(int q, int pivot) {
  return ((q >> pivot) << (pivot + 1)) | (q & ((1 << pivot) - 1));
}

// Element-wise diagonal and 4x4 groups (no gradients): one state.
__device__ __noinline__ void other_group(const RGroup& g, const double2* mat, double2* s, int n, bool adj) {
  if (g.kind == RG_DIAG) {
    for (int p = threadIdx.x; p < (1 << n); p += blockDim.x) {
      unsigned idx = par(g.r & p) ^ g.rc;
      for (int c = 0; c < g.nctl; ++c) idx |= (par(g.ctl[c] & p) ^ ((g.cbits >> c) & 1u)) << (c + 1);
      const double2 f = mat[g.op0 + idx];
      s[rswz(p)] = cmul(adj ? cconj(f) : f, s[rswz(p)]);
    }
    return;
  }
  const int lo = min(g.pivot, g.pivot2), hi = max(g.pivot, g.pivot2);
  for (int q = threadIdx.x; q < (1 << (n - 2)); q += blockDim.x) {
    const int p = insert0(insert0(q, lo), hi);
    const unsigned a0 = par(g.r & p) ^ g.rc, a1 = par(g.r2 & p) ^ g.rc2;
    int at[4];
    double2 x[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      at[m] = rswz(p ^ (((m & 1) ^ a0) ? g.v : 0) ^ (((m >> 1) ^ a1) ? g.v2 : 0));
      x[m] = s[at[m]];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      double2 acc = cz();
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const double2 u = adj ? cconj(mat[g.op0 + m + 4 * r]) : mat[g.op0 + r + 4 * m];
        acc = cfma(u, x[m], acc);
      }
      s[at[r]] = acc;
    }
  }
}

// PAIRS pairs per thread; the block has 2^(n-1) / PAIRS threads (at least a warp: below 6 qubits the
// threads past the last pair carry zeros and store nothing).
template <int PAIRS>
__global__ void __launch_bounds__(kResMaxThreads) k_resident(const RArgs a) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int n = a.n, dim = 1 << n, npairs = dim >> 1, T = blockDim.x, tx = threadIdx.x, b = blockIdx.x;
  double2* psi = reinterpret_cast<double2*>(raw);
  double2* del = psi + dim;
  M2* gm = reinterpret_cast<M2*>(del + (a.grad ? dim : 0));   // fused matrix of every group
  double2* cs = reinterpret_cast<double2*>(gm + a.ngroups);
  double2* mat = cs + a.ncs;
  double2* sc = mat + a.nmat;                              // string coefficients
  double* gbuf = reinterpret_cast<double*>(sc + a.nstr);   // chunk rows of T partial cross sums
  double* gsum = gbuf + (a.grad ? a.chunk * T : 0);        // four cross sums per group with gradients
  RGroup* groups = reinterpret_cast<RGroup*>(gsum + (a.grad ? 4 * a.ngrad : 0));
  uint32_t* sz = reinterpret_cast<uint32_t*>(groups + a.ngroups);   // parity mask | constant << 31
  uint32_t* fv = sz + a.nstr;                              // flip masks, first strings
  int* fs = reinterpret_cast<int*>(fv + a.nflips);
  __shared__ double2 wsum[kResMaxThreads / 32];
  __shared__ bool last;

  const double2* init = a.init + (int64_t(b) << n);
  for (int p = tx; p < dim; p += T) psi[rswz(p)] = init[p];
  for (int i = tx; i < a.ncs; i += T) {
    const RAngle ang = a.angles[i];
    const double t = ang.slot >= 0 ? a.theta[ang.slot] : ang.value;
    double s, c;
    sincos(ang.family == MB_FAM_PHASE ? t : 0.5 * t, &s, &c);
    cs[i] = make_double2(c, s);
  }
  for (int i = tx; i < a.nmat; i += T) mat[i] = a.table[a.mat_off[i]];
  for (int i = tx; i < a.nstr; i += T) {
    const PString p = a.strings[i];
    uint32_t m = 0, k = 0;
    for (int t = 0; t < n; ++t)
      if ((p.z >> t) & 1) m ^= a.row[t], k ^= (a.rconst >> t) & 1u;
    sz[i] = m | (k << 31);
    sc[i] = p.c;
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
  __syncthreads();
  for (int i = tx; i < a.ngroups; i += T) {
    const RGroup g = a.groups[i];
    groups[i] = g;
    if (g.kind != RG_PAIR) continue;
    const M2 first = op_matrix(a.ops[g.op0], cs, a.table);
    M2DD m{wide(first.m00), wide(first.m10), wide(first.m01), wide(first.m11)};
    for (int o = 1; o < g.nops; ++o) m = mul(op_matrix(a.ops[g.op0 + o], cs, a.table), m);
    gm[i] = M2{narrow(m.m00), narrow(m.m10), narrow(m.m01), narrow(m.m11)};
  }
  __syncthreads();

  // Forward.
  for (int gi = 0; gi < a.ngroups; ++gi) {
    const RGroup g = groups[gi];
    if (g.kind != RG_PAIR) {
      other_group(g, mat, psi, n, false);
      __syncthreads();
      continue;
    }
    const M2 m = gm[gi];
    const int sv = rswz(g.v);
    // every pair is loaded before one is stored: the loads of a thread overlap
    int i0[PAIRS];
    double2 x[PAIRS], y[PAIRS];
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int p = insert0(tx + k * T, g.pivot);
      i0[k] = tx + k * T < npairs && controls_on(g, p) ? rswz(p) ^ ((par(g.r & p) ^ g.rc) ? sv : 0) : -1;
      if (i0[k] >= 0) x[k] = psi[i0[k]], y[k] = psi[i0[k] ^ sv];
    }
#pragma unroll
    for (int k = 0; k < PAIRS; ++k)
      if (i0[k] >= 0) {
        apply(m, x[k], y[k]);
        psi[i0[k]] = x[k];
        psi[i0[k] ^ sv] = y[k];
      }
    __syncthreads();
  }

  // <H>, and delta = 2 H psi for the reverse (Hermitian H, expectation.jl:4-73).
  double2 e = cz();
  for (int p = tx; p < dim; p += T) {
    double2 h = cz();
    for (int f = 0; f < a.nflips; ++f) {
      const unsigned src = unsigned(p) ^ fv[f];
      double2 c = cz();
      for (int s = fs[f]; s < fs[f + 1]; ++s) {
        const bool odd = (par(sz[s] & 0x7fffffffu & src) ^ (sz[s] >> 31)) != 0;
        c.x += odd ? -sc[s].x : sc[s].x;
        c.y += odd ? -sc[s].y : sc[s].y;
      }
      h = cfma(c, psi[rswz(int(src))], h);
    }
    e = cfma_conj(psi[rswz(p)], h, e);
    if (a.grad) del[rswz(p)] = make_double2(2.0 * h.x, 2.0 * h.y);
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
  for (int gi = a.ngroups - 1; gi >= 0; --gi) {
    const RGroup g = groups[gi];
    if (g.kind != RG_PAIR) {
      other_group(g, mat, psi, n, true);
      other_group(g, mat, del, n, true);
      __syncthreads();
      continue;
    }
    const M2 m = dagger(gm[gi]);
    const int sv = rswz(g.v);
    const bool want = g.grad >= 0;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int i0[PAIRS];
    double2 x[PAIRS], y[PAIRS], dx[PAIRS], dy[PAIRS];
#pragma unroll
    for (int k = 0; k < PAIRS; ++k) {
      const int p = insert0(tx + k * T, g.pivot);
      i0[k] = tx + k * T < npairs && controls_on(g, p) ? rswz(p) ^ ((par(g.r & p) ^ g.rc) ? sv : 0) : -1;
      if (i0[k] >= 0) {
        x[k] = psi[i0[k]];
        y[k] = psi[i0[k] ^ sv];
        dx[k] = del[i0[k]];
        dy[k] = del[i0[k] ^ sv];
      }
    }
#pragma unroll
    for (int k = 0; k < PAIRS; ++k)
      if (i0[k] >= 0) {
        if (want) {
          s0 = fma(dx[k].y, x[k].x, fma(-dx[k].x, x[k].y, s0));
          s1 = fma(dy[k].y, y[k].x, fma(-dy[k].x, y[k].y, s1));
          s2 = fma(dx[k].y, y[k].x, fma(-dx[k].x, y[k].y, fma(dy[k].y, x[k].x, fma(-dy[k].x, x[k].y, s2))));
          s3 = fma(dx[k].x, y[k].x, fma(dx[k].y, y[k].y, fma(-dy[k].x, x[k].x, fma(-dy[k].y, x[k].y, s3))));
        }
        apply(m, x[k], y[k]);
        apply(m, dx[k], dy[k]);
        psi[i0[k]] = x[k];
        psi[i0[k] ^ sv] = y[k];
        del[i0[k]] = dx[k];
        del[i0[k] ^ sv] = dy[k];
      }
    if (want) {
      // lane bits 0 and 1 choose the sum a lane keeps
      const bool b0 = tx & 1, b1 = tx & 2;
      const double u0 = (b0 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, b0 ? s0 : s1, 1);
      const double u1 = (b0 ? s3 : s2) + __shfl_xor_sync(0xffffffffu, b0 ? s2 : s3, 1);
      gbuf[row * T + tx] = (b1 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b1 ? u0 : u1, 2);
      ++row;
    }
    __syncthreads();
    if (row == a.chunk) {
      add_rows();
      __syncthreads();
    }
  }
  add_rows();

  double* gs = a.B > 1 ? a.gsample + int64_t(b) * a.nslots : a.gout;
  for (int s = tx; s < a.nslots; s += T) gs[s] = 0.0;
  __syncthreads();
  const double scale = a.B > 1 ? 1.0 : a.weights[0];
  auto gate_gradient = [&](int o) {
    const ROp op = a.ops[o];
    const RGroup g = groups[op.group];
    M2 V = dagger(op_matrix(a.ops[g.op0 + g.nops - 1], cs, a.table));
    for (int k = g.op0 + g.nops - 2; k >= o; --k) V = mul(dagger(op_matrix(a.ops[k], cs, a.table)), V);
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
      const int slot = a.ops[o].slot;
      if (slot >= 0) gs[slot] = gate_gradient(o);
    }
  } else if (tx == 0) {
    for (int o = 0; o < a.nops; ++o) {
      const int slot = a.ops[o].slot;
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
  std::vector<RGroup> groups;
  std::vector<ROp> ops;
  std::vector<RAngle> angles;
  std::vector<int> mats;
  struct Held {
    ROp op;
    RGroup ctl;   // its controls
  };
  std::vector<Held> open[kResMaxBits];
  uint16_t row[kResMaxBits], col[kResMaxBits], rconst = 0;

  uint16_t bit(int t) const { return uint16_t((rconst >> t) & 1); }
  static uint16_t high_bit(unsigned v) { return uint16_t(31 - __builtin_clz(v)); }

  RGroup target(int q) const {
    RGroup g{};
    g.v = col[q];
    g.r = row[q];
    g.rc = bit(q);
    g.pivot = high_bit(col[q]);
    return g;
  }
  void close(int q) {
    if (open[q].empty()) return;
    RGroup g = target(q);
    const RGroup& last = open[q].back().ctl;
    // a controlled gate is a group by itself: its predecessors on the target go before it
    const size_t count = open[q].size() - (last.nctl ? 1 : 0);
    if (count) emit(g, open[q].data(), count);
    if (last.nctl) {
      g.nctl = last.nctl;
      std::memcpy(g.ctl, last.ctl, sizeof(g.ctl));
      g.cbits = last.cbits;
      emit(g, &open[q].back(), 1);
    }
    open[q].clear();
  }
  void emit(RGroup g, const Held* h, size_t count) {
    g.kind = RG_PAIR;
    g.op0 = uint16_t(ops.size());
    g.nops = uint16_t(count);
    g.grad = -1;
    for (size_t i = 0; i < count; ++i) {
      ops.push_back(h[i].op);
      ops.back().group = uint16_t(groups.size());
      if (h[i].op.slot >= 0) g.grad = 0;
    }
    groups.push_back(g);
  }
  void controls(RGroup& g, const int* q, int count) {
    g.nctl = uint16_t(count);
    for (int j = 0; j < count; ++j) {
      g.ctl[j] = row[q[j]];
      g.cbits |= uint16_t(bit(q[j]) << j);
    }
  }
  // A single-target gate: it joins the target's open group; with controls it also ends it, so that
  // later gates on a control cannot be emitted before it.
  void single(ROp op, int t, const int* ctl, int nctl) {
    for (int j = 0; j < nctl; ++j) close(ctl[j]);
    Held h{op, RGroup{}};
    controls(h.ctl, ctl, nctl);
    open[t].push_back(h);
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
    RGroup g = target(o.pos[0]);
    g.grad = -1;
    if (o.cls == CLS_DIAG) {
      g.kind = RG_DIAG;
      int e[32];
      for (int i = 0; i < d; ++i) e[i] = i * (d + 1);
      g.op0 = matrix(o, d, e);
      controls(g, o.pos + 1, o.k - 1);
    } else if (o.k == 2) {
      g.kind = RG_U2;
      int e[16];
      for (int i = 0; i < 16; ++i) e[i] = i;
      g.op0 = matrix(o, 16, e);
      const int q = o.pos[1];
      g.v2 = col[q];
      g.r2 = row[q];
      g.rc2 = bit(q);
      const unsigned w = ((g.v2 >> g.pivot) & 1) ? g.v2 ^ g.v : g.v2;   // v2 without the first pivot
      g.pivot2 = high_bit(w);
    } else {
      return false;
    }
    groups.push_back(g);
    return true;
  }
};

size_t resident_shared(const ResidentPlan& P, int nflips, int nstr, bool grad, int T, int chunk) {
  size_t s = (sizeof(double2) << P.n) * (grad ? 2 : 1);
  s += sizeof(double2) * (size_t(P.ncs) + P.nmat + nstr) + sizeof(M2) * size_t(P.ngroups);
  if (grad) s += sizeof(double) * (size_t(chunk) * T + 4 * size_t(P.ngrad));
  s += sizeof(RGroup) * size_t(P.ngroups);
  s += sizeof(uint32_t) * (size_t(nstr) + 2 * size_t(nflips) + 1);
  return (s + 15) & ~size_t(15);
}

int build_plan(mb_circuit c, ResidentPlan* P) {
  P->n = c->n;
  Builder B;
  B.c = c;
  B.P = P;
  for (int t = 0; t < c->n; ++t) B.row[t] = B.col[t] = uint16_t(1 << t);
  for (const COp& o : c->ops) {
    // 16-bit indexes, and room left in shared memory in any case
    if (B.groups.size() > 4000 || B.ops.size() > 16000 || c->nslots > 32767 || B.angles.size() > 4000 || B.mats.size() > 8000) return MB_OK;
    if (!B.add(o)) return MB_OK;
  }
  for (int q = 0; q < c->n; ++q) B.close(q);
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
  put(B.groups.data(), sizeof(RGroup) * B.groups.size());
  P->off_ops = put(B.ops.data(), sizeof(ROp) * B.ops.size());
  P->off_ang = put(B.angles.data(), sizeof(RAngle) * B.angles.size());
  P->off_mat = put(B.mats.data(), sizeof(int) * B.mats.size());
  if (int rc = dev_alloc(&P->d, h.size())) return rc;
  MB_CHECK_CUDA(cudaMemcpyAsync(P->d, h.data(), h.size(), cudaMemcpyHostToDevice, g_ctx.stream));
  MB_CHECK_CUDA(cudaStreamSynchronize(g_ctx.stream));
  P->ok = true;
  return MB_OK;
}

int resident_threads(int n) { return n <= 6 ? 32 : n <= 10 ? 1 << (n - 1) : kResMaxThreads; }

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
  ObsStrings os;
  if (!observable_strings(o, n, &os) || os.nstr > 1024) return MB_OK;
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
  const int pairs = std::max(1, (1 << (n - 1)) / T);
  // Rows per chunk: 32 KiB of partial cross sums.
  const int chunk = std::max(4, 4096 / T);
  const size_t shm = resident_shared(P, os.nflips, os.nstr, grad != nullptr, T, chunk);
  if (shm > kResMaxShared) return MB_OK;

  // Parameters and weights go up and results come back in one copy each, through pinned memory;
  // the call waits for its results, so the buffers are free again when it returns.
  const size_t up = size_t(c->nslots) + (grad ? size_t(B) : 0);
  const size_t down = 2 * size_t(B) + (grad ? size_t(c->nslots) : 0);
  const size_t rows = grad && B > 1 ? size_t(B) * c->nslots : 0;
  if (int rc = small_reserve(up + down, up + down + rows)) return rc;
  double* hp = g_ctx.h_small;
  double* dp = g_ctx.d_small;
  std::copy(theta, theta + c->nslots, hp);
  if (grad) std::copy(weights, weights + B, hp + c->nslots);
  cudaStream_t st = g_ctx.stream;
  if (up) MB_CHECK_CUDA(cudaMemcpyAsync(dp, hp, sizeof(double) * up, cudaMemcpyHostToDevice, st));

  RArgs a{};
  a.n = n;
  a.grad = grad ? 1 : 0;
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
  a.groups = reinterpret_cast<const RGroup*>(d);
  a.ops = reinterpret_cast<const ROp*>(d + P.off_ops);
  a.angles = reinterpret_cast<const RAngle*>(d + P.off_ang);
  a.mat_off = reinterpret_cast<const int*>(d + P.off_mat);
  a.table = c->d_table;
  a.theta = dp;
  a.weights = dp + c->nslots;
  a.init = init->d;
  a.flips = os.flips;
  a.strings = os.strings;
  double* res = dp + up;
  a.values = reinterpret_cast<double2*>(res + (up & 1));   // 16-byte aligned; small_reserve leaves room
  a.gout = reinterpret_cast<double*>(a.values + B);
  a.gsample = a.gout + c->nslots;
  a.counter = g_ctx.counters;
  auto launch = [&](auto kern) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(shm));
    kern<<<B, T, shm, st>>>(a);
  };
  {
    ProfScope ps("k_resident", 16.0 * double(init->elems) * B, st);
    if (pairs == 1) launch(k_resident<1>);
    else if (pairs == 2) launch(k_resident<2>);
    else launch(k_resident<4>);
  }
  MB_LAUNCHED();
  double* hr = hp + up;
  MB_CHECK_CUDA(cudaMemcpyAsync(hr, a.values, sizeof(double) * down, cudaMemcpyDeviceToHost, st));
  MB_CHECK_CUDA(cudaStreamSynchronize(st));
  std::memcpy(values, hr, sizeof(double2) * B);
  if (grad) std::copy(hr + 2 * size_t(B), hr + down, grad);
  *done = true;
  return MB_OK;
}

}  // namespace mb
