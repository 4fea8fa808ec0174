// Gradient of a k-qubit gate application with respect to the operator:
//   G_s[a, c] = sum_rest g_s[rest | a] * conj(psi_s[rest | c])
// where g = dL/d(out) and (rest | a) is the amplitude whose target bits
// spell matrix index a.  This is torch's convention for out = U @ psi
// (grad_U = grad_out @ psi^H), summed over every non-target qubit.  With a
// shared operator (out_stride == 0) the per-state matrices are summed too.
//
// k <= 4 runs in opgrad_rows_kernel: a thread takes whole groups of 2^k
// amplitudes and sums a few rows of G in registers; for k <= 2 that is all
// of G, and the same read of g also gives the state's gradient U^H g.
// k = 5, 6 run in opgrad_kernel, one block per (state, matrix entry, slice
// of groups).  FP64 partials go to caller scratch when a matrix needs more
// than one block, and a second kernel sums them in a fixed order
// (deterministic, no atomics).
#include "common.cuh"

namespace gbsv {

constexpr int OG_THREADS = 256;

struct OpGradArgs {
  int n, k;
  int64_t num_states;
  int64_t in_stride;   // amplitudes between psi states (0 = broadcast)
  int64_t groups;      // 2^(n-k)
  int parts;
  int64_t part_len;    // groups per part
  int sorted[GBSV_MAX_DENSE_QUBITS];
  int pos[GBSV_MAX_DENSE_QUBITS];
};

__device__ __forceinline__ uint64_t offset_of(const OpGradArgs& a, int idx) {
  uint64_t o = 0;
  for (int j = 0; j < a.k; ++j)
    if ((idx >> (a.k - 1 - j)) & 1) o |= uint64_t(1) << a.pos[j];
  return o;
}

__device__ __forceinline__ double warp_sum_og(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename R>
__global__ void __launch_bounds__(OG_THREADS)
    opgrad_kernel(const Cx<R>* g, const Cx<R>* psi, OpGradArgs a,
                  void* out, int direct, double* partial) {
  const int d = 1 << a.k;
  const int64_t per_state = (int64_t)d * d * a.parts;
  const int64_t s = blockIdx.x / per_state;
  const int64_t rem = blockIdx.x % per_state;
  const int e = (int)(rem / a.parts);
  const int p = (int)(rem % a.parts);
  const int ra = e / d, rc = e % d;
  const uint64_t oa = offset_of(a, ra), oc = offset_of(a, rc);
  const Cx<R>* gs = g + (s << a.n);
  const Cx<R>* ps = psi + s * a.in_stride;
  const int64_t lo = (int64_t)p * a.part_len;
  int64_t hi = lo + a.part_len;
  if (hi > a.groups) hi = a.groups;
  Acc<R> ax, ay;
  for (int64_t t = lo + threadIdx.x; t < hi; t += OG_THREADS) {
    uint64_t base = (uint64_t)t;
    for (int j = 0; j < a.k; ++j) {
      const int q = a.sorted[j];
      base = ((base >> q) << (q + 1)) | (base & ((uint64_t(1) << q) - 1));
    }
    const Cx<R> u = gs[base + oa];
    const Cx<R> v = ps[base + oc];
    // u * conj(v)
    ax.add_prod(u.x, v.x);
    ax.add_prod(u.y, v.y);
    ay.add_prod(u.y, v.x);
    ay.add_prod(-u.x, v.y);
  }
  double x = ax.value(), y = ay.value();
  __shared__ double sx[OG_THREADS / 32], sy[OG_THREADS / 32];
  x = warp_sum_og(x);
  y = warp_sum_og(y);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sx[w] = x;
    sy[w] = y;
  }
  __syncthreads();
  if (w == 0) {
    x = l < OG_THREADS / 32 ? sx[l] : 0.0;
    y = l < OG_THREADS / 32 ? sy[l] : 0.0;
    x = warp_sum_og(x);
    y = warp_sum_og(y);
    if (l == 0) {
      if (direct) {
        Cx<R> r;
        r.x = (R)x;
        r.y = (R)y;
        static_cast<Cx<R>*>(out)[s * d * d + e] = r;
      } else {
        partial[2 * blockIdx.x] = x;
        partial[2 * blockIdx.x + 1] = y;
      }
    }
  }
}

// Halving sum over a warp: V = 2^j values per lane become one value per
// lane group, value v in lanes [32 v / V, 32 (v + 1) / V).
__device__ __forceinline__ void og_combine(Acc<float>& a, float hi,
                                           float lo) {
  const float s = a.hi + hi;
  const float bp = s - a.hi;
  a.lo += lo + ((a.hi - (s - bp)) + (hi - bp));
  a.hi = s;
}
__device__ __forceinline__ Acc<float> og_exchange(const Acc<float>& send,
                                                  int o) {
  Acc<float> r;
  r.hi = __shfl_xor_sync(0xffffffffu, send.hi, o);
  r.lo = __shfl_xor_sync(0xffffffffu, send.lo, o);
  return r;
}
__device__ __forceinline__ Acc<double> og_exchange(const Acc<double>& send,
                                                   int o) {
  Acc<double> r;
  r.s = __shfl_xor_sync(0xffffffffu, send.s, o);
  return r;
}
__device__ __forceinline__ void og_add(Acc<float>& a, const Acc<float>& b) {
  og_combine(a, b.hi, b.lo);
}
__device__ __forceinline__ void og_add(Acc<double>& a, const Acc<double>& b) {
  a.s += b.s;
}
template <typename R, int V>
__device__ __forceinline__ double og_warp_sum(Acc<R>* acc) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int w = V / 2; w > 0; w >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < V / 2; ++j) {
      if (j >= w) continue;
      const Acc<R> send = up ? acc[j] : acc[j + w];
      if (up) acc[j] = acc[j + w];
      og_add(acc[j], og_exchange(send, o));
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) og_add(acc[0], og_exchange(acc[0], o));
  return acc[0].value();
}

struct OgRowArgs {
  int n;
  int lg;              // log2 groups per state (n - k)
  int64_t in_stride;   // amplitudes between psi states (0 = broadcast)
  int per_state;       // a gradient per state (1) or one for all (0)
  uint64_t groups;     // groups of one gradient
  int parts;
  uint64_t part_len;   // groups per part
  int sorted[4];
  int pos[4];
  int64_t op_stride;
};

// Block (run, row block, part): rows [RT * row block, + RT) of gradient
// `run` over one slice of groups.  Each real product enters its sum exactly
// (Acc); about 10 FP32 operations per product and 4 * RT * 2^K products per
// group bound the kernel, so the rows are split only where a thread's sums
// (RT * 2^K complex pairs) leave no registers: k = 1, 2 take all rows, k = 3
// two, k = 4 one.  STATE (all rows, complex64): also gs = U^H g, rounded as
// the gate kernel rounds it.  Two-qubit gate on 5 states of 18 qubits: 27 us
// for the sums (one block per entry, g and psi read four times each) and
// 10 us for the adjoint gate before, 18 us for both here.
template <typename R, int K, int RT, bool STATE>
__global__ void __launch_bounds__(OG_THREADS, 2)
    opgrad_rows_kernel(const Cx<R>* g, const Cx<R>* psi, const Cx<R>* ops,
                       Cx<R>* gs, OgRowArgs a, Cx<R>* out, double* partial) {
  using C = Cx<R>;
  constexpr int D = 1 << K, V = 2 * RT * D, RB = D / RT;
  static_assert(!STATE || RT == D, "the state needs every row");
  const int part = blockIdx.x % a.parts;
  const int rb = (blockIdx.x / a.parts) % RB;
  const uint64_t run = blockIdx.x / ((unsigned)a.parts * RB);
  const uint64_t lo = (uint64_t)part * a.part_len;
  uint64_t hi = lo + a.part_len;
  if (hi > a.groups) hi = a.groups;
  const uint64_t gmask = (uint64_t(1) << a.lg) - 1;
  Acc<R> acc[V];
  C m[STATE ? D * D : 1];
  uint64_t have = ~uint64_t(0);  // state whose operator is in m
  for (uint64_t t = lo + threadIdx.x; t < hi; t += OG_THREADS) {
    const uint64_t s = a.per_state ? run : t >> a.lg;
    uint64_t base = a.per_state ? t : t & gmask;
#pragma unroll
    for (int j = 0; j < K; ++j) base = insert_zero(base, a.sorted[j]);
    const C* gp = g + (s << a.n) + base;
    const C* pp = psi + (int64_t)s * a.in_stride + base;
    C x[D], y[RT];
#pragma unroll
    for (int b = 0; b < D; ++b) {
      uint64_t off = 0;
#pragma unroll
      for (int j = 0; j < K; ++j)
        if ((b >> (K - 1 - j)) & 1) off += uint64_t(1) << a.pos[j];
      x[b] = pp[off];
      if (RT == D) y[b % RT] = gp[off];
    }
    if constexpr (RT < D) {
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        uint64_t off = 0;
#pragma unroll
        for (int j = 0; j < K; ++j)
          if (((rb * RT + r) >> (K - 1 - j)) & 1)
            off += uint64_t(1) << a.pos[j];
        y[r] = gp[off];
      }
    }
    if constexpr (STATE) {
      const uint64_t want = a.op_stride ? s : 0;
      if (want != have) {
#pragma unroll
        for (int j = 0; j < D * D; ++j) {
          m[j] = __ldg(ops + (int64_t)want * a.op_stride + j);
          m[j].y = -m[j].y;
        }
        have = want;
      }
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int c = 0; c < D; ++c) {  // y[r] * conj(x[c])
        Acc<R>&re = acc[2 * (r * D + c)], &im = acc[2 * (r * D + c) + 1];
        re.add_prod(y[r].x, x[c].x);
        re.add_prod(y[r].y, x[c].y);
        im.add_prod(y[r].y, x[c].x);
        im.add_prod(-y[r].x, x[c].y);
      }
    if constexpr (STATE) {
      C* dst = gs + (s << a.n) + base;
#pragma unroll
      for (int c = 0; c < D; ++c) {
        C o = cmul(m[c], y[0]);
#pragma unroll
        for (int r = 1; r < D; ++r) o = cmad(m[r * D + c], y[r], o);
        uint64_t off = 0;
#pragma unroll
        for (int j = 0; j < K; ++j)
          if ((c >> (K - 1 - j)) & 1) off += uint64_t(1) << a.pos[j];
        __stcs(dst + off, o);
      }
    }
  }
  const double v = og_warp_sum<R, V>(acc);
  __shared__ double red[OG_THREADS / 32][V];
  constexpr int LPV = 32 / V;  // lanes per value
  if ((threadIdx.x & 31) % LPV == 0)
    red[threadIdx.x >> 5][(threadIdx.x & 31) / LPV] = v;
  __syncthreads();
  if (threadIdx.x >= V) return;
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < OG_THREADS / 32; ++w) t += red[w][threadIdx.x];
  // entry of the matrix, and its real or imaginary part
  const int e = rb * RT * D + (threadIdx.x >> 1);
  if (partial)
    partial[2 * ((run * (D * D) + e) * a.parts + part) + (threadIdx.x & 1)] =
        t;
  else
    reinterpret_cast<R*>(out)[2 * (run * (D * D) + e) + (threadIdx.x & 1)] =
        (R)t;
}

// One block per (output matrix m, entry e): sum the partials in order.
template <typename R>
__global__ void __launch_bounds__(OG_THREADS)
    opgrad_finalize(const double* partial, int64_t num_states, int d2,
                    int parts, int shared, void* out) {
  const int64_t m = blockIdx.x / d2;
  const int e = blockIdx.x % d2;
  const int64_t s_lo = shared ? 0 : m;
  const int64_t s_hi = shared ? num_states : m + 1;
  const int64_t count = (s_hi - s_lo) * parts;
  double x = 0.0, y = 0.0;
  for (int64_t t = threadIdx.x; t < count; t += OG_THREADS) {
    const int64_t s = s_lo + t / parts;
    const int p = (int)(t % parts);
    const int64_t idx = (s * d2 + e) * parts + p;
    x += partial[2 * idx];
    y += partial[2 * idx + 1];
  }
  __shared__ double sx[OG_THREADS / 32], sy[OG_THREADS / 32];
  x = warp_sum_og(x);
  y = warp_sum_og(y);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sx[w] = x;
    sy[w] = y;
  }
  __syncthreads();
  if (w == 0) {
    x = l < OG_THREADS / 32 ? sx[l] : 0.0;
    y = l < OG_THREADS / 32 ? sy[l] : 0.0;
    x = warp_sum_og(x);
    y = warp_sum_og(y);
    if (l == 0) {
      Cx<R> r;
      r.x = (R)x;
      r.y = (R)y;
      static_cast<Cx<R>*>(out)[m * d2 + e] = r;
    }
  }
}

struct OgPlan {
  int parts;
  int64_t part_len;
  bool direct;
};

static OgPlan og_plan(int64_t num_states, int n, int k, bool shared) {
  OgPlan p{1, int64_t(1) << (n - k), true};
  const int64_t groups = int64_t(1) << (n - k);
  const int64_t d2 = int64_t(1) << (2 * k);
  const int64_t blocks = num_states * d2;
  const int64_t want = (int64_t)sm_count() * 4;
  if (blocks < want && groups > 4096) {
    int64_t parts = (want + blocks - 1) / blocks;
    const int64_t max_parts = (groups + 4095) / 4096;
    if (parts > max_parts) parts = max_parts;
    if (parts > 1) {
      p.part_len = (groups + parts - 1) / parts;
      p.parts = (int)((groups + p.part_len - 1) / p.part_len);
    }
  }
  p.direct = (p.parts == 1) && !(shared && num_states > 1);
  return p;
}

// k <= 4: gradients are runs of groups; each is cut into parts of at least
// 512 groups (2 per thread) until the chip has four blocks per SM.
constexpr int OG_ROWS_MAX = 4;

static OgPlan og_rows_plan(int64_t num_states, int n, int k, bool shared) {
  const int64_t runs = shared ? 1 : num_states;
  const int64_t groups = (shared ? num_states : 1) << (n - k);
  const int rows = k == 3 ? 4 : k == 4 ? 16 : 1;  // row blocks
  OgPlan p{1, groups, true};
  const int64_t want = (int64_t)sm_count() * 4;
  int64_t parts = (want + runs * rows - 1) / (runs * rows);
  const int64_t most = (groups + 511) / 512;
  if (parts > most) parts = most;
  if (parts > 1) {
    p.part_len = (groups + parts - 1) / parts;
    p.parts = (int)((groups + p.part_len - 1) / p.part_len);
  }
  p.direct = p.parts == 1;
  return p;
}

static size_t og_scratch(const OgPlan& p, int64_t runs, int k) {
  return p.direct ? 0
                  : (size_t)runs * ((size_t)1 << (2 * k)) * p.parts * 2 *
                        sizeof(double);
}

template <typename R>
static int og_rows(const void* g, const void* psi, const void* ops,
                   void* grad_state, int k, int64_t runs, const OgRowArgs& a,
                   void* out, double* partial, cudaStream_t st) {
  using C = Cx<R>;
  const C* gp = static_cast<const C*>(g);
  const C* pp = static_cast<const C*>(psi);
  const C* mp = static_cast<const C*>(ops);
  C* sp = static_cast<C*>(grad_state);
  C* op = static_cast<C*>(out);
  const uint64_t blocks =
      (uint64_t)runs * a.parts * (k == 3 ? 4 : k == 4 ? 16 : 1);
  if (blocks > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "grid too large");
#define OG_ROWS(K, RT, S)                                               \
  opgrad_rows_kernel<R, K, RT, S><<<(unsigned)blocks, OG_THREADS, 0, st>>>( \
      gp, pp, mp, sp, a, op, partial)
  if (k == 1) {
    if (sizeof(R) == 4 && sp) OG_ROWS(1, 2, sizeof(R) == 4);
    else OG_ROWS(1, 2, false);
  } else if (k == 2) {
    if (sizeof(R) == 4 && sp) OG_ROWS(2, 4, sizeof(R) == 4);
    else OG_ROWS(2, 4, false);
  } else if (k == 3) {
    OG_ROWS(3, 2, false);
  } else {
    OG_ROWS(4, 1, false);
  }
#undef OG_ROWS
  return after_launch("opgrad_rows_kernel");
}

}  // namespace gbsv

using namespace gbsv;

extern "C" size_t gbsv_operator_grad_scratch_bytes(int64_t num_states, int n,
                                                   int k, int shared) {
  if (n < 0 || k < 0 || k > n || k > GBSV_MAX_DENSE_QUBITS || num_states <= 0)
    return 0;
  if (k >= 1 && k <= OG_ROWS_MAX)
    return og_scratch(og_rows_plan(num_states, n, k, shared != 0),
                      shared ? 1 : num_states, k);
  return og_scratch(og_plan(num_states, n, k, shared != 0), num_states, k);
}

extern "C" int gbsv_operator_grad(const void* grad_out, const void* state_in,
                                  int dtype, int num_qubits,
                                  int64_t num_states, int64_t in_stride,
                                  const int32_t* qubits, int num_targets,
                                  void* grad_ops, int shared, void* scratch,
                                  size_t scratch_bytes, void* stream) {
  return gbsv_apply_operator_grad(grad_out, state_in, dtype, num_qubits,
                                  num_states, in_stride, nullptr, 0, qubits,
                                  num_targets, nullptr, grad_ops, shared,
                                  scratch, scratch_bytes, stream);
}

extern "C" int gbsv_apply_operator_grad(
    const void* grad_out, const void* state_in, int dtype, int num_qubits,
    int64_t num_states, int64_t in_stride, const void* ops, int64_t op_stride,
    const int32_t* qubits, int num_targets, void* grad_state, void* grad_ops,
    int shared, void* scratch, size_t scratch_bytes, void* stream) {
  if (dtype != GBSV_C64 && dtype != GBSV_C128)
    return set_error(GBSV_ERR_INVALID_ARG, "state dtype must be complex");
  const int n = num_qubits, k = num_targets;
  if (n < 0 || n > 62 || k < 0 || k > n)
    return set_error(GBSV_ERR_INVALID_ARG, "bad qubit counts n=%d k=%d", n, k);
  if (k > 6)
    return set_error(GBSV_ERR_UNSUPPORTED,
                     "operator gradients for more than 6 qubits");
  if (num_states < 0 || in_stride < 0)
    return set_error(GBSV_ERR_INVALID_ARG, "negative size or stride");
  if (num_states == 0) return GBSV_OK;
  if (!grad_out || !state_in || !grad_ops || (k > 0 && !qubits))
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  if (grad_state && (dtype != GBSV_C64 || k < 1 || k > 2))
    return set_error(GBSV_ERR_UNSUPPORTED,
                     "the state's gradient comes with complex64 operators on "
                     "1 or 2 qubits");
  if (grad_state && (!ops || op_stride < 0))
    return set_error(GBSV_ERR_INVALID_ARG, "bad operators");
  OpGradArgs a{};
  a.n = n;
  a.k = k;
  a.num_states = num_states;
  a.in_stride = in_stride;
  a.groups = int64_t(1) << (n - k);
  uint64_t seen = 0;
  for (int j = 0; j < k; ++j) {
    const int q = qubits[j];
    if (q < 0 || q >= n || ((seen >> q) & 1))
      return set_error(GBSV_ERR_INVALID_ARG, "bad or repeated qubit %d", q);
    seen |= uint64_t(1) << q;
    a.pos[j] = n - 1 - q;
    a.sorted[j] = a.pos[j];
  }
  for (int i = 1; i < k; ++i)
    for (int j = i; j > 0 && a.sorted[j - 1] > a.sorted[j]; --j) {
      const int t = a.sorted[j];
      a.sorted[j] = a.sorted[j - 1];
      a.sorted[j - 1] = t;
    }
  if (k >= 1 && k <= OG_ROWS_MAX) {
    const OgPlan p = og_rows_plan(num_states, n, k, shared != 0);
    const int64_t runs = shared ? 1 : num_states;
    const size_t need = og_scratch(p, runs, k);
    if (need && (!scratch || scratch_bytes < need))
      return set_error(GBSV_ERR_SCRATCH,
                       "operator gradient needs %zu scratch bytes", need);
    OgRowArgs r{};
    r.n = n;
    r.lg = n - k;
    r.in_stride = in_stride;
    r.per_state = !shared;
    r.groups = (uint64_t)(shared ? num_states : 1) << (n - k);
    r.parts = p.parts;
    r.part_len = (uint64_t)p.part_len;
    r.op_stride = op_stride;
    for (int j = 0; j < k; ++j) {
      r.sorted[j] = a.sorted[j];
      r.pos[j] = a.pos[j];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    double* partial = p.direct ? nullptr : static_cast<double*>(scratch);
    int rc = dtype == GBSV_C64
                 ? og_rows<float>(grad_out, state_in, ops, grad_state, k,
                                  runs, r, grad_ops, partial, st)
                 : og_rows<double>(grad_out, state_in, ops, grad_state, k,
                                   runs, r, grad_ops, partial, st);
    if (rc || p.direct) return rc;
    const int d2 = 1 << (2 * k);
    const unsigned fb = (unsigned)(runs * d2);
    if (dtype == GBSV_C64)
      opgrad_finalize<float><<<fb, OG_THREADS, 0, st>>>(partial, runs, d2,
                                                        p.parts, 0, grad_ops);
    else
      opgrad_finalize<double><<<fb, OG_THREADS, 0, st>>>(
          partial, runs, d2, p.parts, 0, grad_ops);
    return after_launch("opgrad_finalize");
  }
  const OgPlan p = og_plan(num_states, n, k, shared != 0);
  a.parts = p.parts;
  a.part_len = p.part_len;
  const int d2 = 1 << (2 * k);
  const uint64_t blocks = (uint64_t)num_states * d2 * p.parts;
  if (blocks > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "grid too large");
  if (!p.direct) {
    const size_t need = (size_t)blocks * 2 * sizeof(double);
    if (!scratch || scratch_bytes < need)
      return set_error(GBSV_ERR_SCRATCH,
                       "operator gradient needs %zu scratch bytes", need);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double* partial = static_cast<double*>(scratch);
  if (dtype == GBSV_C64)
    opgrad_kernel<float><<<(unsigned)blocks, OG_THREADS, 0, st>>>(
        static_cast<const float2*>(grad_out),
        static_cast<const float2*>(state_in), a, grad_ops, p.direct, partial);
  else
    opgrad_kernel<double><<<(unsigned)blocks, OG_THREADS, 0, st>>>(
        static_cast<const double2*>(grad_out),
        static_cast<const double2*>(state_in), a, grad_ops, p.direct,
        partial);
  int rc = after_launch("opgrad_kernel");
  if (rc || p.direct) return rc;
  const int64_t outs = shared ? 1 : num_states;
  const unsigned fblocks = (unsigned)(outs * d2);
  if (dtype == GBSV_C64)
    opgrad_finalize<float><<<fblocks, OG_THREADS, 0, st>>>(
        partial, num_states, d2, p.parts, shared, grad_ops);
  else
    opgrad_finalize<double><<<fblocks, OG_THREADS, 0, st>>>(
        partial, num_states, d2, p.parts, shared, grad_ops);
  return after_launch("opgrad_finalize");
}
