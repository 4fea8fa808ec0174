// A 2x2 operator on every qubit of each state (apply_all_qubits and its
// per-qubit form) and its gradient.
//
// unitair loops over the qubits, one einsum with two permuted copies each
// (src/unitair/simulation/operations.py:332-413).  The operators act on
// different qubits, so they commute and many of them can share one read and
// write of the state: a pass takes a tile of 2^12 amplitudes, applies the
// operators of up to 12 of its index bits, and writes it back.
#include <algorithm>

#include "common.cuh"

namespace gbsv {

constexpr int AQ_THREADS = 256;
constexpr int AQ_TILE = 12;   // log2 amplitudes a CTA holds
constexpr int AQ_HIGH = 8;    // most tile bits above the contiguous run

struct AllqArgs {
  int n;
  int64_t num_states;
  int64_t in_stride;   // amplitudes between input states (0 = broadcast)
  int64_t op_stride;   // complex elements between states' operators
  int64_t op_qstride;  // between qubits' operators (0 = one for all)
  int cl;              // tile bits 0 .. cl - 1 are index bits 0 .. cl - 1,
  int p;               // tile bits cl .. are index bits p ..
  uint32_t mask;       // tile bits whose qubit this pass applies
};

// Tile index of register i of thread u when the registers are tile bits
// RB .. RB + 3.
template <int RB>
__device__ __forceinline__ int aq_index(int u, int i) {
  return (u & ((1 << RB) - 1)) | (i << RB) | ((u >> RB) << (RB + 4));
}
// Shared-memory slot of a tile index: the low four bits (the 8-byte bank of
// a half warp's access) XOR the next four, so that every register layout
// reads and writes without bank conflicts.
__device__ __forceinline__ int aq_swz(int l) { return l ^ ((l >> 4) & 15); }

// The register layouts of a tile of 2^M amplitudes: registers on tile bits
// R0 .. R0 + 3 (the top four), then R1 .., then 0 ..; -1 where the bits are
// used up.  A layout applies the bits that no earlier one has.
template <int M> struct AqRounds {
  static constexpr int R0 = M - 4;
  static constexpr int R1 = M >= 8 ? M - 8 : M > 4 ? 0 : -1;
  static constexpr int R2 = M > 8 ? 0 : -1;
};

// The operator of one qubit.  Most layers are rotations, whose entries are
// real or imaginary in a fixed pattern; leaving out the products with the
// zero parts halves the FMAs, which bound the kernel.
struct AqOp {
  float2 m[4];
  int kind;
};
constexpr int AQ_FULL = 0, AQ_REAL = 1, AQ_RX = 2, AQ_DIAG = 3;

// The operator of amplitude-index bit pos.
__device__ __forceinline__ AqOp aq_load_op(const float2* ops,
                                           const AllqArgs& a, int pos) {
  const float2* o = ops + (int64_t)(a.n - 1 - pos) * a.op_qstride;
  AqOp r;
#pragma unroll
  for (int j = 0; j < 4; ++j) r.m[j] = __ldg(o + j);
  const bool re0 = r.m[0].y == 0 && r.m[3].y == 0;
  if (re0 && r.m[1].y == 0 && r.m[2].y == 0) r.kind = AQ_REAL;
  else if (re0 && r.m[1].x == 0 && r.m[2].x == 0) r.kind = AQ_RX;
  else if (r.m[1].x == 0 && r.m[1].y == 0 && r.m[2].x == 0 && r.m[2].y == 0)
    r.kind = AQ_DIAG;
  else r.kind = AQ_FULL;
  return r;
}

// Whether all 16 amplitudes stay finite through a layout.  Where one is not,
// or a sum overflows, the products with zeros that the structured forms leave
// out are NaN in a loop of gates, so the full form runs.  Four operators with
// entries up to 2^26 make at most (4 * 2^26)^4 = 2^112 of the largest
// component, so below 2^16 nothing reaches 2^128.  (A look at the entries, or
// one before each operator, costs registers this kernel does not have: layers
// of full matrices 81 -> 85 us on 7 states of 20 qubits, 11.3 -> 12.6 us on
// 1000 of 10.)
__device__ __forceinline__ bool aq_bounded(const float2* r) {
  float e = 0.f;  // largest |component|; NaN stays
#pragma unroll
  for (int i = 0; i < 16; ++i)
    asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(e) : "f"(r[i].x), "f"(r[i].y));
  return e < 0x1p16f;
}

// m * a, rounded as the gate kernels' products are.
__device__ __forceinline__ float2 aq_mul(float2 m, float2 a) {
  return make_float2(fmaf(m.x, a.x, -(m.y * a.y)),
                     fmaf(m.x, a.y, m.y * a.x));
}

// The 2x2 on register bit B of 16 amplitudes.
template <int B>
__device__ __forceinline__ void aq_apply(float2* r, const AqOp& o,
                                         int kind) {
  constexpr int H = 1 << B;
  if (kind == AQ_REAL) {
    const float m0 = o.m[0].x, m1 = o.m[1].x, m2 = o.m[2].x, m3 = o.m[3].x;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i & H) continue;
      const float2 a0 = r[i], a1 = r[i | H];
      r[i].x = fmaf(m1, a1.x, m0 * a0.x);
      r[i].y = fmaf(m1, a1.y, m0 * a0.y);
      r[i | H].x = fmaf(m3, a1.x, m2 * a0.x);
      r[i | H].y = fmaf(m3, a1.y, m2 * a0.y);
    }
  } else if (kind == AQ_RX) {  // real diagonal, imaginary off-diagonal
    const float m0 = o.m[0].x, m1 = o.m[1].y, m2 = o.m[2].y, m3 = o.m[3].x;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i & H) continue;
      const float2 a0 = r[i], a1 = r[i | H];
      r[i].x = fmaf(-m1, a1.y, m0 * a0.x);
      r[i].y = fmaf(m1, a1.x, m0 * a0.y);
      r[i | H].x = fmaf(m3, a1.x, -(m2 * a0.y));
      r[i | H].y = fmaf(m3, a1.y, m2 * a0.x);
    }
  } else if (kind == AQ_DIAG) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i & H)  // rounded as cmad onto m2 * a0 = 0 rounds
        r[i] = make_float2(fmaf(-o.m[3].y, r[i].y, o.m[3].x * r[i].x),
                           fmaf(o.m[3].y, r[i].x, o.m[3].x * r[i].y));
      else
        r[i] = aq_mul(o.m[0], r[i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (i & H) continue;
      const float2 a0 = r[i], a1 = r[i | H];
      r[i] = cmad(o.m[1], a1, aq_mul(o.m[0], a0));
      r[i | H] = cmad(o.m[3], a1, aq_mul(o.m[2], a0));
    }
  }
}

__device__ __forceinline__ int aq_pos(const AllqArgs& a, int bit) {
  return bit < a.cl ? bit : a.p + (bit - a.cl);
}

// The operators of tile bits LO .. HI in the layout with registers RB ..
template <int RB, int LO, int HI>
__device__ __forceinline__ void aq_round(float2* r, const float2* ops,
                                         const AllqArgs& a) {
  AqOp o = aq_load_op(ops, a, aq_pos(a, HI));
  const bool bounded = aq_bounded(r);
#pragma unroll
  for (int b = HI; b >= LO; --b) {
    if (!((a.mask >> b) & 1)) continue;
    if (a.op_qstride) o = aq_load_op(ops, a, aq_pos(a, b));
    const int kind = bounded ? o.kind : AQ_FULL;
    if (b - RB == 0) aq_apply<0>(r, o, kind);
    else if (b - RB == 1) aq_apply<1>(r, o, kind);
    else if (b - RB == 2) aq_apply<2>(r, o, kind);
    else aq_apply<3>(r, o, kind);
  }
}

template <int LO, int HI>
__device__ __forceinline__ bool aq_any(uint32_t mask) {
  return (mask & (((2u << HI) - 1) & ~((1u << LO) - 1))) != 0;
}

// Where a CTA's tile sits: tile (or, for M < 12, states of 2^M amplitudes)
// `tile`; returns the state and sets the index of its first amplitude.
template <int M>
__device__ __forceinline__ uint64_t aq_place(const AllqArgs& a, uint64_t tile,
                                             int sub, uint64_t* base) {
  if constexpr (M == AQ_TILE) {
    const int lt = a.n - AQ_TILE;
    const uint64_t rest = tile & ((uint64_t(1) << lt) - 1);
    const uint64_t mid = rest & ((uint64_t(1) << (a.p - a.cl)) - 1);
    const uint64_t hi = rest >> (a.p - a.cl);
    *base = (mid << a.cl) | (hi << (a.p + AQ_TILE - a.cl));
    return tile >> lt;
  } else {
    *base = 0;
    return (tile << (AQ_TILE - M)) + sub;
  }
}

__device__ __forceinline__ uint64_t aq_offset(const AllqArgs& a, int l) {
  return (uint64_t)(l & ((1 << a.cl) - 1)) + ((uint64_t)(l >> a.cl) << a.p);
}

// The layouts a pass runs through, from the top tile bits down.
struct AqPlan {
  int m;           // log2 amplitudes of a tile (min(n, 12))
  int rounds;
  int rb[3];       // layout k: registers on tile bits rb[k] .. rb[k] + 3,
  int bits[3];     // applies these of the four (mask), which are the
  int pos[3];      // amplitude-index bits pos[k] ..
  int64_t lstride; // amplitudes between a thread's registers: first layout,
  int64_t sstride; // last layout where it stores directly, 0 where the tile
                   // goes back to the first layout for the store
  uint32_t slot[3][16];  // byte offset of register i's slot part, layout k
};

// One pass.  256 threads hold the CTA's 4096 amplitudes, 16 each, with four
// tile bits on a thread's registers: four operators cost no data movement,
// and between the (at most three) register layouts the tile goes through
// 32 KB of shared memory.  Below 12 qubits (m < 12) the CTA holds
// 2^(12 - m) whole states.  A tile is read before any of it is written and
// tiles are disjoint, so in place is safe.
//
// Bound: instruction issue (4 or 8 FMAs per amplitude and operator) about
// as much as HBM, so the layouts share one copy of the operator code (three
// copies missed the instruction cache: 2.6 of 9 stall cycles per issue) and
// every global address is a base plus i strides.  One layer on 256 states
// of 16 qubits (134 MB): 16 passes of the gate kernel 655 us, two passes
// with a kernel per tile size and unrolled layouts 165 us, here 108 us (HBM
// alone 80 us); on 7 states of 20 qubits 315, 66 and 54 us, 145 and 78 us
// where the operator has no zero part.  Two-lane FMAs, which halve the FMA
// instructions, were no faster: the lanes of a complex product cross, and
// the moves cost what the FMAs gave.
__global__ void __launch_bounds__(AQ_THREADS, 4)
    allq_kernel(const float2* in, float2* out, const float2* ops,
                const __grid_constant__ AllqArgs a,
                const __grid_constant__ AqPlan w) {
  __shared__ float2 sm[1 << AQ_TILE];
  __shared__ AqOp sop[AQ_TILE];  // of tile bit b, where the CTA has one state
  const int sub = threadIdx.x >> (w.m - 4);
  const int u = threadIdx.x & ((1 << (w.m - 4)) - 1);
  uint64_t base, s;
  bool live = true;
  if (w.m == AQ_TILE) {
    s = aq_place<AQ_TILE>(a, blockIdx.x, sub, &base);
  } else {
    base = 0;
    s = ((uint64_t)blockIdx.x << (AQ_TILE - w.m)) + sub;
    live = s < (uint64_t)a.num_states;
  }
  const uint64_t first = base + aq_offset(a, u);
  if (live) ops += (int64_t)s * a.op_stride;

  float2 r[16];
  if (live) {
    const float2* src = in + (int64_t)s * a.in_stride + first;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      r[i] = __ldcs(src);
      src += w.lstride;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = make_float2(0.f, 0.f);
  }
  // One load and one look at an operator's kind per CTA instead of one per
  // thread and layout, behind the amplitudes' loads: 16 qubits x 256 with an
  // operator per qubit 126 -> 108 us.  Smaller states have too many
  // operators in a CTA for that.
  const bool staged = w.m == AQ_TILE;
  if (staged) {
    if (threadIdx.x < AQ_TILE && ((a.mask >> threadIdx.x) & 1))
      sop[threadIdx.x] = aq_load_op(ops, a, aq_pos(a, threadIdx.x));
    __syncthreads();
  }
  // byte offset of the slot of tile index (thread part) | (register part):
  // the swizzle is linear over XOR
  auto slot = [&](int rb) {
    const int lo = (1 << rb) - 1;
    return (uint32_t)((sub << w.m) + aq_swz((u & lo) | ((u & ~lo) << 4))) * 8;
  };
  auto at_slot = [&](uint32_t off) -> float2& {
    return *reinterpret_cast<float2*>(reinterpret_cast<char*>(sm) + off);
  };
#pragma unroll 1
  for (int k = 0;; ++k) {
    const int bits = w.bits[k];
    AqOp o;
    if (!staged) o = aq_load_op(ops, a, w.pos[k]);
    const bool bounded = aq_bounded(r);
#define AQ_BIT(J)                                                      \
  if ((bits >> J) & 1) {                                               \
    if (staged) o = sop[w.rb[k] + J];                                  \
    else if (a.op_qstride) o = aq_load_op(ops, a, w.pos[k] + J);       \
    aq_apply<J>(r, o, bounded ? o.kind : AQ_FULL);                      \
  }
    AQ_BIT(3)
    AQ_BIT(2)
    AQ_BIT(1)
    AQ_BIT(0)
#undef AQ_BIT
    const bool last = k + 1 == w.rounds;
    if (last && (k == 0 || w.sstride)) break;
    // to the next layout, or back to the first for the store.  Each thread
    // writes the slots it read last, so one barrier is enough.
    uint32_t at = slot(w.rb[k]);
#pragma unroll
    for (int i = 0; i < 16; ++i) at_slot(at ^ w.slot[k][i]) = r[i];
    __syncthreads();
    const int to = last ? 0 : k + 1;
    at = slot(w.rb[to]);
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = at_slot(at ^ w.slot[to][i]);
    if (last) break;
  }
  if (!live) return;
  float2* dst = out + (s << a.n) + first;
  int64_t step = w.lstride;
  if (w.sstride && w.rounds > 1) {  // the second layout's own addresses
    dst = out + (s << a.n) + base +
          aq_offset(a, (u & 15) | ((u & ~15) << 4));
    step = w.sstride;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    __stcs(dst, r[i]);
    dst += step;
  }
}

// The passes of an n-qubit state: up to 8 of the bits above the lowest 12
// at a time, last the lowest min(n, 12).  A pass over high bits has four or
// eight neighbouring ones in its tile (some of them perhaps not to be
// applied) beside the lowest 8 or 4, so that registers are a fixed stride
// apart and every access moves runs of at least 16 amplitudes.  Qubit 0, the
// top bit, comes first, so every amplitude sees the operators in the order
// of a loop over the qubits and rounds as it would there.
static int aq_passes(int n) {
  return n <= AQ_TILE ? 1 : 1 + (n - AQ_TILE + AQ_HIGH - 1) / AQ_HIGH;
}

static void aq_slots(AqPlan* w) {
  for (int k = 0; k < w->rounds; ++k)
    for (int i = 0; i < 16; ++i) {
      const int l = i << w->rb[k];
      w->slot[k][i] = (uint32_t)(l ^ ((l >> 4) & 15)) * 8;
    }
}

static AqPlan aq_pass(AllqArgs* a, int pass) {
  const int m = std::min(a->n, AQ_TILE);
  AqPlan w{};
  w.m = m;
  w.rb[0] = m - 4;
  const int up = aq_passes(a->n) - 1 - pass;  // passes below this one
  if (up == 0) {
    a->cl = a->p = m;
    a->mask = (1u << m) - 1;
    w.lstride = int64_t(1) << (m - 4);
    int done = m;  // tile bits from here up are applied
    for (w.rounds = 0; done > 0; ++w.rounds) {
      const int rb = std::max(done - 4, 0);
      w.rb[w.rounds] = w.pos[w.rounds] = rb;
      w.bits[w.rounds] = (1 << (done - rb)) - 1;
      done = rb;
    }
    aq_slots(&w);
    return w;
  }
  const int low = AQ_TILE + (up - 1) * AQ_HIGH;
  const int h = std::min(AQ_HIGH, a->n - low);  // bits to apply
  const int t = h <= 4 ? 4 : 8;                 // bits in the tile
  a->cl = AQ_TILE - t;
  a->p = low + h - t;
  a->mask = ((1u << h) - 1) << (AQ_TILE - h);
  w.pos[0] = a->p + t - 4;
  w.bits[0] = (a->mask >> 8) & 15;
  w.lstride = int64_t(1) << w.pos[0];
  w.rounds = 1;
  if (t == 8) {
    w.rounds = 2;
    w.rb[1] = 4;
    w.pos[1] = a->p;
    w.bits[1] = (a->mask >> 4) & 15;
    w.sstride = int64_t(1) << a->p;
  }
  aq_slots(&w);
  return w;
}

static int aq_launch(const float2* in, float2* out, const float2* ops,
                     const AllqArgs& a, const AqPlan& w, cudaStream_t st) {
  const uint64_t tiles = a.n >= AQ_TILE
                             ? (uint64_t)a.num_states << (a.n - AQ_TILE)
                             : ((uint64_t)a.num_states +
                                (uint64_t(1) << (AQ_TILE - w.m)) - 1) >>
                                   (AQ_TILE - w.m);
  if (tiles > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "grid too large (%llu blocks)",
                     (unsigned long long)tiles);
  allq_kernel<<<(unsigned)tiles, AQ_THREADS, 0, st>>>(in, out, ops, a, w);
  return after_launch("allq_kernel");
}

// complex64, n >= 4.
int apply_all_fused(const void* in, void* out, int n, int64_t num_states,
                    int64_t in_stride, const void* ops, int64_t op_stride,
                    int64_t op_qstride, cudaStream_t st) {
  AllqArgs a{};
  a.n = n;
  a.num_states = num_states;
  a.op_stride = op_stride;
  a.op_qstride = op_qstride;
  for (int pass = 0; pass < aq_passes(n); ++pass) {
    const AqPlan w = aq_pass(&a, pass);
    a.in_stride = pass == 0 ? in_stride : int64_t(1) << n;
    const int rc =
        aq_launch(static_cast<const float2*>(pass == 0 ? in : out),
                  static_cast<float2*>(out), static_cast<const float2*>(ops),
                  a, w, st);
    if (rc) return rc;
  }
  return GBSV_OK;
}


// ------------------------------------------------------------- gradient --
// Gradient of a pass: for out = (prod_q U_q) psi and g = dL/d(out),
//   dL/dU_q[a, c] = sum_rest g_q[rest | a] * conj(psi_q[rest | c])
// where, because the U commute, psi_q may be psi with any of the other
// operators applied as long as g_q has the adjoints of the rest.  A CTA
// runs the layouts upwards on psi, keeping psi before each in shared
// memory, and downwards on g; inside a layout it takes the bits from the
// top, with the lower bits' operators applied to a fresh copy of psi and
// the upper bits' adjoints already applied to g.  One read of psi and g and
// one write of dL/dpsi per pass, where a loop over the qubits would save or
// recompute a state per qubit.
//
// Sums: a thread's products enter a float pair exactly (Acc<float>), pairs
// meet across a warp with TwoSum and everything beyond a warp is FP64, in a
// fixed order.  That accumulation bounds the kernel (about 10 FP32
// operations per real product, 16 products per pair and operator).
//
// One autograd node and three or four launches take the place of a node,
// an adjoint gate, a gradient kernel, its sum and an accumulation per
// qubit: a QAOA step (16 states of 14 qubits, 3 layers, forward and
// backward) went from 9.3 to 3.2 ms, most of it host time before and after.
struct AllqGradArgs {
  AllqArgs f;
  int chunk_log;   // log2 tiles of one state that a CTA walks (12 tile bits)
  int store;       // write dL/dpsi
  double* partial; // [state][qubit][chunk][8]: re, im of the four entries
};

__device__ __forceinline__ AqOp aq_dagger(const AqOp& o) {
  AqOp d;
  d.m[0] = make_float2(o.m[0].x, -o.m[0].y);
  d.m[1] = make_float2(o.m[2].x, -o.m[2].y);
  d.m[2] = make_float2(o.m[1].x, -o.m[1].y);
  d.m[3] = make_float2(o.m[3].x, -o.m[3].y);
  d.kind = o.kind;
  return d;
}

__device__ __forceinline__ void aq_pair_add(float& hi, float& lo, float oh,
                                            float ol) {
  const float s = hi + oh;
  const float bp = s - hi;
  lo += ol + ((hi - (s - bp)) + (oh - bp));
  hi = s;
}

// Sums eight pairs over the warp by halving: after three exchanges a lane
// keeps one value, two more finish it.  Lane 4 k holds value k's bits in
// reverse order of the exchanges; *v is the value this lane ends with.
__device__ __forceinline__ float2 aq_warp_sum8(Acc<float>* acc, int* v) {
  const int lane = threadIdx.x & 31;
  float h[8], l[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    h[j] = acc[j].hi;
    l[j] = acc[j].lo;
  }
#pragma unroll
  for (int w = 4, o = 16; w > 0; w >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j >= w) continue;
      const float sh = up ? h[j] : h[j + w], sl = up ? l[j] : l[j + w];
      h[j] = up ? h[j + w] : h[j];
      l[j] = up ? l[j + w] : l[j];
      aq_pair_add(h[j], l[j], __shfl_xor_sync(0xffffffffu, sh, o),
                  __shfl_xor_sync(0xffffffffu, sl, o));
    }
  }
#pragma unroll
  for (int o = 2; o > 0; o >>= 1)
    aq_pair_add(h[0], l[0], __shfl_xor_sync(0xffffffffu, h[0], o),
                __shfl_xor_sync(0xffffffffu, l[0], o));
  *v = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
  return make_float2(h[0], l[0]);
}

// g0 conj(x0), g0 conj(x1), g1 conj(x0), g1 conj(x1) over the pairs of
// register bit B
template <int B>
__device__ __forceinline__ void aq_outer(const float2* g, const float2* x,
                                         Acc<float>* acc) {
  constexpr int H = 1 << B;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (i & H) continue;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 u = g[i | (e & 2 ? H : 0)], v = x[i | (e & 1 ? H : 0)];
      acc[2 * e].add_prod(u.x, v.x);
      acc[2 * e].add_prod(u.y, v.y);
      acc[2 * e + 1].add_prod(u.y, v.x);
      acc[2 * e + 1].add_prod(-u.x, v.y);
    }
  }
}

// One layout of the gradient: registers RB .. RB + 3, tile bits LO .. HI,
// psi before the layout in S (this thread's slots are its own).
template <int RB, int LO, int HI>
__device__ __forceinline__ void aq_grad_round(float2* g, const float2* S,
                                              int u, const float2* ops,
                                              const AllqArgs& a,
                                              float2* wred) {
#pragma unroll 1
  for (int b = HI; b >= LO; --b) {
    if (!((a.mask >> b) & 1)) continue;
    float2 x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = S[aq_swz(aq_index<RB>(u, i))];
    const bool bounded = aq_bounded(x);
#pragma unroll
    for (int c = LO; c < HI; ++c) {
      if (c >= b || !((a.mask >> c) & 1)) continue;
      const AqOp o = aq_load_op(ops, a, aq_pos(a, c));
      const int kind = bounded ? o.kind : AQ_FULL;
      if (c - RB == 0) aq_apply<0>(x, o, kind);
      else if (c - RB == 1) aq_apply<1>(x, o, kind);
      else aq_apply<2>(x, o, kind);
    }
    const AqOp d = aq_dagger(aq_load_op(ops, a, aq_pos(a, b)));
    const int kind = aq_bounded(g) ? d.kind : AQ_FULL;
    Acc<float> acc[8];
    switch (b - RB) {
      case 0: aq_outer<0>(g, x, acc); aq_apply<0>(g, d, kind); break;
      case 1: aq_outer<1>(g, x, acc); aq_apply<1>(g, d, kind); break;
      case 2: aq_outer<2>(g, x, acc); aq_apply<2>(g, d, kind); break;
      default: aq_outer<3>(g, x, acc); aq_apply<3>(g, d, kind); break;
    }
    int v;
    const float2 sum = aq_warp_sum8(acc, &v);
    if ((threadIdx.x & 3) == 0)
      wred[(b * (AQ_THREADS / 32) + (threadIdx.x >> 5)) * 8 + v] = sum;
  }
}

constexpr size_t AQ_GRAD_SMEM =
    (3 * (size_t(1) << AQ_TILE) + AQ_TILE * (AQ_THREADS / 32) * 8) *
    sizeof(float2);

// M = min(n, 12) >= 9, so that a warp's amplitudes belong to one state.
template <int M>
__global__ void __launch_bounds__(AQ_THREADS, 2)
    allq_grad_kernel(const float2* psi, const float2* gin, float2* gout,
                     const float2* ops, AllqGradArgs ga) {
  using W = AqRounds<M>;
  const AllqArgs& a = ga.f;
  constexpr int R0 = W::R0, R1 = W::R1;
  extern __shared__ __align__(16) float2 aq_sm[];
  float2* const wred = aq_sm + 3 * (1 << AQ_TILE);
  const int sub = threadIdx.x >> (M - 4);
  const int u = threadIdx.x & ((1 << (M - 4)) - 1);
  float2* const SA = aq_sm + (sub << M);
  float2* const SB = SA + (1 << AQ_TILE);
  float2* const SC = SB + (1 << AQ_TILE);
  const bool act1 = aq_any<R1, R0 - 1>(a.mask);
  bool act2 = false;
  if constexpr (M > 8) act2 = R1 > 0 && aq_any<0, (R1 > 0 ? R1 - 1 : 0)>(a.mask);

#define AQ_PUT(S, r, A)                                              \
  _Pragma("unroll") for (int i = 0; i < 16; ++i)                     \
      S[aq_swz(aq_index<A>(u, i))] = r[i];                           \
  __syncthreads();
#define AQ_GET(S, r, B)                                              \
  _Pragma("unroll") for (int i = 0; i < 16; ++i) r[i] =              \
      S[aq_swz(aq_index<B>(u, i))];

  const int walk = M == AQ_TILE ? 1 << ga.chunk_log : 1;
  double total = 0.0;  // M = 12: value threadIdx.x & 7 of bit threadIdx.x / 8
  uint64_t s = 0;
  for (int w = 0; w < walk; ++w) {
    uint64_t base;
    s = aq_place<M>(a, (uint64_t)blockIdx.x * walk + w, sub, &base);
    const bool live = M == AQ_TILE || s < (uint64_t)a.num_states;
    const float2* const xs = psi + (int64_t)s * a.in_stride + base;
    const float2* const gs = gin + (s << a.n) + base;
    const float2* const so = ops + (live ? (int64_t)s * a.op_stride : 0);
    {
      float2 r[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        r[i] = make_float2(0.f, 0.f);
        if (live) r[i] = __ldcs(xs + aq_offset(a, aq_index<R0>(u, i)));
      }
      float2* const first = act2 ? SA : act1 ? SB : SC;
      AQ_PUT(first, r, R0)
      if (act2) {
        if constexpr (W::R2 >= 0) {
          AQ_GET(SA, r, 0)
          aq_round<0, 0, (R1 > 0 ? R1 - 1 : 0)>(r, so, a);
          float2* const to = act1 ? SB : SC;
          AQ_PUT(to, r, 0)
        }
      }
      if (act1) {
        AQ_GET(SB, r, R1)
        aq_round<R1, R1, R0 - 1>(r, so, a);
        AQ_PUT(SC, r, R1)
      }
    }
    float2 g[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      g[i] = make_float2(0.f, 0.f);
      if (live) g[i] = __ldcs(gs + aq_offset(a, aq_index<R0>(u, i)));
    }
    aq_grad_round<R0, R0, M - 1>(g, SC, u, so, a, wred);
    int at = 0;
    if (act1) {
      AQ_PUT(SC, g, R0)
      AQ_GET(SC, g, R1)
      aq_grad_round<R1, R1, R0 - 1>(g, SB, u, so, a, wred);
      at = 1;
    }
    if (act2) {
      if constexpr (W::R2 >= 0) {
        if (act1) {
          AQ_PUT(SB, g, R1)
          AQ_GET(SB, g, 0)
        } else {
          AQ_PUT(SC, g, R0)
          AQ_GET(SC, g, 0)
        }
        aq_grad_round<0, 0, (R1 > 0 ? R1 - 1 : 0)>(g, SA, u, so, a, wred);
        at = 2;
      }
    }
    if (ga.store) {
      float2* const dst = gout + (s << a.n) + base;
      if (at == 2) {
        AQ_PUT(SA, g, 0)
        AQ_GET(SA, g, R0)
      } else if (at == 1) {
        AQ_PUT(SB, g, R1)
        AQ_GET(SB, g, R0)
      }
      if (live) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          __stcs(dst + aq_offset(a, aq_index<R0>(u, i)), g[i]);
      }
    }
    __syncthreads();  // wred complete, and the slots free for the next tile
    if constexpr (M == AQ_TILE) {
      const int b = threadIdx.x >> 3, v = threadIdx.x & 7;
      if (b < M && ((a.mask >> b) & 1))
        for (int k = 0; k < AQ_THREADS / 32; ++k) {
          const float2 p = wred[(b * (AQ_THREADS / 32) + k) * 8 + v];
          total += (double)p.x + (double)p.y;
        }
      if (w + 1 < walk) __syncthreads();
    }
  }
#undef AQ_PUT
#undef AQ_GET
  if constexpr (M == AQ_TILE) {
    const int b = threadIdx.x >> 3, v = threadIdx.x & 7;
    if (b < M && ((a.mask >> b) & 1)) {
      const int pos = b < a.cl ? b : a.p + (b - a.cl);
      const int nch = a.n - AQ_TILE - ga.chunk_log;  // log2 chunks
      const uint64_t ch = blockIdx.x & ((uint64_t(1) << nch) - 1);
      ga.partial[((((s * a.n + (a.n - 1 - pos)) << nch) + ch) << 3) + v] =
          total;
    }
  } else {
    constexpr int SUBS = 1 << (AQ_TILE - M), WPS = (AQ_THREADS / 32) / SUBS;
    for (int i = threadIdx.x; i < SUBS * M * 8; i += AQ_THREADS) {
      const int v = i & 7, b = (i >> 3) % M, k = (i >> 3) / M;
      const uint64_t st = ((uint64_t)blockIdx.x << (AQ_TILE - M)) + k;
      if (st >= (uint64_t)a.num_states) continue;
      double t = 0.0;
      for (int w = 0; w < WPS; ++w) {
        const float2 p = wred[(b * (AQ_THREADS / 32) + k * WPS + w) * 8 + v];
        t += (double)p.x + (double)p.y;
      }
      ga.partial[((st * a.n + (a.n - 1 - b)) << 3) + v] = t;
    }
  }
}

// Sums runs of `len` items of eight doubles, starting at run * len: block
// (run, part) sums items part, part + parts, ... ; with out != null (parts
// == 1) the four complex sums go to out[4 run ..], else to next[run * parts
// + part].
__global__ void __launch_bounds__(AQ_THREADS)
    allq_grad_sum_kernel(const double* items, uint64_t len, int parts,
                         double* next, float2* out) {
  const uint64_t run = blockIdx.x / parts;
  const int part = blockIdx.x % parts;
  const int v = threadIdx.x & 7, lane = threadIdx.x >> 3;
  double t = 0.0;
  for (uint64_t i = part + (uint64_t)lane * parts; i < len;
       i += (uint64_t)parts * (AQ_THREADS / 8))
    t += items[((run * len + i) << 3) + v];
  __shared__ double red[AQ_THREADS];
  red[threadIdx.x] = t;
  __syncthreads();
  if (lane) return;
  t = 0.0;
  for (int k = 0; k < AQ_THREADS / 8; ++k) t += red[8 * k + v];
  if (out)
    reinterpret_cast<float*>(out)[(run << 3) + v] = (float)t;
  else
    next[((run * parts + part) << 3) + v] = t;
}

struct AqGradPlan {
  int chunk_log;      // tiles a CTA walks
  uint64_t items;     // [state][qubit][chunk] partials of eight doubles
  uint64_t runs, len; // gradients and the items of each
  int parts;          // second-level partials per gradient (1: none)
};

// Gradients are per (state, qubit), (state), (qubit) or one; items of one
// gradient are contiguous except for (qubit) summed over the states, where
// each state is a run of its own first (see the caller).
static AqGradPlan aq_grad_plan(int64_t num_states, int n, bool shared,
                               bool each) {
  AqGradPlan p{};
  const int lt = n > AQ_TILE ? n - AQ_TILE : 0;
  // at most 512 partials per state and qubit
  p.chunk_log = lt > 9 ? lt - 9 : 0;
  const uint64_t chunks = uint64_t(1) << (lt - p.chunk_log);
  p.items = (uint64_t)num_states * n * chunks;
  if (shared && !each) {
    p.runs = 1;
    p.len = p.items;
  } else if (!shared && !each) {
    p.runs = (uint64_t)num_states;
    p.len = n * chunks;
  } else {
    p.runs = (uint64_t)num_states * n;
    p.len = chunks;
  }
  const uint64_t parts = (p.len + 4095) / 4096;
  p.parts = (int)std::min<uint64_t>(parts, 256);
  return p;
}

// Sums over states of [state][qubit] gradients: one thread per value.
__global__ void allq_grad_states_kernel(const double* items,
                                        uint64_t num_states, int values,
                                        float* out) {
  const int v = blockIdx.x;
  double t = 0.0;
  for (uint64_t s = threadIdx.x; s < num_states; s += blockDim.x)
    t += items[s * values + v];
  __shared__ double red[AQ_THREADS];
  red[threadIdx.x] = t;
  __syncthreads();
  for (int o = AQ_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[v] = (float)red[0];
}

static size_t aq_grad_scratch(const AqGradPlan& p, int64_t num_states, int n,
                              bool shared, bool each) {
  uint64_t items = p.items;
  if (p.parts > 1) items += p.runs * p.parts;
  if (shared && each) items += (uint64_t)num_states * n;
  return items * 8 * sizeof(double);
}

template <int M>
static int aq_grad_launch(const float2* psi, const float2* gin, float2* gout,
                          const float2* ops, const AllqGradArgs& ga,
                          uint64_t ctas, cudaStream_t st) {
  static OncePerDevice once;
  const int rc = allow_smem(once, allq_grad_kernel<M>, (int)AQ_GRAD_SMEM,
                            "allq_grad_kernel");
  if (rc) return rc;
  allq_grad_kernel<M><<<(unsigned)ctas, AQ_THREADS, AQ_GRAD_SMEM, st>>>(
      psi, gin, gout, ops, ga);
  return after_launch("allq_grad_kernel");
}

}  // namespace gbsv

using namespace gbsv;

extern "C" int gbsv_all_qubits_passes(int dtype, int num_qubits) {
  return dtype == GBSV_C64 && num_qubits >= 9 && num_qubits <= 62
             ? aq_passes(num_qubits)
             : 0;
}

static int aq_check(int dtype, int n, int64_t num_states, int64_t in_stride,
                    int64_t op_stride, int64_t op_qubit_stride) {
  if (gbsv_all_qubits_passes(dtype, n) == 0)
    return set_error(GBSV_ERR_UNSUPPORTED,
                     "needs complex64 states of 9 qubits or more");
  if (num_states < 0 || in_stride < 0 || op_stride < 0 || op_qubit_stride < 0)
    return set_error(GBSV_ERR_INVALID_ARG, "negative size or stride");
  return GBSV_OK;
}

extern "C" int gbsv_apply_all_qubits_passes(
    const void* state_in, void* const* pass_out, int dtype, int num_qubits,
    int64_t num_states, int64_t in_stride, const void* ops, int64_t op_stride,
    int64_t op_qubit_stride, void* stream) {
  int rc = aq_check(dtype, num_qubits, num_states, in_stride, op_stride,
                    op_qubit_stride);
  if (rc || num_states == 0) return rc;
  const int np = aq_passes(num_qubits);
  if (!state_in || !ops || !pass_out)
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  for (int i = 0; i < np; ++i)
    if (!pass_out[i]) return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  AllqArgs a{};
  a.n = num_qubits;
  a.num_states = num_states;
  a.op_stride = op_stride;
  a.op_qstride = op_qubit_stride;
  const void* src = state_in;
  for (int i = 0; i < np; ++i) {
    const AqPlan w = aq_pass(&a, i);
    a.in_stride = i == 0 ? in_stride : int64_t(1) << num_qubits;
    rc = aq_launch(static_cast<const float2*>(src),
                   static_cast<float2*>(pass_out[i]),
                   static_cast<const float2*>(ops), a, w,
                   static_cast<cudaStream_t>(stream));
    if (rc) return rc;
    src = pass_out[i];
  }
  return GBSV_OK;
}

extern "C" size_t gbsv_all_qubits_grad_scratch_bytes(int64_t num_states,
                                                     int num_qubits,
                                                     int shared, int each) {
  if (num_states <= 0 || gbsv_all_qubits_passes(GBSV_C64, num_qubits) == 0)
    return 0;
  return aq_grad_scratch(
      aq_grad_plan(num_states, num_qubits, shared != 0, each != 0),
      num_states, num_qubits, shared != 0, each != 0);
}

extern "C" int gbsv_apply_all_qubits_grad(
    const void* grad_out, const void* const* pass_in, int dtype,
    int num_qubits, int64_t num_states, int64_t in_stride, const void* ops,
    int64_t op_stride, int64_t op_qubit_stride, void* grad_state,
    int need_state, void* grad_ops, int shared, void* scratch,
    size_t scratch_bytes, void* stream) {
  int rc = aq_check(dtype, num_qubits, num_states, in_stride, op_stride,
                    op_qubit_stride);
  if (rc || num_states == 0) return rc;
  const int n = num_qubits, np = aq_passes(n);
  const bool each = op_qubit_stride != 0;
  if (!grad_out || !ops || !grad_ops || !pass_in ||
      ((need_state || np > 1) && !grad_state))
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  for (int i = 0; i < np; ++i)
    if (!pass_in[i]) return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  const AqGradPlan p = aq_grad_plan(num_states, n, shared != 0, each);
  const size_t need = aq_grad_scratch(p, num_states, n, shared != 0, each);
  if (!scratch || scratch_bytes < need || (uintptr_t)scratch % 16)
    return set_error(GBSV_ERR_SCRATCH,
                     "all-qubit gradient needs %zu aligned scratch bytes",
                     need);
  const uint64_t ctas =
      n >= AQ_TILE
          ? (uint64_t)num_states << (n - AQ_TILE - p.chunk_log)
          : ((uint64_t)num_states + (uint64_t(1) << (AQ_TILE - n)) - 1) >>
                (AQ_TILE - n);
  if (ctas > 0x7fffffffull || p.runs * p.parts > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "grid too large");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  AllqGradArgs ga{};
  ga.f.n = n;
  ga.f.num_states = num_states;
  ga.f.op_stride = op_stride;
  ga.f.op_qstride = op_qubit_stride;
  ga.chunk_log = p.chunk_log;
  ga.partial = static_cast<double*>(scratch);
  const float2* m = static_cast<const float2*>(ops);
  float2* gs = static_cast<float2*>(grad_state);
  for (int i = np - 1; i >= 0; --i) {
    aq_pass(&ga.f, i);
    ga.f.in_stride = i == 0 ? in_stride : int64_t(1) << n;
    ga.store = i > 0 || need_state;
    const float2* x = static_cast<const float2*>(pass_in[i]);
    const float2* gi =
        i == np - 1 ? static_cast<const float2*>(grad_out) : gs;
    switch (std::min(n, AQ_TILE)) {
      case 9: rc = aq_grad_launch<9>(x, gi, gs, m, ga, ctas, st); break;
      case 10: rc = aq_grad_launch<10>(x, gi, gs, m, ga, ctas, st); break;
      case 11: rc = aq_grad_launch<11>(x, gi, gs, m, ga, ctas, st); break;
      default: rc = aq_grad_launch<12>(x, gi, gs, m, ga, ctas, st); break;
    }
    if (rc) return rc;
  }
  // sums: chunks (and qubits, states) of each gradient, in a fixed order
  const double* items = ga.partial;
  double* next = ga.partial + p.items * 8;
  uint64_t len = p.len;
  if (p.parts > 1) {
    allq_grad_sum_kernel<<<(unsigned)(p.runs * p.parts), AQ_THREADS, 0, st>>>(
        items, len, p.parts, next, nullptr);
    rc = after_launch("allq_grad_sum_kernel");
    if (rc) return rc;
    items = next;
    len = p.parts;
    next += p.runs * p.parts * 8;
  }
  const bool states = shared && each;
  allq_grad_sum_kernel<<<(unsigned)p.runs, AQ_THREADS, 0, st>>>(
      items, len, 1, next, states ? nullptr : static_cast<float2*>(grad_ops));
  rc = after_launch("allq_grad_sum_kernel");
  if (rc || !states) return rc;
  allq_grad_states_kernel<<<(unsigned)(n * 8), AQ_THREADS, 0, st>>>(
      next, (uint64_t)num_states, n * 8, static_cast<float*>(grad_ops));
  return after_launch("allq_grad_states_kernel");
}
