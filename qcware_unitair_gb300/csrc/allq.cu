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

__device__ __forceinline__ AqOp aq_load_op(const float2* ops,
                                           const AllqArgs& a, int bit) {
  const int pos = bit < a.cl ? bit : a.p + (bit - a.cl);
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

// All 16 amplitudes finite: where one is not, the products with zeros that
// the structured forms leave out would be NaN, so the full form runs.
__device__ __forceinline__ bool aq_finite(const float2* r) {
  uint32_t e = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i)
    e = max(e, max(__float_as_uint(r[i].x) & 0x7fffffffu,
                   __float_as_uint(r[i].y) & 0x7fffffffu));
  return e < 0x7f800000u;
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

// The operators of tile bits LO .. HI in the layout with registers RB ..
template <int RB, int LO, int HI>
__device__ __forceinline__ void aq_round(float2* r, const float2* ops,
                                         const AllqArgs& a) {
  AqOp o = aq_load_op(ops, a, HI);
  const bool finite = aq_finite(r);
#pragma unroll
  for (int b = HI; b >= LO; --b) {
    if (!((a.mask >> b) & 1)) continue;
    if (a.op_qstride) o = aq_load_op(ops, a, b);
    const int kind = finite ? o.kind : AQ_FULL;
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

// One pass.  256 threads hold the CTA's 4096 amplitudes, 16 each, with four
// tile bits on a thread's registers: four operators cost no data movement,
// and between the (at most three) register layouts the tile goes through
// 32 KB of shared memory.  M = min(n, 12): below 12 qubits the CTA holds
// 2^(12 - M) whole states.  A tile is read before any of it is written and
// tiles are disjoint, so in place is safe.
//
// Bound: the FMA pipe (4 or 8 FMAs per amplitude and operator at the 66% of
// its rate that three distinct operands allow) about as much as HBM, so the
// bits are split for few passes, not for little arithmetic.  One layer on
// 256 states of 16 qubits (134 MB): 16 passes of the gate kernel 655 us,
// two passes here 165 us (HBM alone 80 us); on 7 states of 20 qubits 315 us
// before, 65 us here.
template <int M>
__global__ void __launch_bounds__(AQ_THREADS, 3)
    allq_kernel(const float2* in, float2* out, const float2* ops,
                AllqArgs a) {
  using W = AqRounds<M>;
  __shared__ float2 sm[1 << AQ_TILE];
  const int sub = threadIdx.x >> (M - 4);
  const int u = threadIdx.x & ((1 << (M - 4)) - 1);
  float2* const S = sm + (sub << M);
  uint64_t base;
  const uint64_t s = aq_place<M>(a, blockIdx.x, sub, &base);
  const bool live = M == AQ_TILE || s < (uint64_t)a.num_states;
  const float2* const src = in + (int64_t)s * a.in_stride + base;
  float2* const dst = out + (s << a.n) + base;
  if (live) ops += (int64_t)s * a.op_stride;

  float2 r[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    r[i] = make_float2(0.f, 0.f);
    if (live) r[i] = __ldcs(src + aq_offset(a, aq_index<W::R0>(u, i)));
  }
  aq_round<W::R0, W::R0, M - 1>(r, ops, a);

  // exchange: registers of layout A out, registers of layout B in.  Each
  // thread writes the slots it read last, so one barrier is enough.
#define AQ_PUT(A)                                                    \
  _Pragma("unroll") for (int i = 0; i < 16; ++i)                     \
      S[aq_swz(aq_index<A>(u, i))] = r[i];                           \
  __syncthreads();
#define AQ_GET(B)                                                    \
  _Pragma("unroll") for (int i = 0; i < 16; ++i) r[i] =              \
      S[aq_swz(aq_index<B>(u, i))];
  int at = 0;  // which layout the registers are in
  if constexpr (W::R1 >= 0) {
    if (aq_any<W::R1, W::R0 - 1>(a.mask)) {
      AQ_PUT(W::R0)
      AQ_GET(W::R1)
      aq_round<W::R1, W::R1, W::R0 - 1>(r, ops, a);
      at = 1;
    }
  }
  if constexpr (W::R2 >= 0) {
    if (aq_any<0, W::R1 - 1>(a.mask)) {
      if (at == 1) {
        AQ_PUT(W::R1)
      } else {
        AQ_PUT(W::R0)
      }
      AQ_GET(W::R2)
      aq_round<W::R2, 0, W::R1 - 1>(r, ops, a);
      at = 2;
    }
  }
  // Store from the layout that writes long runs: the first layout's (and
  // for 12 tile bits the second's, runs of 128 bytes).
  if constexpr (W::R1 >= 0) {
    if (W::R1 >= 4 && at == 1) {
      if (live) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          __stcs(dst + aq_offset(a, aq_index<W::R1>(u, i)), r[i]);
      }
      return;
    }
    if (at == 1) {
      AQ_PUT(W::R1)
      AQ_GET(W::R0)
    }
  }
  if constexpr (W::R2 >= 0) {
    if (at == 2) {
      AQ_PUT(W::R2)
      AQ_GET(W::R0)
    }
  }
  if (live) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      __stcs(dst + aq_offset(a, aq_index<W::R0>(u, i)), r[i]);
  }
}
#undef AQ_PUT
#undef AQ_GET

// The passes of an n-qubit state: up to 8 of the bits above the lowest 12
// at a time (the tile's other bits are the lowest ones, so every pass moves
// contiguous runs of at least 16 amplitudes), last the lowest min(n, 12).
// Qubit 0, the top bit, comes first, so every amplitude sees the operators
// in the order of a loop over the qubits and rounds as it would there.
static int aq_passes(int n) {
  return n <= AQ_TILE ? 1 : 1 + (n - AQ_TILE + AQ_HIGH - 1) / AQ_HIGH;
}

static void aq_pass(AllqArgs* a, int pass) {
  const int m = std::min(a->n, AQ_TILE);
  const int up = aq_passes(a->n) - 1 - pass;  // passes below this one
  if (up == 0) {
    a->cl = a->p = m;
    a->mask = (1u << m) - 1;
    return;
  }
  const int p = AQ_TILE + (up - 1) * AQ_HIGH;
  const int h = std::min(AQ_HIGH, a->n - p);
  a->cl = AQ_TILE - h;
  a->p = p;
  a->mask = ((1u << h) - 1) << a->cl;
}

static int aq_launch(const float2* in, float2* out, const float2* ops,
                     const AllqArgs& a, cudaStream_t st) {
  const int m = std::min(a.n, AQ_TILE);
  const uint64_t tiles = a.n >= AQ_TILE
                             ? (uint64_t)a.num_states << (a.n - AQ_TILE)
                             : ((uint64_t)a.num_states +
                                (uint64_t(1) << (AQ_TILE - m)) - 1) >>
                                   (AQ_TILE - m);
  if (tiles > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "grid too large (%llu blocks)",
                     (unsigned long long)tiles);
#define AQ_CASE(MM)                                                       \
  case MM:                                                                \
    allq_kernel<MM><<<(unsigned)tiles, AQ_THREADS, 0, st>>>(in, out, ops, \
                                                            a);           \
    break;
  switch (m) {
    AQ_CASE(4) AQ_CASE(5) AQ_CASE(6) AQ_CASE(7) AQ_CASE(8) AQ_CASE(9)
    AQ_CASE(10) AQ_CASE(11) AQ_CASE(12)
    default: return set_error(GBSV_ERR_INVALID_ARG, "bad tile size %d", m);
  }
#undef AQ_CASE
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
    aq_pass(&a, pass);
    a.in_stride = pass == 0 ? in_stride : int64_t(1) << n;
    const int rc =
        aq_launch(static_cast<const float2*>(pass == 0 ? in : out),
                  static_cast<float2*>(out), static_cast<const float2*>(ops),
                  a, st);
    if (rc) return rc;
  }
  return GBSV_OK;
}

}  // namespace gbsv
