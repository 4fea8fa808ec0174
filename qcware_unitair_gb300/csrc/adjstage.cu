// Fused backward stages of the adjoint method in registers.
//
// Same contract as the shared-memory stages of adjoint.cu (tiles of psi and
// lambda, the circuit's gates in reverse, one read and write of each state
// per stage), which walk both tiles once per rotation with a block barrier
// and a warp reduction each.  Here the host groups a stage's ops into
// layouts of RB tile bits (gbsv_adjoint_layouts): a thread holds the 2^RB
// amplitudes of psi and of lambda along those bits and runs all of the
// layout's ops on them; the tiles go through shared memory once per layout.
// Diagonal ops on other bits are a per-thread factor, sign-only ones (CZ, Z)
// a mask of signs.  unitair has no counterpart: torch autograd keeps every
// intermediate state of its gates
// (src/unitair/simulation/operations.py:45-148).
#include <algorithm>

#include "common.cuh"

namespace gbsv {

using AdjRegOp = gbsv_adjoint_regop_t;
using AdjLayout = gbsv_adjoint_layout_t;
static_assert(sizeof(AdjRegOp) == 64 && sizeof(AdjLayout) == 32, "");

enum {
  // 0 .. 11: rotation X / Y / Z (type / 4) on register bit type % 4
  AR_RZ_TILE = 12,  // Z rotation on tile bit t[0] of the thread index
  AR_RZ_OUT = 13,   // on position o[0] outside the tile
  AR_SIGN = 14,     // -1 on registers `signs` where tile bits t[0] are set
  AR_DIAG = 15,     // fixed diagonal on nq qubits
  AR_DENSE1 = 16,   // 2x2 on k[0], nq == 2: qubit 1 controls
  AR_DENSE2 = 17,   // 4x4 on k[0] (MSB), k[1]
  AR_END = 18       // end of a layout
};

constexpr int AR_MAX_BITS = 12;
// gradient sums a CTA collects before reducing them: 16 KB
template <typename R> constexpr int AR_BATCH = 64 / (int)sizeof(R);

struct AdjRegArgs {
  int n, m, c;
  int hpos[AR_MAX_BITS];  // position of tile bit c + j
  int spos[AR_MAX_BITS];  // tile positions, ascending
  const AdjRegOp* ops;
  int num_ops;
  const AdjLayout* layouts;
  int num_layouts;
  const double* angles;   // (cos, sin) of theta / 2: [state][total][2]
  int64_t total_slots;
  int64_t slot0;          // this stage's first slot
  int num_slots;
  double* partial;        // [slot of this stage][tile]
  uint64_t tiles;
};

// Slot of a tile index: its low bits XOR the next two groups of as many
// (four 8-byte or three 16-byte bank bits).  With one thread bit of each
// residue in the low lanes, every layout's accesses are conflict-free.
template <typename R>
__device__ __forceinline__ int ar_swz(int l) {
  if constexpr (sizeof(R) == 4)
    return l ^ (((l >> 4) ^ (l >> 8)) & 15);
  else
    return l ^ (((l >> 3) ^ (l >> 6) ^ (l >> 9)) & 7);
}

template <typename R>
__device__ __forceinline__ R ar_neg(R v, uint32_t bit31);
template <>
__device__ __forceinline__ float ar_neg<float>(float v, uint32_t s) {
  return __uint_as_float(__float_as_uint(v) ^ s);
}
template <>
__device__ __forceinline__ double ar_neg<double>(double v, uint32_t s) {
  return __hiloint2double(__double2hiint(v) ^ (int)s, __double2loint(v));
}

// Rotation GEN on register bit K: adds Im <lambda|P|psi> over the thread's
// pairs to g (two chains), then uncomputes both with cos I + i sin P.
template <typename R, int NR, int GEN, int K>
__device__ __forceinline__ R ar_rot(Cx<R>* x, Cx<R>* l, R c, R s) {
  constexpr int H = 1 << K;
  R g[2] = {0, 0};
  int turn = 0;
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    if (i & H) continue;
    const Cx<R> x0 = x[i], x1 = x[i | H], l0 = l[i], l1 = l[i | H];
    R& a = g[turn & 1];
    ++turn;
    if constexpr (GEN == 0) {
      a = fma(l0.x, x1.y, a);
      a = fma(-l0.y, x1.x, a);
      a = fma(l1.x, x0.y, a);
      a = fma(-l1.y, x0.x, a);
      x[i].x = c * x0.x - s * x1.y; x[i].y = c * x0.y + s * x1.x;
      x[i | H].x = c * x1.x - s * x0.y; x[i | H].y = c * x1.y + s * x0.x;
      l[i].x = c * l0.x - s * l1.y; l[i].y = c * l0.y + s * l1.x;
      l[i | H].x = c * l1.x - s * l0.y; l[i | H].y = c * l1.y + s * l0.x;
    } else if constexpr (GEN == 1) {
      a = fma(l1.x, x0.x, a);
      a = fma(l1.y, x0.y, a);
      a = fma(-l0.x, x1.x, a);
      a = fma(-l0.y, x1.y, a);
      x[i].x = c * x0.x + s * x1.x; x[i].y = c * x0.y + s * x1.y;
      x[i | H].x = c * x1.x - s * x0.x; x[i | H].y = c * x1.y - s * x0.y;
      l[i].x = c * l0.x + s * l1.x; l[i].y = c * l0.y + s * l1.y;
      l[i | H].x = c * l1.x - s * l0.x; l[i | H].y = c * l1.y - s * l0.y;
    } else {
      a = fma(l0.x, x0.y, a);
      a = fma(-l0.y, x0.x, a);
      a = fma(-l1.x, x1.y, a);
      a = fma(l1.y, x1.x, a);
      x[i].x = c * x0.x - s * x0.y; x[i].y = c * x0.y + s * x0.x;
      x[i | H].x = c * x1.x + s * x1.y; x[i | H].y = c * x1.y - s * x1.x;
      l[i].x = c * l0.x - s * l0.y; l[i].y = c * l0.y + s * l0.x;
      l[i | H].x = c * l1.x + s * l1.y; l[i | H].y = c * l1.y - s * l1.x;
    }
  }
  return g[0] + g[1];
}

// Registers whose register bit k is set.
__device__ __forceinline__ uint32_t ar_regs(int k) {
  return k == 0 ? 0xAAAAu : k == 1 ? 0xCCCCu : k == 2 ? 0xF0F0u : 0xFF00u;
}

// Sums the buffered per-thread gradients buf[0 .. cnt) over the CTA, a warp
// each: float pairs for complex64 (TwoSum), FP64 beyond.
template <typename R>
__device__ __forceinline__ void ar_reduce(const R* buf, const int* slots,
                                          int cnt, const AdjRegArgs& a) {
  const int T = blockDim.x, warps = T >> 5;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int b = w; b < cnt; b += warps) {
    Acc<R> s;
    for (int j = lane; j < T; j += 32) s.add(buf[b * T + j]);
    double t;
    if constexpr (sizeof(R) == 4) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, s.hi, o);
        const float ol = __shfl_xor_sync(0xffffffffu, s.lo, o);
        s.add(oh);
        s.lo += ol;
      }
      t = s.value();
    } else {
      t = s.s;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (lane == 0)
      a.partial[(uint64_t)slots[b] * a.tiles + blockIdx.x] = t;
  }
}

// Ops of a stage kept in shared memory (more are read from global memory).
constexpr int AR_OPS = 128;

// One CTA per tile, 2^(m - RB) threads.  Bound by instruction issue (about
// 170 instructions per thread and rotation of 16 amplitudes of each state)
// and by the instruction cache, so only the rotations are unrolled per
// register bit; signs are monomials of bits (one test each), and fixed dense
// gates go through the thread's own slots.  Four register bits for
// complex64, three for complex128, are what two states leave of 128
// registers at two CTAs of 256 threads per SM.  32 states of 16 qubits, 24
// rotations and 16 CZ: 120 us in the shared-memory stage, 85 us with every
// op unrolled and one test per sign entry, 59 us here (HBM: 10 us).
template <typename R, int RB>
__global__ void __launch_bounds__(256, 2)
    adjoint_reg_kernel(Cx<R>* psi, Cx<R>* lam, const Cx<R>* pool,
                       const __grid_constant__ AdjRegArgs a) {
  using C = Cx<R>;
  constexpr int NR = 1 << RB;
  extern __shared__ __align__(16) unsigned char ar_sm[];
  const int M = 1 << a.m, T = blockDim.x, tid = threadIdx.x;
  C* const SP = reinterpret_cast<C*>(ar_sm);
  C* const SL = SP + M;
  R* const buf = reinterpret_cast<R*>(SL + M);      // [AR_BATCH][T]
  R* const csn = buf + AR_BATCH<R> * T;             // (cos, sin) per slot
  __shared__ __align__(16) AdjRegOp sops[AR_OPS];
  __shared__ int slots[AR_BATCH<R>];
  __shared__ uint64_t ioff[NR];  // offset of tile index T i
  const uint64_t tps = uint64_t(1) << (a.n - a.m);
  const uint64_t s = blockIdx.x / tps;
  uint64_t base = blockIdx.x % tps;
  for (int j = 0; j < a.m; ++j) base = insert_zero(base, a.spos[j]);
  auto offset = [&](int l) {
    uint64_t off = (uint64_t)(l & ((1 << a.c) - 1));
    const int r = l >> a.c;
    for (int j = 0; j < a.m - a.c; ++j)
      if ((r >> j) & 1) off += uint64_t(1) << a.hpos[j];
    return off;
  };
  if (tid < NR) ioff[tid] = offset(T * tid);
  const bool staged = a.num_ops <= AR_OPS;
  if (staged)
    for (int i = tid; i < a.num_ops * 4; i += T)
      reinterpret_cast<int4*>(sops)[i] =
          reinterpret_cast<const int4*>(a.ops)[i];
  for (int k = tid; k < 2 * a.num_slots; k += T)
    csn[k] = (R)a.angles[2 * (s * a.total_slots + a.slot0) + k];
  const AdjRegOp* const ops = staged ? sops : a.ops;
  C* const gp = psi + (s << a.n) + base + offset(tid);
  C* const gl = lam + (s << a.n) + base + offset(tid);
  __syncthreads();
#pragma unroll 4
  for (int i = 0; i < NR; ++i) {
    const int at = ar_swz<R>(tid + T * i);
    if constexpr (sizeof(R) == 4) {
      cp_async8(&SP[at], gp + ioff[i]);
      cp_async8(&SL[at], gl + ioff[i]);
    } else {
      cp_async16<R>(&SP[at], gp + ioff[i]);
      cp_async16<R>(&SL[at], gl + ioff[i]);
    }
  }
  cp_async_wait_all();
  __syncthreads();

  int pending = 0;  // gradient sums in buf (block-uniform)
  C x[NR], l[NR];
  for (int li = 0; li < a.num_layouts; ++li) {
    const AdjLayout& L = a.layouts[li];
    int tb = 0;  // tile bits of this thread
    for (int j = 0; j < a.m - RB; ++j)
      if ((tid >> j) & 1) tb |= 1 << L.tb[j];
    const int at = ar_swz<R>(tb);
    int ro[RB];
#pragma unroll
    for (int k = 0; k < RB; ++k) ro[k] = ar_swz<R>(1 << L.rb[k]);
    auto reg = [&](int i) {  // slot of register i
      int o = at;
#pragma unroll
      for (int k = 0; k < RB; ++k)
        if ((i >> k) & 1) o ^= ro[k];
      return o;
    };
    auto take = [&]() {
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int o = reg(i);
        x[i] = SP[o];
        l[i] = SL[o];
      }
    };
    auto put = [&]() {
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        const int o = reg(i);
        SP[o] = x[i];
        SL[o] = l[i];
      }
    };
    take();
    C tf;  // factor of diagonals on bits that are not registers
    tf.x = 1;
    tf.y = 0;
    uint32_t neg = 0;  // registers whose sign is still to be flipped
    const int end = L.first + L.count;
    for (int oi = L.first; oi <= end; ++oi) {  // a layout has ops
      const AdjRegOp& op = ops[oi < end ? oi : end - 1];
      const int type = oi < end ? op.type : (int)AR_END;
      if (type < AR_END && (base & op.cmask) != op.cval) continue;
      if (type == AR_SIGN) {
        if ((tb & op.t[0]) == op.t[0]) neg ^= (uint32_t)op.signs;
        continue;
      }
      // signs and factors commute with diagonals; everything else sees them
      if ((type < 8 || type >= AR_DENSE1) && neg) {
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          const uint32_t sg = (neg << (31 - i)) & 0x80000000u;
          x[i].x = ar_neg<R>(x[i].x, sg);
          x[i].y = ar_neg<R>(x[i].y, sg);
          l[i].x = ar_neg<R>(l[i].x, sg);
          l[i].y = ar_neg<R>(l[i].y, sg);
        }
        neg = 0;
      }
      if (type <= AR_RZ_OUT) {
        const R c = csn[2 * op.slot], sr = csn[2 * op.slot + 1];
        R g = 0;
        switch (type) {
          case 0: g = ar_rot<R, NR, 0, 0>(x, l, c, sr); break;
          case 1: g = ar_rot<R, NR, 0, 1>(x, l, c, sr); break;
          case 2: g = ar_rot<R, NR, 0, 2>(x, l, c, sr); break;
          case 3: g = ar_rot<R, NR, 0, RB - 1>(x, l, c, sr); break;
          case 4: g = ar_rot<R, NR, 1, 0>(x, l, c, sr); break;
          case 5: g = ar_rot<R, NR, 1, 1>(x, l, c, sr); break;
          case 6: g = ar_rot<R, NR, 1, 2>(x, l, c, sr); break;
          case 7: g = ar_rot<R, NR, 1, RB - 1>(x, l, c, sr); break;
          case 8: g = ar_rot<R, NR, 2, 0>(x, l, c, sr); break;
          case 9: g = ar_rot<R, NR, 2, 1>(x, l, c, sr); break;
          case 10: g = ar_rot<R, NR, 2, 2>(x, l, c, sr); break;
          case 11: g = ar_rot<R, NR, 2, RB - 1>(x, l, c, sr); break;
          default: {
            // Z on a bit that is one value for the thread: +-Im
            // <lambda|psi>, and the same factor on both states
#pragma unroll
            for (int i = 0; i < NR; ++i) {
              g = fma(l[i].x, x[i].y, g);
              g = fma(-l[i].y, x[i].x, g);
            }
            const bool one = type == AR_RZ_TILE ? (tb & op.t[0]) != 0
                                                : (base >> op.o[0]) & 1;
            if (one) g = -g;
            C f;
            f.x = c;
            f.y = one ? -sr : sr;
            tf = cmul(tf, f);
          }
        }
        buf[pending * T + tid] = g;
        if (tid == 0) slots[pending] = op.slot;
        if (++pending == AR_BATCH<R>) {
          __syncthreads();
          ar_reduce<R>(buf, slots, pending, a);
          __syncthreads();
          pending = 0;
        }
      } else if (type == AR_DIAG) {
        // registers where qubit 0 / qubit 1 is set (all or none where the
        // qubit is not a register bit)
        uint32_t q[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (j >= op.nq) continue;
          q[j] = op.k[j] >= 0 ? ar_regs(op.k[j])
                 : (op.t[j] ? (tb & op.t[j]) != 0 : (base >> op.o[j]) & 1)
                     ? 0xFFFFu
                     : 0u;
        }
        const int hi = op.nq - 1;  // qubit 0 is the index's high bit
        if (op.k[0] < 0 && (op.nq < 2 || op.k[1] < 0)) {
          const int e = ((q[0] ? 1 : 0) << hi) |
                        (op.nq == 2 && q[1] ? 1 : 0);
          tf = cmul(pool[op.mat + e], tf);
        } else {
          C d[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            d[e] = pool[op.mat + (e < (1 << op.nq) ? e : 0)];
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            const int e = (((q[0] >> i) & 1) << hi) |
                          (op.nq == 2 ? (q[1] >> i) & 1 : 0);
            const C lo = e & 1 ? d[1] : d[0], up = e & 1 ? d[3] : d[2];
            const C f = e & 2 ? up : lo;
            x[i] = cmul(f, x[i]);
            l[i] = cmul(f, l[i]);
          }
        }
      } else if (type < AR_END) {
        // fixed dense gates, through the thread's own slots
        put();
        const int f0 = ar_swz<R>(1 << L.rb[op.k[0]]);
        const C* mp = pool + op.mat;
        if (type == AR_DENSE1) {
          uint32_t cm = 0xFFFFu;  // registers the gate acts on
          if (op.nq == 2) {
            cm = op.k[1] >= 0 ? ar_regs(op.k[1])
                 : (op.t[1] ? (tb & op.t[1]) != 0 : (base >> op.o[1]) & 1)
                     ? 0xFFFFu
                     : 0u;
            mp += 10;
          }
          const int row = op.nq == 2 ? 4 : 2;
          const C m0 = mp[0], m1 = mp[1], m2 = mp[row], m3 = mp[row + 1];
          const uint32_t half = ar_regs(op.k[0]);
#pragma unroll 1
          for (int i = 0; i < NR; ++i) {
            if (((half >> i) & 1) || !((cm >> i) & 1)) continue;
            int o = at;
            for (int k = 0; k < RB; ++k)
              if ((i >> k) & 1) o ^= ar_swz<R>(1 << L.rb[k]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              C* const S = h ? SL : SP;
              const C a0 = S[o], a1 = S[o ^ f0];
              S[o] = cmad(m1, a1, cmul(m0, a0));
              S[o ^ f0] = cmad(m3, a1, cmul(m2, a0));
            }
          }
        } else {
          const int f1 = ar_swz<R>(1 << L.rb[op.k[1]]);
          const uint32_t skip = ar_regs(op.k[0]) | ar_regs(op.k[1]);
#pragma unroll 1
          for (int i = 0; i < NR; ++i) {
            if ((skip >> i) & 1) continue;
            int o = at;
            for (int k = 0; k < RB; ++k)
              if ((i >> k) & 1) o ^= ar_swz<R>(1 << L.rb[k]);
            const int p[4] = {o, o ^ f1, o ^ f0, o ^ f0 ^ f1};
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
              C* const S = h ? SL : SP;
              C v[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) v[j] = S[p[j]];
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                C acc = cmul(mp[4 * r], v[0]);
                acc = cmad(mp[4 * r + 1], v[1], acc);
                acc = cmad(mp[4 * r + 2], v[2], acc);
                acc = cmad(mp[4 * r + 3], v[3], acc);
                S[p[r]] = acc;
              }
            }
          }
        }
        take();
      }
    }
    if (!(tf.x == 1 && tf.y == 0)) {
#pragma unroll
      for (int i = 0; i < NR; ++i) {
        x[i] = cmul(tf, x[i]);
        l[i] = cmul(tf, l[i]);
      }
    }
    put();
    __syncthreads();
  }
  if (pending) ar_reduce<R>(buf, slots, pending, a);
#pragma unroll 4
  for (int i = 0; i < NR; ++i) {
    const int at = ar_swz<R>(tid + T * i);
    __stcs(gp + ioff[i], SP[at]);
    __stcs(gl + ioff[i], SL[at]);
  }
}

// (cos, sin) of half * params[s, pidx] for every state and slot, FP64.
struct AdjRot {
  int32_t pidx;
  int32_t pad_;
  double half;
};

template <typename P>
__global__ void __launch_bounds__(256)
    adjoint_table_kernel(const P* params, int64_t num_params,
                         int64_t num_states, const AdjRot* rots,
                         int64_t total, double* out) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= num_states * total) return;
  const AdjRot r = rots[i % total];
  double sn, cs;
  sincos((double)params[(i / total) * num_params + r.pidx] * r.half, &sn,
         &cs);
  reinterpret_cast<double2*>(out)[i] = make_double2(cs, sn);
}

// grad[s, param[slot]] += scale[slot] * (sum of the state's tile partials)
// for slots [slot0, slot1), partials [slot - slot0][tile].  Slots of one
// parameter are chained (prev, next; -1 ends): the block of the chain's
// first slot in the range walks it, so a parameter that drives several
// rotations has one writer and a fixed order.
__global__ void __launch_bounds__(128)
    adjoint_grad_sum_kernel(const double* partial, int64_t slot0,
                            int64_t slot1, uint64_t tiles_per_state,
                            uint64_t tiles, const int32_t* param,
                            const double* scale, const int32_t* prev,
                            const int32_t* next, double* grad,
                            int64_t num_params) {
  const uint64_t num_states = tiles / tiles_per_state;
  const int64_t first = slot0 + (int64_t)(blockIdx.x / num_states);
  const uint64_t s = blockIdx.x % num_states;
  if (prev[first] >= slot0) return;
  __shared__ double red[4];
  double total = 0.0;
  for (int64_t k = first; k >= 0 && k < slot1; k = next[k]) {
    double acc = 0.0;
    for (uint64_t t = threadIdx.x; t < tiles_per_state; t += 128)
      acc += partial[(uint64_t)(k - slot0) * tiles + s * tiles_per_state + t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    total += scale[k] * (((red[0] + red[1]) + red[2]) + red[3]);
    __syncthreads();
  }
  if (threadIdx.x == 0) grad[s * num_params + param[first]] += total;
}

template <typename R, int RB>
static int ar_launch(void* psi, void* lam, const void* pool,
                     const AdjRegArgs& a, cudaStream_t st) {
  const int T = 1 << (a.m - RB);
  const size_t smem = ((size_t)4 * sizeof(R) << a.m) +
                      (size_t)AR_BATCH<R> * T * sizeof(R) +
                      (size_t)2 * a.num_slots * sizeof(R);
  constexpr size_t kMost = 200 * 1024;
  if (smem > kMost)
    return set_error(GBSV_ERR_UNSUPPORTED,
                     "adjoint stage with %d rotations needs %zu bytes of "
                     "shared memory", a.num_slots, smem);
  static OncePerDevice once;
  const int rc = allow_smem(once, adjoint_reg_kernel<R, RB>, (int)kMost,
                            "adjoint_reg_kernel");
  if (rc) return rc;
  adjoint_reg_kernel<R, RB><<<(unsigned)a.tiles, T, smem, st>>>(
      static_cast<Cx<R>*>(psi), static_cast<Cx<R>*>(lam),
      static_cast<const Cx<R>*>(pool), a);
  return after_launch("adjoint_reg_kernel");
}

}  // namespace gbsv

using namespace gbsv;

extern "C" int gbsv_adjoint_register_bits(int dtype) {
  return dtype == GBSV_C64 ? 4 : dtype == GBSV_C128 ? 3 : 0;
}

extern "C" int gbsv_adjoint_stage_regs(
    void* psi, void* lam, int dtype, int num_qubits, int64_t num_states,
    int tile_qubits, int contiguous_qubits, const int32_t* tile_positions,
    const void* ops, int num_ops, const void* layouts, int num_layouts,
    const void* pool, const double* angles, int64_t total_slots,
    int64_t slot0, int num_slots, double* partial, void* stream) {
  if (dtype != GBSV_C64 && dtype != GBSV_C128)
    return set_error(GBSV_ERR_INVALID_ARG, "state dtype must be complex");
  const int n = num_qubits, m = tile_qubits, c = contiguous_qubits;
  const int rb = gbsv_adjoint_register_bits(dtype);
  if (n < 1 || n > 62 || m < rb + 5 || m > n || m > rb + 8 ||
      c < 0 || c > m || num_states < 0 || num_ops < 0 || num_layouts < 0 ||
      num_slots < 0 || slot0 < 0 || slot0 + num_slots > total_slots)
    return set_error(GBSV_ERR_INVALID_ARG, "bad adjoint stage n=%d m=%d c=%d",
                     n, m, c);
  if (num_states == 0) return GBSV_OK;
  if (!psi || !lam || psi == lam || !tile_positions ||
      (num_ops > 0 && (!ops || !pool || !layouts)) ||
      (num_slots > 0 && (!angles || !partial)))
    return set_error(GBSV_ERR_INVALID_ARG, "null or aliased pointer");
  const uintptr_t amp = (uintptr_t)dtype_bytes(dtype);
  if ((uintptr_t)psi % amp || (uintptr_t)lam % amp)
    return set_error(GBSV_ERR_INVALID_ARG, "psi or lambda is not aligned");
  AdjRegArgs a{};
  a.n = n;
  a.m = m;
  a.c = c;
  a.ops = static_cast<const AdjRegOp*>(ops);
  a.num_ops = num_ops;
  a.layouts = static_cast<const AdjLayout*>(layouts);
  a.num_layouts = num_ops > 0 ? num_layouts : 0;
  a.angles = angles;
  a.total_slots = total_slots;
  a.slot0 = slot0;
  a.num_slots = num_slots;
  a.partial = partial;
  uint64_t seen = 0;
  for (int j = 0; j < m; ++j) {
    const int p = tile_positions[j];
    if (p < 0 || p >= n || ((seen >> p) & 1) || (j < c && p != j))
      return set_error(GBSV_ERR_INVALID_ARG, "bad tile position %d", p);
    seen |= uint64_t(1) << p;
    if (j >= c) a.hpos[j - c] = p;
    a.spos[j] = p;
  }
  std::sort(a.spos, a.spos + m);
  a.tiles = (uint64_t)num_states << (n - m);
  if (a.tiles > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "too many tiles");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return dtype == GBSV_C64 ? ar_launch<float, 4>(psi, lam, pool, a, st)
                           : ar_launch<double, 3>(psi, lam, pool, a, st);
}

extern "C" int gbsv_adjoint_angles(const void* params, int params_dtype,
                                   int64_t num_params, int64_t num_states,
                                   const void* rots, int64_t total_slots,
                                   double* angles, void* stream) {
  if (params_dtype != GBSV_F32 && params_dtype != GBSV_F64)
    return set_error(GBSV_ERR_INVALID_ARG, "params must be float32/float64");
  if (num_params < 0 || num_states < 0 || total_slots < 0)
    return set_error(GBSV_ERR_INVALID_ARG, "negative size");
  if (num_states == 0 || total_slots == 0) return GBSV_OK;
  if (!params || !rots || !angles)
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  const uint64_t grid = ((uint64_t)num_states * total_slots + 255) / 256;
  if (grid > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "too many rotations");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const AdjRot* r = static_cast<const AdjRot*>(rots);
  if (params_dtype == GBSV_F32)
    adjoint_table_kernel<float><<<(unsigned)grid, 256, 0, st>>>(
        static_cast<const float*>(params), num_params, num_states, r,
        total_slots, angles);
  else
    adjoint_table_kernel<double><<<(unsigned)grid, 256, 0, st>>>(
        static_cast<const double*>(params), num_params, num_states, r,
        total_slots, angles);
  return after_launch("adjoint_table_kernel");
}

extern "C" int gbsv_adjoint_grad_sum(const double* partial, int64_t slot0,
                                     int64_t slot1, int64_t num_states,
                                     int64_t tiles_per_state,
                                     const int32_t* slot_param,
                                     const double* slot_scale,
                                     const int32_t* prev, const int32_t* next,
                                     double* grad, int64_t num_params,
                                     void* stream) {
  if (slot0 < 0 || slot1 < slot0 || num_states < 0 || tiles_per_state < 1 ||
      num_params < 0)
    return set_error(GBSV_ERR_INVALID_ARG, "bad sizes");
  if (slot1 == slot0 || num_states == 0) return GBSV_OK;
  if (!partial || !slot_param || !slot_scale || !prev || !next || !grad)
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  const uint64_t grid = (uint64_t)(slot1 - slot0) * num_states;
  if (grid > 0x7fffffffull)
    return set_error(GBSV_ERR_UNSUPPORTED, "too many gradient slots");
  adjoint_grad_sum_kernel<<<(unsigned)grid, 128, 0,
                            static_cast<cudaStream_t>(stream)>>>(
      partial, slot0, slot1, (uint64_t)tiles_per_state,
      (uint64_t)num_states * tiles_per_state, slot_param, slot_scale, prev,
      next, grad, num_params);
  return after_launch("adjoint_grad_sum_kernel");
}
