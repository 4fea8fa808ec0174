// Tensor-core fused stages (complex64).
//
// A stage owns 12 "tile bits" of the amplitude index (the lowest c bits and
// 12 - c higher ones, as in the register stages of fused.cu), so every tile
// is 4096 amplitudes (32 KiB) and the stage costs one read and one write of
// the state.  The host planner groups the stage's gates into "blocks": the
// product of a run of gates on at most 5 tile bits is one 32x32 complex
// matrix U, multiplied into the tile on the tensor cores.
//
// Per block, the tile is viewed as a 32 x 128 matrix: row index = the 5
// block bits, column = the other 7 tile bits.  Thread r (one warpgroup,
// r = 0..127) gathers column r from shared memory (32 amplitudes), writes
// it to tensor memory as row r of the MMA's A operand (K = 64 reals), and
// tcgen05.mma multiplies it by the real form of U^T (64 x 64, B operand in
// shared memory): D = A * B, M = 128 columns, N = 64 output reals.  The
// result comes back with tcgen05.ld into the same thread, which scatters it
// into the tile for the next block.
//
// Precision (kind::f16, FP32 accumulation).  GB300's tensor cores truncate
// the FP32 accumulation (measured: sums round toward zero), so a plain
// fp16 split would shrink every amplitude a little per block.  Instead the
// split makes the dominant product exact:
//   * each thread scales its 64 reals by a power of two s so the largest is
//     below 2^10, and splits x*s = hi + lo with hi an integer (|hi| <=
//     1024, exact in fp16) and lo (|lo| <= 1/2) rounded to fp16;
//   * the host splits 1024 * B the same way into an integer matrix Bh and
//     an fp16 residual Bl = 1024 * B - Bh (|Bl| <= 1/2);
//   * D1 = hi * Bh is a sum of integer products bounded by
//     1024 * (1024 * 8 + 32) < 2^24 (a unitary's real-form columns have
//     L1 norm <= 8; other matrices are scaled into that, tc_columns), so
//     every partial sum is an exact FP32 integer and the truncating
//     accumulator makes no error;
//   * Dc = hi * Bl + lo * Bh + lo * Bl (the split of Ootomo & Yokota 2022,
//     the first two as one K = 128 product [hi | lo] * [Bl; Bh]) carries the
//     correction, about 2^-11 of D1's magnitude, where the truncation
//     costs about 2^-34 relative;
//   * y = (D1 + Dc) / (1024 s), an exact power-of-two scaling.
// The last product is a quarter more tensor work on a pipe that is 13%
// busy, and most of the accuracy: a block's matrix has few exact entries, so
// each lo * Bl is up to 1/4 and 64 of them about 2^-21 of the column's
// largest amplitude; with it the fp16 rounding of lo and Bl is left, about
// 2^-23 (120 gates on 26 qubits in 10 blocks: 3.7e-6 of the state without,
// 8.5e-7 with it).
//
// Diagonal gates whose bits are all outside a block's bits (thread bits,
// or positions outside the tile) commute with the block.  The host folds
// them into a per-block table of per-thread factors indexed by up to 5 bits
// outside the tile; the rare rest stay a list of post-diagonals.
//
// Two kernels.  tc_wide_kernel, below, runs stages of up to eight blocks.
// tc_stage_kernel runs longer ones, split by role (two CTAs of 192 threads
// per SM, 107 KiB of shared memory and 256 tensor-memory columns each): four
// compute warps (gather, split, tcgen05.st, tcgen05.ld, scatter), one warp
// whose lane 0 issues the MMAs and streams block images (16 KiB, two buffers
// by cp.async.bulk), and one warp that loads tiles by 16-byte cp.async into two
// buffers and writes finished tiles back, so the memory pipeline never
// stalls the compute warps.
#include "common.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace gbsv {

constexpr int TC_M = 12;             // tile bits
constexpr int TC_RB = 5;             // block (register) bits
constexpr int TC_TB = TC_M - TC_RB;  // thread bits
constexpr int TC_THREADS = 1 << TC_TB;
constexpr int TC_TILE = 1 << TC_M;
constexpr int TC_MAX_BLOCKS = 64;
constexpr int TC_MAX_SDIAG = 64;     // post-diagonals staged in shared memory
constexpr int TC_IMG_BYTES = 16384;
constexpr int TC_SMEM_BYTES = 2 * TC_TILE * 8 + 2 * TC_IMG_BYTES + 1024;

// Block record (gbsv_tc_block_t).  Shared-memory offsets are in amplitudes
// after the tile swizzle; the swizzle is linear over GF(2), so amplitude
// (thread bits of r) | (register bits of i) sits at
// XOR(tspo[j] : bit j of r) ^ XOR(rspo[k] : bit k of i).
struct TcBlock {
  int16_t rspo[TC_RB];  // register-index bit k -> swizzled offset
  int16_t tspo[TC_TB];  // thread-index bit j -> swizzled offset
  int32_t mat;          // image index (16 KiB each)
  int32_t first_diag;   // post-diagonals [first_diag, first_diag + num_diag)
  int32_t num_diag;
  int32_t flags;        // TC_PAIRS: register bit 0 is tile bit 0; TC_COLS
  int32_t fac;          // factor table: factors[fac + p * 128 + thread]
  int8_t nout;          // p's bits: the state's bits at positions opos[]
  int8_t opos[7];
  int32_t cols;         // TC_COLS: 32 column scales (floats) at factors[cols]
  int32_t pad_[2];
};
static_assert(sizeof(TcBlock) == 64, "gbsv_tc_block_t is 64 bytes");
constexpr int TC_PAIRS = 1, TC_COLS = 2;

// Post-diagonal: a 1- or 2-qubit diagonal applied after its block.  Each
// qubit is encoded as a register bit (0..4), a thread-index bit (5 + j) or
// -1 - its position outside the tile; the first qubit is the index MSB.
struct TcDiag {
  int32_t nq;
  int32_t enc[2];
  int32_t reg;  // nonzero when a qubit is a register bit
  float2 d[4];
};
static_assert(sizeof(TcDiag) == 48, "gbsv_tc_diag_t is 48 bytes");

struct TcArgs {
  int n, c, num_blocks;
  int64_t num_states;
  int64_t in_stride;       // amplitudes between input states (0 = bcast)
  int hpos[TC_M];          // global position of tile bit c + j
  int spos[TC_M];          // all tile positions, ascending
  const TcBlock* blocks;
  const TcDiag* diags;
  const unsigned char* images;
  const float2* factors;
};

static __device__ int g_tc_status;  // nonzero after a bounded wait ran out

// Tile swizzle: amplitude bits 1-3 ^= bits 4-6 ^ 7-9 ^ 10-12.  Bit 0 stays,
// so 16-byte pieces (two amplitudes) stay whole for the copies, and every
// tile bit >= 1 has a non-zero image in the bank bits.
__device__ __forceinline__ int tc_swz(int l) {
  return l ^ ((((l >> 4) ^ (l >> 7) ^ (l >> 10)) & 7) << 1);
}

// Lowest set bit of a (compile-time) register index.
__host__ __device__ constexpr int tc_ctz(int i) {
  return (i & 1) ? 0 : (i & 2) ? 1 : (i & 4) ? 2 : (i & 8) ? 3 : 4;
}

__device__ __forceinline__ uint32_t tc_smem(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Wait for phase `parity` of an mbarrier, for at most about 2^31 cycles.
// try_wait suspends the thread until the phase completes or the hinted
// time (1 ms) passes, so a waiting warp takes no issue slots.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(1000000u)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > (1ll << 31)) return false;
  }
}

__device__ __forceinline__ void tc_load_image(uint32_t dst, const void* src,
                                              uint32_t bar) {
  asm volatile(
      "mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
      "r"(TC_IMG_BYTES)
      : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(src), "r"(TC_IMG_BYTES), "r"(bar)
      : "memory");
}

// Shared-memory matrix descriptor: K-major, no swizzle; core matrices of
// 8 rows x 16 bytes, K-adjacent ones 128 bytes apart (leading byte offset),
// 8-row groups 2048 bytes apart (stride byte offset).
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)(128 >> 4) << 16) |
         ((uint64_t)(2048 >> 4) << 32) | ((uint64_t)1 << 46);
}

// D (f32) = A (f16, tensor memory) * B (f16, shared memory), M = 128,
// N = 64 or 128, K = 16; accumulate into D when acc != 0.
template <int N>
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint64_t b,
                                       uint32_t acc) {
  constexpr uint32_t idesc = (1u << 4)  // D f32; A, B f16; both K-major
                             | ((uint32_t)(N >> 3) << 17) |
                             ((uint32_t)(128 >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(
          d),
      "r"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

#define TC_R16(r)                                                            \
  "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),          \
      "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),    \
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])

// 16 consecutive 32-bit columns of this thread's lane.
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      TC_R16(r)
      : "memory");
}

#define TC_W32(r)                                                            \
  "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),    \
      "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),           \
      "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),       \
      "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),       \
      "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),       \
      "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),       \
      "=r"(r[31])
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : TC_W32(r)
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ uint32_t tc_pack(float lo_k, float hi_k) {
  const __half2 h = __floats2half2_rn(lo_k, hi_k);
  return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint64_t tc_tile_base(const TcArgs& a,
                                                 uint64_t t) {
  uint64_t base = t;
#pragma unroll
  for (int j = 0; j < TC_M; ++j) base = insert_zero(base, a.spos[j]);
  return base;
}

// Global offset of tile amplitude l (bits < c contiguous, bit c + j at
// position hpos[j]).
__device__ __forceinline__ uint64_t tc_tile_offset(const TcArgs& a, int l) {
  uint64_t off = (uint64_t)(l & ((1 << a.c) - 1));
  const int r = l >> a.c;
  for (int j = 0; j < TC_M - a.c; ++j)
    if ((r >> j) & 1) off += uint64_t(1) << a.hpos[j];
  return off;
}

// The pieces of a block that a thread does on its column of 32 amplitudes;
// register i lives in the tile at sb ^ (XOR of rs[j] over the bits j of i).
__device__ __forceinline__ void tc_addresses(int sb, const int* rs, int* ad) {
  ad[0] = sb;
#pragma unroll
  for (int i = 1; i < 32; ++i) ad[i] = ad[i & (i - 1)] ^ rs[tc_ctz(i)];
}
__device__ __forceinline__ void tc_gather(const float2* S, int sb,
                                          const int* rs, bool pairs,
                                          float2* v) {
  int ad[32];
  tc_addresses(sb, rs, ad);
  if (pairs) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float4 w = *reinterpret_cast<const float4*>(&S[ad[i]]);
      v[i] = make_float2(w.x, w.y);
      v[i + 1] = make_float2(w.z, w.w);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = S[ad[i]];
  }
}
__device__ __forceinline__ void tc_scatter(float2* S, int sb, const int* rs,
                                           bool pairs, const float2* v) {
  int ad[32];
  tc_addresses(sb, rs, ad);
  if (pairs) {
#pragma unroll
    for (int i = 0; i < 32; i += 2)
      *reinterpret_cast<float4*>(&S[ad[i]]) =
          make_float4(v[i].x, v[i].y, v[i + 1].x, v[i + 1].y);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) S[ad[i]] = v[i];
  }
}

// Blocks that are not unitary: the image's entries were scaled by column into
// its range (rows' L1 norm at most 8, largest entry near 1; without, entries
// beyond 64 are infinite in fp16 and small ones have 11 bits), and the powers
// of two go to the amplitudes, exactly.  Stages with such a block have
// kernels of their own (SCALED): in one kernel the branches cost the others 5%
// of their time (26 qubits 1647 -> 1732 us), and a second copy of the compute
// loop 2% of a short program's (16 qubits x 10: 35.4 -> 36.1 us).
__device__ __forceinline__ void tc_columns(const TcArgs& a, const TcBlock& B,
                                           float2* v) {
  if (!(B.flags & TC_COLS)) return;
  const float2* sc = a.factors + B.cols;
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    const float2 w = __ldg(sc + i / 2);
    v[i] = make_float2(v[i].x * w.x, v[i].y * w.x);
    v[i + 1] = make_float2(v[i + 1].x * w.y, v[i + 1].y * w.y);
  }
}

// Power-of-two scaling (largest |x| of the column, tree reduction): x * sc
// is below 2^10, inv undoes it and the images' 1024.  A column below 2^-107,
// where inv would be no normal float, is first taken times 2^64, and inv is
// negative to say so (tc_unscale).  Only stages with a scaled block do this,
// whose states can shrink.
constexpr float TC_TINY = 18446744073709551616.f;  // 2^64
template <bool SCALED>
__device__ __forceinline__ void tc_scale(float2* v, float* sc, float* inv) {
  float mx[16];
#pragma unroll
  for (int i = 0; i < 16; ++i)
    mx[i] = fmaxf(fmaxf(fabsf(v[i].x), fabsf(v[i].y)),
                  fmaxf(fabsf(v[i + 16].x), fabsf(v[i + 16].y)));
#pragma unroll
  for (int w = 8; w > 0; w >>= 1)
#pragma unroll
    for (int i = 0; i < w; ++i) mx[i] = fmaxf(mx[i], mx[i + w]);
  uint32_t bits = __float_as_uint(mx[0]), sign = 0;
  if (SCALED && bits - 1 < (20u << 23) - 1) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      v[i] = make_float2(v[i].x * TC_TINY, v[i].y * TC_TINY);
    bits = __float_as_uint(mx[0] * TC_TINY);
    sign = 0x80000000u;
  }
  const int E = max((int)(bits >> 23), 20);
  *sc = __uint_as_float((uint32_t)(263 - E) << 23);
  *inv = __uint_as_float((uint32_t)(E - 19) << 23 | sign);
}
__device__ __forceinline__ void tc_unscale(float2* v, float inv) {
  if (inv >= 0.f) return;
#pragma unroll
  for (int i = 0; i < 32; ++i)
    v[i] = make_float2(v[i].x * (-1.f / TC_TINY), v[i].y * (-1.f / TC_TINY));
}

// x * sc = hi + lo for COUNT amplitudes: hi = x * sc rounded to an integer
// (adding and removing 1.5 * 2^23 rounds to nearest; |x * sc| < 2^10), lo
// the exact remainder (|lo| <= 1/2), both to fp16.
template <int COUNT>
__device__ __forceinline__ void tc_split(const float2* v, float sc,
                                         uint32_t* hi, uint32_t* lo) {
  constexpr float RND = 12582912.f;
#pragma unroll
  for (int j = 0; j < COUNT; ++j) {
    const float hr = fmaf(v[j].x, sc, RND) - RND;
    const float hm = fmaf(v[j].y, sc, RND) - RND;
    hi[j] = tc_pack(hr, hm);
    lo[j] = tc_pack(fmaf(v[j].x, sc, -hr), fmaf(v[j].y, sc, -hm));
  }
}

// A thread's factor of the diagonals folded into the block's table.
__device__ __forceinline__ float2 tc_factor(const TcArgs& a, const TcBlock& B,
                                            uint64_t base, int tid) {
  if (B.fac < 0) return make_float2(1.f, 0.f);
  int p = 0;
  for (int j = 0; j < B.nout; ++j)
    p |= (int)((base >> B.opos[j]) & 1) << j;
  return __ldg(a.factors + B.fac + p * TC_THREADS + tid);
}

// The post-diagonals left in the list (a register bit, or too many outside
// bits): those without a register bit into f; returns whether there are
// others.
__device__ __forceinline__ bool tc_outer_diags(const TcBlock& B,
                                               const TcDiag* dtab,
                                               uint64_t base, int tid,
                                               float2* f) {
  bool regdiag = false;
  for (int q = B.first_diag; q < B.first_diag + B.num_diag; ++q) {
    const TcDiag& dg = dtab[q];
    if (dg.reg) {
      regdiag = true;
      continue;
    }
    int idx = 0;
    for (int u = 0; u < dg.nq; ++u) {
      const int en = dg.enc[u];
      const int bit = en >= TC_RB ? (tid >> (en - TC_RB)) & 1
                                  : (int)((base >> (-1 - en)) & 1);
      idx = (idx << 1) | bit;
    }
    *f = cmul(*f, dg.d[idx]);
  }
  return regdiag;
}
__device__ __forceinline__ void tc_register_diags(const TcBlock& B,
                                                  const TcDiag* dtab,
                                                  uint64_t base, int tid,
                                                  float2* v) {
  for (int q = B.first_diag; q < B.first_diag + B.num_diag; ++q) {
    const TcDiag& dg = dtab[q];
    if (!dg.reg) continue;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      int idx = 0;
      for (int u = 0; u < dg.nq; ++u) {
        const int en = dg.enc[u];
        const int bit = en < 0 ? (int)((base >> (-1 - en)) & 1)
                        : en < TC_RB ? (i >> en) & 1
                                     : (tid >> (en - TC_RB)) & 1;
        idx = (idx << 1) | bit;
      }
      v[i] = cmul(dg.d[idx], v[i]);
    }
  }
}

// Roles (192 threads): warps 0-3 compute (thread r owns column r of the
// tile and TMEM lane r), warp 4 lane 0 issues the MMAs and streams block
// images, warp 5 loads and stores tiles.  They hand over through mbarriers:
//   full[b]   tile buffer b loaded      (warp 5 cp.async -> compute)
//   empty[b]  tile buffer b computed    (compute -> warp 5: store, refill)
//   a_ready   A written to TMEM         (compute -> MMA lane)
//   mma_done  MMAs of a block complete  (tcgen05.commit -> compute)
//   img[b]    block image b landed      (cp.async.bulk -> MMA lane)
// Every wait is bounded (tc_wait); one that runs out sets the CTA's abort
// flag and the error status, and every role then leaves its loop.
constexpr int TC_ROLE_THREADS = TC_THREADS + 64;

// Barrier 1 over the compute warps, returning the OR of x over them.
__device__ __forceinline__ bool tc_compute_sync_or(bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)x), "n"(TC_THREADS)
      : "memory");
  return r != 0;
}

template <bool SCALED>
__global__ void __launch_bounds__(TC_ROLE_THREADS, 2)
    tc_stage_kernel(const float2* in, float2* out, TcArgs a) {
  extern __shared__ __align__(1024) unsigned char tc_smem_raw[];
  // 1024-byte alignment of the dynamic area is not guaranteed: round up
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023) & ~uintptr_t(1023));
  float2* const tiles = reinterpret_cast<float2*>(smem);
  unsigned char* const imgs = smem + 2 * TC_TILE * 8;
  __shared__ TcBlock sblk[TC_MAX_BLOCKS];
  __shared__ TcDiag sdiag[TC_MAX_SDIAG];
  __shared__ uint64_t offh[16];
  __shared__ __align__(8) uint64_t bar_full[2], bar_empty[2], bar_img[2];
  __shared__ __align__(8) uint64_t bar_a, bar_mma;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane_id = tid & 31;
  const int nb = a.num_blocks;
  const uint64_t tps = uint64_t(1) << (a.n - TC_M);
  const uint64_t num_tiles = (uint64_t)a.num_states * tps;
  const uint64_t t0 = (uint64_t)blockIdx.x * num_tiles / gridDim.x;
  const uint64_t t1 = (uint64_t)(blockIdx.x + 1) * num_tiles / gridDim.x;
  if (t0 >= t1) return;
  const uint64_t ntile = t1 - t0;
  const uint64_t total_exec = ntile * (uint64_t)nb;

  if (warp == 0) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::
            "r"(tc_smem(&s_tmem))
        : "memory");
    asm volatile(
        "tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::
            : "memory");
  }
  if (tid == 0) {
    auto init = [](uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(
                       tc_smem(bar)),
                   "r"(count));
    };
    init(&bar_full[0], 32);  // one cp.async arrival per loader lane
    init(&bar_full[1], 32);
    init(&bar_empty[0], TC_THREADS);
    init(&bar_empty[1], TC_THREADS);
    init(&bar_img[0], 1);
    init(&bar_img[1], 1);
    init(&bar_a, TC_THREADS);
    init(&bar_mma, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = tid; i < nb * 16; i += TC_ROLE_THREADS)
    reinterpret_cast<int32_t*>(sblk)[i] =
        reinterpret_cast<const int32_t*>(a.blocks)[i];
  // the stage's post-diagonals: one contiguous range, staged in shared
  // memory when it fits (read from global memory otherwise)
  const int dfirst = a.blocks[0].first_diag;
  const int dcount =
      a.blocks[nb - 1].first_diag + a.blocks[nb - 1].num_diag - dfirst;
  const bool dshared = dcount <= TC_MAX_SDIAG;
  if (dshared)
    for (int i = tid; i < dcount * 12; i += TC_ROLE_THREADS)
      reinterpret_cast<int32_t*>(sdiag)[i] =
          reinterpret_cast<const int32_t*>(a.diags + dfirst)[i];
  const TcDiag* const dtab = dshared ? sdiag - dfirst : a.diags;
  if (tid < 16) offh[tid] = tc_tile_offset(a, 256 * tid);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;

  // tiles of a CTA are consecutive: the base (the tile's amplitude bits
  // outside the tile) steps by a masked increment over the outside bits
  uint64_t tmask = ~((uint64_t(1) << a.n) - 1);
  for (int j = 0; j < TC_M; ++j) tmask |= uint64_t(1) << a.spos[j];
  auto next_base = [&](uint64_t b) { return ((b | tmask) + 1) & ~tmask; };
  auto fail = [&](int code) {
    s_abort = 1;
    atomicOr(&g_tc_status, code);
  };

  if (warp == 5) {
    // ---------------------------------------------- tile loader / storer
    // lane l moves 16-byte pieces l, l + 32, ... (amplitudes 2 * piece);
    // piece p = 32 i + l has tile index 2p = 64 i + 2 l
    const uint64_t offl = tc_tile_offset(a, 2 * lane_id);
    uint64_t offs[4];  // 64 i = 256 (i >> 2) + 64 (i & 3)
#pragma unroll
    for (int q = 0; q < 4; ++q) offs[q] = tc_tile_offset(a, 64 * q) + offl;
    auto load = [&](uint64_t s, uint64_t base, int b) {
      float2* S = tiles + b * TC_TILE;
      const float2* src = in + (int64_t)s * a.in_stride + base;
#pragma unroll 8
      for (int i = 0; i < 64; ++i) {
        const int l = 64 * i + 2 * lane_id;
        cp_async16<float>(&S[tc_swz(l)], src + offh[i >> 2] + offs[i & 3]);
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::
                       "r"(tc_smem(&bar_full[b]))
                   : "memory");
    };
    uint64_t s = t0 / tps, base = tc_tile_base(a, t0 % tps);
    uint64_t ls = s, lbase = base;  // next tile to load
    for (uint64_t k = 0; k < 2 && k < ntile; ++k) {
      load(ls, lbase, (int)k);
      lbase = next_base(lbase);
      ls += lbase == 0;
    }
    for (uint64_t k = 0; k < ntile; ++k) {
      const int b = (int)(k & 1);
      if (!tc_wait(tc_smem(&bar_empty[b]), (uint32_t)((k >> 1) & 1))) {
        fail(16);
        break;
      }
      const float2* S = tiles + b * TC_TILE;
      float2* dst = out + (s << a.n) + base;
#pragma unroll 8
      for (int i = 0; i < 64; ++i) {
        const int l = 64 * i + 2 * lane_id;
        const float4 w = *reinterpret_cast<const float4*>(&S[tc_swz(l)]);
        __stcs(reinterpret_cast<float4*>(dst + offh[i >> 2] + offs[i & 3]),
               w);
      }
      __syncwarp();  // every lane's reads done before the buffer refills
      if (k + 2 < ntile) {
        load(ls, lbase, b);
        lbase = next_base(lbase);
        ls += lbase == 0;
      }
      base = next_base(base);
      s += base == 0;
      if (s_abort) break;
    }
    cp_async_wait_all();
  } else if (warp == 4) {
    // -------------------------------------------------------- MMA issuer
    if (lane_id == 0) {
      uint32_t img_phase = 0;  // bit b: parity of the next wait on img[b]
      int img_pending = 0;
      const int first = total_exec < 2 ? (int)total_exec : 2;
      for (int e = 0; e < first; ++e) {
        tc_load_image(tc_smem(imgs + e * TC_IMG_BYTES),
                      a.images + (size_t)sblk[e % nb].mat * TC_IMG_BYTES,
                      tc_smem(&bar_img[e]));
        img_pending |= 1 << e;
      }
      for (uint64_t e = 0; e < total_exec; ++e) {
        const int buf = (int)(e & 1);
        if (!tc_wait(tc_smem(&bar_a), (uint32_t)(e & 1))) {
          fail(32);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        bool ok = true;
        if ((img_pending >> buf) & 1) {
          ok = tc_wait(tc_smem(&bar_img[buf]), (img_phase >> buf) & 1);
          img_pending &= ~(1 << buf);
          img_phase ^= 1u << buf;
        }
        if (ok) {
          // image: [Bl; Bh] as a K = 128 x N = 64 operand (8-row groups
          // 2048 bytes apart); Bh alone starts 1024 bytes in
          const uint32_t im = tc_smem(imgs + buf * TC_IMG_BYTES);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tc_mma<64>(tmem + 64, tmem + 8 * j, tc_desc(im + 1024 + 256 * j),
                       j > 0);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            tc_mma<64>(tmem + 128, tmem + 8 * j, tc_desc(im + 256 * j), j > 0);
          // lo * Bl
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tc_mma<64>(tmem + 128, tmem + 32 + 8 * j, tc_desc(im + 256 * j),
                       1);
        } else {
          fail(1);
        }
        // commit even after a failed wait: it then arrives at once
        asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::"
            "cluster.b64 [%0];" ::"r"(tc_smem(&bar_mma))
            : "memory");
        if (!ok) break;
        if (e + 2 < total_exec) {
          // image buffer `buf` is free once these MMAs complete
          if (!tc_wait(tc_smem(&bar_mma), (uint32_t)(e & 1))) {
            fail(2);
            break;
          }
          tc_load_image(
              tc_smem(imgs + buf * TC_IMG_BYTES),
              a.images + (size_t)sblk[(int)((e + 2) % nb)].mat * TC_IMG_BYTES,
              tc_smem(&bar_img[buf]));
          img_pending |= 1 << buf;
        }
        if (s_abort) break;
      }
      for (int b = 0; b < 2; ++b)
        if ((img_pending >> b) & 1)
          if (!tc_wait(tc_smem(&bar_img[b]), (img_phase >> b) & 1)) fail(4);
    }
  } else {
    // ---------------------------------------------------------- compute
    const uint32_t lane = (uint32_t)(warp * 32) << 16;
    const uint32_t tA = tmem, tD1 = tmem + 64, tDc = tmem + 128;
    uint64_t s = t0 / tps, base = tc_tile_base(a, t0 % tps);
    // A wait that runs out only sets `bad`: every compute thread runs the
    // same tcgen05 and barrier sequence, and all leave together after the
    // reduction barrier that ends each block.
    uint64_t e = 0;
    bool bad = false;
    bool late = false;  // an MMA completion wait ran out
    for (uint64_t k = 0; k < ntile && !bad; ++k) {
      const int b = (int)(k & 1);
      float2* const S = tiles + b * TC_TILE;
      if (!tc_wait(tc_smem(&bar_full[b]), (uint32_t)((k >> 1) & 1))) {
        fail(64);
        bad = true;
      }
      for (int bi = 0; bi < nb; ++bi, ++e) {
        const TcBlock& B = sblk[bi];
        int sb = 0;
#pragma unroll
        for (int j = 0; j < TC_TB; ++j)
          if ((tid >> j) & 1) sb ^= B.tspo[j];
        int rs[TC_RB];
#pragma unroll
        for (int j = 0; j < TC_RB; ++j) rs[j] = B.rspo[j];
        const bool pairs = B.flags & TC_PAIRS;
        // loaded now and used after the MMAs
        const float2 fv = tc_factor(a, B, base, tid);
        float2 v[32];
        tc_gather(S, sb, rs, pairs, v);
        if constexpr (SCALED) tc_columns(a, B, v);
        float sc, inv;
        tc_scale<SCALED>(v, &sc, &inv);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t hi[16], lo[16];
          tc_split<16>(&v[16 * h], sc, hi, lo);
          tc_st16(tA + lane + 16 * h, hi);
          tc_st16(tA + 32 + lane + 16 * h, lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                         tc_smem(&bar_a))
                     : "memory");
        // post-diagonals left in the list (a register bit, or too many
        // outside bits), while the MMAs run
        float2 f = make_float2(fv.x * inv, fv.y * inv);
        const bool has_diag = B.num_diag > 0 || B.fac >= 0;
        const bool regdiag = tc_outer_diags(B, dtab, base, tid, &f);
        if (!tc_wait(tc_smem(&bar_mma), (uint32_t)(e & 1))) {
          fail(2);
          late = true;
          bad = true;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // read back D1 + Dc, undo the scaling, apply the factors
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t d1[32], dc[32];
          tc_ld32(tD1 + lane + 32 * h, d1);
          tc_ld32(tDc + lane + 32 * h, dc);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float re =
                __uint_as_float(d1[2 * j]) + __uint_as_float(dc[2 * j]);
            const float im = __uint_as_float(d1[2 * j + 1]) +
                             __uint_as_float(dc[2 * j + 1]);
            v[16 * h + j] = has_diag ? cmul(f, make_float2(re, im))
                                     : make_float2(re * inv, im * inv);
          }
        }
        if constexpr (SCALED) tc_unscale(v, inv);
        if (regdiag) tc_register_diags(B, dtab, base, tid, v);
        // scatter back (the same addresses the gather read)
        tc_scatter(S, sb, rs, pairs, v);
        // the next block reads other threads' results; errors anywhere
        // stop every compute thread here
        bad = tc_compute_sync_or(bad || s_abort);
        if (bad) break;
      }
      if (bad) break;
      // this thread's part of the tile is final: the storer may take it
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                       tc_smem(&bar_empty[b]))
                   : "memory");
      base = next_base(base);
      s += base == 0;
    }
    if (late && !tc_wait(tc_smem(&bar_mma), (uint32_t)((e & 1)))) fail(8);
  }
  // every role is done (waits are bounded): free tensor memory
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile(
        "tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem)
        : "memory");
  }
}


// The same stage for at most TW_BLOCKS blocks: one CTA per SM with three
// compute warpgroups, which take tiles g, g + 3, ... out of a ring of up to
// six buffers, and a warpgroup that loads and stores the tiles.  The images
// stay in shared memory, one copy per SM.
//
// A stage is bound by the chain of a block (gather, split, tensor-memory
// store, MMA, tensor-memory load, scatter: 4100 cycles alone) and by how
// many chains an SM runs at once; no pipe is above 60%.  tc_stage_kernel
// runs two, and a third does not fit: its two products take 192 tensor-
// memory columns of 512, and images per CTA fill shared memory.  Here a
// group has 128 columns: A in 64, and D1 is read back into registers before
// the correction takes its 64 columns.  Arithmetic and results are those of
// tc_stage_kernel.
//
// 120 gates on 26 qubits: 1890 -> 1665 us (1770 -> 1570 another circuit),
// 60 gates on 16 states of 20: 297 -> 251 us, 200 gates on 22: 229 ->
// 194 us.  Slower: four groups of 112 registers (spills, 2170 us), A in
// shared memory instead of tensor memory (1750 us: gather, scatter and the
// tile copies already use that path), a separate MMA warp (1760 us), hi and
// lo split apart so that the first product runs under the second (1800 us).
constexpr int TW_GROUPS = 3;
constexpr int TW_LOADERS = 128;
constexpr int TW_THREADS = TW_GROUPS * TC_THREADS + TW_LOADERS;
constexpr int TW_LOAD_REGS = 56;   // of 128 at launch: 3 * 152 + 56 = 4 * 128
constexpr int TW_CALC_REGS = 152;
constexpr int TW_BUFS = 6;
constexpr int TW_BLOCKS = 8;
constexpr int TW_SDIAG = 24;
constexpr int TW_SMEM_BYTES = 14 * TC_IMG_BYTES;  // images and tile buffers

// Tile buffers beside nb images: six for one or two blocks, at least three.
__host__ __device__ constexpr int tw_bufs(int nb) {
  const int b = (14 - nb) / 2;
  return b < TW_BUFS ? b : TW_BUFS;
}

// Barrier `id` over a warpgroup; the second form returns the OR of x.
__device__ __forceinline__ void tw_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(TC_THREADS) : "memory");
}
__device__ __forceinline__ bool tw_sync_or(int id, bool x) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)x), "r"(id), "n"(TC_THREADS)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void tc_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
      "r"(r[6]), "r"(r[7])
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::"
      "cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

template <bool SCALED>
__global__ void __launch_bounds__(TW_THREADS, 1)
    tc_wide_kernel(const float2* in, float2* out,
                   const __grid_constant__ TcArgs a) {
  extern __shared__ __align__(1024) unsigned char tw_smem[];
  __shared__ TcBlock sblk[TW_BLOCKS];
  __shared__ TcDiag sdiag[TW_SDIAG];
  __shared__ uint64_t offh[16];
  __shared__ __align__(8) uint64_t bar_full[TW_BUFS], bar_empty[TW_BUFS];
  __shared__ __align__(8) uint64_t bar_mma[TW_GROUPS], bar_img;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;

  const int nb = a.num_blocks;
  const int nbuf = tw_bufs(nb);
  unsigned char* const imgs = tw_smem;
  float2* const tiles =
      reinterpret_cast<float2*>(tw_smem + nb * TC_IMG_BYTES);
  const int warp = threadIdx.x >> 5;
  const uint64_t tps = uint64_t(1) << (a.n - TC_M);
  const uint64_t num_tiles = (uint64_t)a.num_states * tps;
  const uint64_t t0 = (uint64_t)blockIdx.x * num_tiles / gridDim.x;
  const uint64_t t1 = (uint64_t)(blockIdx.x + 1) * num_tiles / gridDim.x;
  if (t0 >= t1) return;
  const uint64_t ntile = t1 - t0;

  if (warp == 0) {
    asm volatile(
        "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::
            "r"(tc_smem(&s_tmem))
        : "memory");
    asm volatile(
        "tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::
            : "memory");
  }
  if (threadIdx.x == 0) {
    auto init = [](uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(
                       tc_smem(bar)),
                   "r"(count));
    };
    for (int b = 0; b < TW_BUFS; ++b) {
      init(&bar_full[b], TW_LOADERS);
      init(&bar_empty[b], TC_THREADS);
    }
    for (int g = 0; g < TW_GROUPS; ++g) init(&bar_mma[g], 1);
    init(&bar_img, nb);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int i = threadIdx.x; i < nb * 16; i += TW_THREADS)
    reinterpret_cast<int32_t*>(sblk)[i] =
        reinterpret_cast<const int32_t*>(a.blocks)[i];
  const int dfirst = a.blocks[0].first_diag;
  const int dcount =
      a.blocks[nb - 1].first_diag + a.blocks[nb - 1].num_diag - dfirst;
  const bool dshared = dcount <= TW_SDIAG;
  if (dshared)
    for (int i = threadIdx.x; i < dcount * 12; i += TW_THREADS)
      reinterpret_cast<int32_t*>(sdiag)[i] =
          reinterpret_cast<const int32_t*>(a.diags + dfirst)[i];
  const TcDiag* const dtab = dshared ? sdiag - dfirst : a.diags;
  if (threadIdx.x < 16)
    offh[threadIdx.x] = tc_tile_offset(a, 256 * threadIdx.x);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  uint64_t tmask = ~((uint64_t(1) << a.n) - 1);
  for (int j = 0; j < TC_M; ++j) tmask |= uint64_t(1) << a.spos[j];
  auto next_base = [&](uint64_t b) { return ((b | tmask) + 1) & ~tmask; };
  auto fail = [&](int code) {
    s_abort = 1;
    atomicOr(&g_tc_status, code);
  };

  if (warp >= TW_GROUPS * 4) {
    // --------------------------------------------- tile loaders / storers
    // lane L of 128 moves 16-byte pieces L, L + 128, ...
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TW_LOAD_REGS));
    const int L = threadIdx.x - TW_GROUPS * TC_THREADS;
    if (L == 0)  // bar_img expects one arrival per image
      for (int e = 0; e < nb; ++e)
        tc_load_image(tc_smem(imgs + e * TC_IMG_BYTES),
                      a.images + (size_t)sblk[e].mat * TC_IMG_BYTES,
                      tc_smem(&bar_img));
    const uint64_t off0 = tc_tile_offset(a, 2 * L);
    auto load = [&](uint64_t s, uint64_t base, int b) {
      float2* S = tiles + b * TC_TILE;
      const float2* src = in + (int64_t)s * a.in_stride + base + off0;
#pragma unroll 4
      for (int i = 0; i < 16; ++i)
        cp_async16<float>(&S[tc_swz(256 * i + 2 * L)], src + offh[i]);
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::
                       "r"(tc_smem(&bar_full[b]))
                   : "memory");
    };
    uint64_t s = t0 / tps, base = tc_tile_base(a, t0 % tps);
    uint64_t ls = s, lbase = base;  // next tile to load
    for (int k = 0; k < nbuf && k < ntile; ++k) {
      load(ls, lbase, k);
      lbase = next_base(lbase);
      ls += lbase == 0;
    }
    int b = 0;
    uint32_t ph = 0;
    for (uint64_t k = 0; k < ntile; ++k) {
      if (!tc_wait(tc_smem(&bar_empty[b]), ph)) {
        fail(16);
        break;
      }
      const float2* S = tiles + b * TC_TILE;
      float2* dst = out + (s << a.n) + base + off0;
#pragma unroll 4
      for (int i = 0; i < 16; ++i) {
        const float4 w =
            *reinterpret_cast<const float4*>(&S[tc_swz(256 * i + 2 * L)]);
        __stcs(reinterpret_cast<float4*>(dst + offh[i]), w);
      }
      __syncwarp();  // every lane's reads done before the buffer refills
      if (k + nbuf < ntile) {
        load(ls, lbase, b);
        lbase = next_base(lbase);
        ls += lbase == 0;
      }
      base = next_base(base);
      s += base == 0;
      if (++b == nbuf) {
        b = 0;
        ph ^= 1;
      }
      if (s_abort) break;
    }
    cp_async_wait_all();
    // the images have landed before the CTA can end
    if (L == 0 && !tc_wait(tc_smem(&bar_img), 0)) fail(4);
  } else {
    // ---------------------------------------------------------- compute
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TW_CALC_REGS));
    const int g = warp >> 2;
    const int tid = threadIdx.x & (TC_THREADS - 1);
    const uint32_t tmem = s_tmem + 128 * g;
    const uint32_t lane = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tA = tmem + lane, tD = tmem + 64 + lane;
    const uint32_t bar = tc_smem(&bar_mma[g]);
    uint32_t par = 0;  // parity of the group's next MMA wait
    uint64_t base = tc_tile_base(a, t0 % tps);
    for (int j = 0; j < g; ++j) base = next_base(base);
    bool bad = false, late = false, image = false;
    int b = g % nbuf;
    uint32_t ph = g >= nbuf;
    // As in tc_stage_kernel a wait that runs out only sets `bad`, and the
    // group leaves together after the barrier that ends each block.
    for (uint64_t k = g; k < ntile && !bad; k += TW_GROUPS) {
      float2* const S = tiles + b * TC_TILE;
      if (!tc_wait(tc_smem(&bar_full[b]), ph)) {
        fail(64);
        bad = true;
      }
      for (int bi = 0; bi < nb; ++bi) {
        const TcBlock& B = sblk[bi];
        int sb = 0;
#pragma unroll
        for (int j = 0; j < TC_TB; ++j)
          if ((tid >> j) & 1) sb ^= B.tspo[j];
        int rs[TC_RB];
#pragma unroll
        for (int j = 0; j < TC_RB; ++j) rs[j] = B.rspo[j];
        const bool pairs = B.flags & TC_PAIRS;
        const float2 fv = tc_factor(a, B, base, tid);
        float2 v[32];
        tc_gather(S, sb, rs, pairs, v);
        if constexpr (SCALED) tc_columns(a, B, v);
        float sc, inv;
        tc_scale<SCALED>(v, &sc, &inv);
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          uint32_t hi[8], lo[8];
          tc_split<8>(&v[8 * h], sc, hi, lo);
          tc_st8(tA + 8 * h, hi);
          tc_st8(tA + 32 + 8 * h, lo);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        tw_sync(1 + g);
        // D1 = hi * Bh; each group's issuer sits on its own scheduler
        const uint32_t im = tc_smem(imgs + bi * TC_IMG_BYTES);
        if (tid == 32 * g) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (!image && !tc_wait(tc_smem(&bar_img), 0)) fail(1);
          image = true;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tc_mma<64>(tmem + 64, tmem + 8 * j, tc_desc(im + 1024 + 256 * j),
                       j > 0);
          tc_commit(bar);
        }
        __syncwarp();
        float2 f = make_float2(fv.x * inv, fv.y * inv);
        const bool has_diag = B.num_diag > 0 || B.fac >= 0;
        const bool regdiag = tc_outer_diags(B, dtab, base, tid, &f);
        auto finished = [&]() {
          if (!tc_wait(bar, par)) {
            fail(2);
            late = true;
            bad = true;
          }
          par ^= 1;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        };
        finished();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t d[32];
          tc_ld32(tD + 32 * h, d);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j)
            v[16 * h + j] = make_float2(__uint_as_float(d[2 * j]),
                                        __uint_as_float(d[2 * j + 1]));
        }
        // the correction, in D1's columns
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        tw_sync(1 + g);
        if (tid == 32 * g) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j)
            tc_mma<64>(tmem + 64, tmem + 8 * j, tc_desc(im + 256 * j), j > 0);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            tc_mma<64>(tmem + 64, tmem + 32 + 8 * j, tc_desc(im + 256 * j),
                       1);
          tc_commit(bar);
        }
        __syncwarp();
        finished();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t d[32];
          tc_ld32(tD + 32 * h, d);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float re = v[16 * h + j].x + __uint_as_float(d[2 * j]);
            const float im = v[16 * h + j].y + __uint_as_float(d[2 * j + 1]);
            v[16 * h + j] = has_diag ? cmul(f, make_float2(re, im))
                                    : make_float2(re * inv, im * inv);
          }
        }
        if constexpr (SCALED) tc_unscale(v, inv);
        if (regdiag) tc_register_diags(B, dtab, base, tid, v);
        tc_scatter(S, sb, rs, pairs, v);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        bad = tw_sync_or(1 + g, bad || s_abort);
        if (bad) break;
      }
      if (bad) break;
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(
                       tc_smem(&bar_empty[b]))
                   : "memory");
#pragma unroll
      for (int j = 0; j < TW_GROUPS; ++j) base = next_base(base);
      b += TW_GROUPS;
      if (b >= nbuf) {
        b -= nbuf;
        ph ^= 1;
      }
    }
    if (late && !tc_wait(bar, par ^ 1)) fail(8);
  }
  // every role is done (waits are bounded): free tensor memory
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile(
        "tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(s_tmem)
        : "memory");
  }
}

}  // namespace gbsv

using gbsv::set_error;

template <bool SCALED>
static int run_stage_tc(const void* state_in, void* state_out, int dtype,
                        int n, int64_t num_states, int64_t in_stride, int m,
                        int c, const int32_t* positions, const void* blocks,
                        int num_blocks, const void* diags, const void* images,
                        const void* factors, void* stream) {
  using namespace gbsv;
  if (dtype != GBSV_C64)
    return set_error(GBSV_ERR_UNSUPPORTED,
                     "tensor-core stages are complex64 only");
  if (m != TC_M)
    return set_error(GBSV_ERR_INVALID_ARG, "tensor-core stages use %d tile "
                     "bits, got %d", TC_M, m);
  if (n < TC_M || n > 40)
    return set_error(GBSV_ERR_INVALID_ARG, "need %d..40 qubits, got %d", TC_M,
                     n);
  if (num_blocks < 1 || num_blocks > TC_MAX_BLOCKS)
    return set_error(GBSV_ERR_INVALID_ARG, "num_blocks %d not in 1..%d",
                     num_blocks, TC_MAX_BLOCKS);
  if (c < 1 || c > TC_M)
    return set_error(GBSV_ERR_INVALID_ARG, "contiguous bits %d not in 1..%d",
                     c, TC_M);
  if (num_states < 0) return set_error(GBSV_ERR_INVALID_ARG, "num_states < 0");
  if (num_states == 0) return GBSV_OK;
  if (!state_in || !state_out || !positions || !blocks || !images)
    return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  if ((reinterpret_cast<uintptr_t>(state_in) |
       reinterpret_cast<uintptr_t>(state_out) |
       reinterpret_cast<uintptr_t>(images)) & 15)
    return set_error(GBSV_ERR_INVALID_ARG, "states and images must be "
                     "16-byte aligned");
  TcArgs a{};
  a.n = n;
  a.c = c;
  a.num_blocks = num_blocks;
  a.num_states = num_states;
  a.in_stride = in_stride;
  uint64_t seen = 0;
  for (int j = 0; j < TC_M; ++j) {
    const int p = positions[j];
    if (p < 0 || p >= n || ((seen >> p) & 1))
      return set_error(GBSV_ERR_INVALID_ARG, "bad tile position %d", p);
    if (j < c && p != j)
      return set_error(GBSV_ERR_INVALID_ARG,
                       "tile bit %d must be position %d", j, j);
    seen |= uint64_t(1) << p;
    a.spos[j] = p;
    if (j >= c) a.hpos[j - c] = p;
  }
  for (int i = 1; i < TC_M; ++i)
    for (int j = i; j > 0 && a.spos[j - 1] > a.spos[j]; --j) {
      const int tmp = a.spos[j];
      a.spos[j] = a.spos[j - 1];
      a.spos[j - 1] = tmp;
    }
  a.blocks = static_cast<const TcBlock*>(blocks);
  a.diags = static_cast<const TcDiag*>(diags);
  a.images = static_cast<const unsigned char*>(images);
  a.factors = static_cast<const float2*>(factors);
  const uint64_t tiles =
      (uint64_t)num_states << (n - TC_M);
  // up to TW_BLOCKS images stay in shared memory beside three tile buffers;
  // longer stages stream them
  if (num_blocks <= TW_BLOCKS) {
    static OncePerDevice once;
    const int rc = allow_smem(once, tc_wide_kernel<SCALED>, TW_SMEM_BYTES,
                              "tc_wide_kernel");
    if (rc) return rc;
    const uint64_t grid = std::min<uint64_t>(tiles, (uint64_t)sm_count());
    tc_wide_kernel<SCALED><<<(unsigned)grid, TW_THREADS, TW_SMEM_BYTES,
                             static_cast<cudaStream_t>(stream)>>>(
        static_cast<const float2*>(state_in),
        static_cast<float2*>(state_out), a);
    return after_launch("tc_wide_kernel");
  }
  static OncePerDevice once;
  const int rc = allow_smem(once, tc_stage_kernel<SCALED>, TC_SMEM_BYTES,
                            "tc_stage_kernel");
  if (rc) return rc;
  const uint64_t grid = std::min<uint64_t>(tiles, (uint64_t)sm_count() * 2);
  tc_stage_kernel<SCALED><<<(unsigned)grid, TC_ROLE_THREADS, TC_SMEM_BYTES,
                            static_cast<cudaStream_t>(stream)>>>(
      static_cast<const float2*>(state_in), static_cast<float2*>(state_out),
      a);
  return after_launch("tc_stage_kernel");
}

extern "C" int gbsv_run_stage_tc(
    const void* state_in, void* state_out, int dtype, int n,
    int64_t num_states, int64_t in_stride, int m, int c,
    const int32_t* positions, const void* blocks, int num_blocks,
    const void* diags, const void* images, const void* factors,
    void* stream) {
  return run_stage_tc<false>(state_in, state_out, dtype, n, num_states,
                       in_stride, m, c, positions, blocks, num_blocks,
                       diags, images, factors, stream);
}

extern "C" int gbsv_run_stage_tc_scaled(
    const void* state_in, void* state_out, int dtype, int n,
    int64_t num_states, int64_t in_stride, int m, int c,
    const int32_t* positions, const void* blocks, int num_blocks,
    const void* diags, const void* images, const void* factors,
    void* stream) {
  return run_stage_tc<true>(state_in, state_out, dtype, n, num_states,
                      in_stride, m, c, positions, blocks, num_blocks,
                      diags, images, factors, stream);
}

extern "C" int gbsv_tc_status(int* status, int clear) {
  if (!status) return set_error(GBSV_ERR_INVALID_ARG, "null pointer");
  cudaError_t e = cudaMemcpyFromSymbol(status, gbsv::g_tc_status, sizeof(int));
  if (e != cudaSuccess)
    return set_error(GBSV_ERR_CUDA, "tc status: %s", cudaGetErrorString(e));
  if (clear) {
    const int zero = 0;
    e = cudaMemcpyToSymbol(gbsv::g_tc_status, &zero, sizeof(int));
    if (e != cudaSuccess)
      return set_error(GBSV_ERR_CUDA, "tc status: %s", cudaGetErrorString(e));
  }
  return GBSV_OK;
}
