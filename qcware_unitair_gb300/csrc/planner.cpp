// Host-side circuit planner: gate list -> fused stages, register layouts,
// gate records and the matrix pool, ready for one transfer to the device.
//
// It follows the same rules as the Python reference implementation in
// fusion.py (plan, _plan_layouts, _record, _layout_record); a CPU test
// checks that both produce identical bytes.  Stages: greedy in circuit
// order, each owning m tile bits of which the lowest c_min are always
// present; a gate needs its dense target bits (a controlled-U only its
// target, a diagonal nothing).  Layouts: greedy groups of a stage's gates
// whose register-needing bits fit rb register bits.
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <complex>
#include <vector>

#include "gbsv.h"

namespace {

using cd = std::complex<double>;

enum { K_DENSE = 0, K_DIAG = 1, K_CTRL = 2 };
enum {
  FG_DENSE1 = 0, FG_DENSE2 = 1, FG_DIAG = 2, FG_CDENSE1 = 3, FG_REAL1 = 4,
  FG_ANTI1 = 5, FG_CANTI1 = 6, FG_PERM2 = 7, FG_RDIAG = 8
};

struct Ctx {
  const gbsv_gate_desc_t* g;
  const cd* mats;
  int n, m, c_min, rb;
};

int pos_of(const Ctx& c, int q) { return c.n - 1 - q; }

// element (r, col) of batch entry b of gate gi's d x d matrix
cd el(const Ctx& c, int gi, int b, int r, int col) {
  const gbsv_gate_desc_t& d = c.g[gi];
  const int dim = 1 << d.nq;
  return c.mats[d.mat + (int64_t)b * d.mat_bstride + r * dim + col];
}

int batch_of(const gbsv_gate_desc_t& d) {
  return d.mat_bstride > 0 ? (int)d.num_batch : 1;
}

// 2x2 block (r0.., c0..) predicates over every batch entry
bool all_b(const Ctx& c, int gi, bool (*pred)(const Ctx&, int, int, int),
           int off) {
  for (int b = 0; b < batch_of(c.g[gi]); ++b)
    if (!pred(c, gi, b, off)) return false;
  return true;
}
bool anti_p(const Ctx& c, int gi, int b, int o) {
  return el(c, gi, b, o, o) == cd(0) && el(c, gi, b, o + 1, o + 1) == cd(0);
}
bool unit_p(const Ctx& c, int gi, int b, int o) {
  return el(c, gi, b, o, o + 1) == cd(1) && el(c, gi, b, o + 1, o) == cd(1);
}
bool real_p(const Ctx& c, int gi, int b, int o) {
  for (int r = 0; r < 2; ++r)
    for (int k = 0; k < 2; ++k)
      if (el(c, gi, b, o + r, o + k).imag() != 0) return false;
  return true;
}

// kind and flag for a 2x2 (offset o = 0 for a 1-qubit gate, 2 for the U
// block of a controlled gate)
void dense1_kind(const Ctx& c, int gi, int o, int* kind, int* flag) {
  if (all_b(c, gi, anti_p, o)) {
    *kind = FG_ANTI1;
    *flag = all_b(c, gi, unit_p, o) ? 1 : 0;
  } else if (all_b(c, gi, real_p, o)) {
    *kind = FG_REAL1;
    *flag = 0;
  } else {
    *kind = FG_DENSE1;
    *flag = 0;
  }
}

int perm_code(const Ctx& c, int gi) {
  const int B = batch_of(c.g[gi]);
  int code = 0;
  for (int r = 0; r < 4; ++r) {
    int src = -1;
    for (int col = 0; col < 4; ++col) {
      bool one = true, zero = true;
      for (int b = 0; b < B; ++b) {
        const cd v = el(c, gi, b, r, col);
        if (v != cd(1)) one = false;
        if (v != cd(0)) zero = false;
        if (v != cd(0) && v != cd(1)) return -1;
      }
      if (one) {
        if (src >= 0) return -1;
        src = col;
      } else if (!zero) {
        return -1;
      }
    }
    if (src < 0) return -1;
    code |= src << (2 * r);
  }
  return code;
}

// needed tile bits (positions) of a gate, or -1 when it cannot be staged
int64_t needs(const Ctx& c, int gi) {
  const gbsv_gate_desc_t& d = c.g[gi];
  if (d.nq > 2) return -1;
  const int p0 = pos_of(c, d.q0);
  const int p1 = d.nq == 2 ? pos_of(c, d.q1) : 0;
  if (d.kind == K_DIAG) return 0;
  if (d.kind == K_CTRL && d.nq == 2) return int64_t(1) << p1;
  int64_t s = int64_t(1) << p0;
  if (d.nq == 2) s |= int64_t(1) << p1;
  return s;
}

int popc(uint64_t x) { return __builtin_popcountll(x); }

struct Out {
  gbsv_plan_t* p;
  int num_ops = 0, num_records = 0, num_layouts = 0;
  int64_t pool_len = 0;
  bool overflow = false;
};

gbsv_fused_gate_t* new_record(Out& o) {
  if (o.num_records >= o.p->max_records) {
    o.overflow = true;
    return nullptr;
  }
  gbsv_fused_gate_t* r = &o.p->records[o.num_records++];
  memset(r, 0, sizeof(*r));
  return r;
}

// append the values of gate gi (rows r0.., cols c0.., diagonal or block)
// for every batch entry; returns (offset, bstride)
void add_pool(Out& o, const Ctx& c, int gi, int which, int nvals,
              gbsv_fused_gate_t* rec) {
  const gbsv_gate_desc_t& d = c.g[gi];
  const int B = batch_of(d);
  const int dim = 1 << d.nq;
  if (o.pool_len + (int64_t)B * nvals > o.p->max_pool) {
    o.overflow = true;
    return;
  }
  rec->mat = o.pool_len;
  rec->mat_bstride = d.mat_bstride > 0 ? nvals : 0;
  for (int b = 0; b < B; ++b) {
    for (int k = 0; k < nvals; ++k) {
      cd v;
      if (which == 0) {  // whole matrix, row-major
        v = el(c, gi, b, k / dim, k % dim);
      } else if (which == 1) {  // diagonal
        v = el(c, gi, b, k, k);
      } else {  // lower-right 2x2 block of a 4x4
        v = el(c, gi, b, 2 + k / 2, 2 + k % 2);
      }
      const int64_t at = o.pool_len + (int64_t)b * nvals + k;
      if (o.p->dtype == GBSV_C64) {
        static_cast<float*>(o.p->pool)[2 * at] = (float)v.real();
        static_cast<float*>(o.p->pool)[2 * at + 1] = (float)v.imag();
      } else {
        static_cast<double*>(o.p->pool)[2 * at] = v.real();
        static_cast<double*>(o.p->pool)[2 * at + 1] = v.imag();
      }
    }
  }
  o.pool_len += (int64_t)B * nvals;
}

// gate record for a shared-memory stage (tile bits = local indices)
void plain_record(Out& o, const Ctx& c, int gi, const int* local) {
  const gbsv_gate_desc_t& d = c.g[gi];
  gbsv_fused_gate_t* r = new_record(o);
  if (!r) return;
  const int p0 = pos_of(c, d.q0);
  const int p1 = d.nq == 2 ? pos_of(c, d.q1) : 0;
  if (d.kind == K_DIAG) {
    r->kind = FG_DIAG;
    r->nq = d.nq;
    r->b0 = local[p0] >= 0 ? local[p0] : -1 - p0;
    r->b1 = d.nq == 2 ? (local[p1] >= 0 ? local[p1] : -1 - p1) : 0;
    add_pool(o, c, gi, 1, 1 << d.nq, r);
  } else if (d.kind == K_CTRL && local[p0] < 0) {
    r->kind = FG_DENSE1;
    r->b0 = local[p1];
    r->cmask = r->cval = uint64_t(1) << p0;
    add_pool(o, c, gi, 2, 4, r);
  } else if (d.nq == 1) {
    r->kind = FG_DENSE1;
    r->b0 = local[p0];
    add_pool(o, c, gi, 0, 4, r);
  } else {
    r->kind = FG_DENSE2;
    r->b0 = local[p0];
    r->b1 = local[p1];
    add_pool(o, c, gi, 0, 16, r);
  }
}

// gate record for a register-blocked stage; kreg[tile bit] = register bit
void layout_record(Out& o, const Ctx& c, int gi, const int* local,
                   const int* kreg) {
  const gbsv_gate_desc_t& d = c.g[gi];
  gbsv_fused_gate_t* r = new_record(o);
  if (!r) return;
  const int p0 = pos_of(c, d.q0);
  const int p1 = d.nq == 2 ? pos_of(c, d.q1) : 0;
  auto enc = [&](int p) {
    if (local[p] < 0) return -1 - p;
    if (kreg[local[p]] >= 0) return kreg[local[p]];
    return c.rb + local[p];
  };
  if (d.kind == K_DIAG) {
    r->kind = FG_RDIAG;
    r->nq = d.nq;
    r->b0 = enc(p0);
    r->b1 = d.nq == 2 ? enc(p1) : 0;
    add_pool(o, c, gi, 1, 1 << d.nq, r);
    return;
  }
  if (d.kind == K_CTRL && d.nq == 2) {
    const int t = local[p1];
    if (local[p0] < 0) {
      int kind, flag;
      dense1_kind(c, gi, 2, &kind, &flag);
      r->kind = kind;
      r->nq = flag;
      r->b0 = kreg[t];
      r->cmask = r->cval = uint64_t(1) << p0;
      add_pool(o, c, gi, 2, 4, r);
      return;
    }
    if (kreg[local[p0]] < 0) {
      if (all_b(c, gi, anti_p, 2)) {
        r->kind = FG_CANTI1;
        r->nq = all_b(c, gi, unit_p, 2) ? 1 : 0;
      } else {
        r->kind = FG_CDENSE1;
      }
      r->b0 = kreg[t];
      r->b1 = local[p0];
      add_pool(o, c, gi, 2, 4, r);
      return;
    }
  }
  if (d.nq == 1) {
    int kind, flag;
    dense1_kind(c, gi, 0, &kind, &flag);
    r->kind = kind;
    r->nq = flag;
    r->b0 = kreg[local[p0]];
    add_pool(o, c, gi, 0, 4, r);
    return;
  }
  const int code = perm_code(c, gi);
  r->b0 = kreg[local[p0]];
  r->b1 = kreg[local[p1]];
  if (code >= 0) {
    r->kind = FG_PERM2;
    r->nq = code;
  } else {
    r->kind = FG_DENSE2;
  }
  add_pool(o, c, gi, 0, 16, r);
}

void emit_stage(Out& o, const Ctx& c, uint64_t tile,
                const std::vector<int>& gates, bool layouts) {
  // top up to m bits with the lowest free positions
  for (int p = 0; popc(tile) < c.m; ++p) tile |= uint64_t(1) << p;
  int cc = 0;
  while ((tile >> cc) & 1) ++cc;
  cc = std::min(cc, c.m);
  int order[64], local[64];
  int no = 0;
  for (int p = 0; p < cc; ++p) order[no++] = p;
  for (int p = cc; p < c.n; ++p)
    if ((tile >> p) & 1) order[no++] = p;
  for (int p = 0; p < 64; ++p) local[p] = -1;
  for (int i = 0; i < no; ++i) local[order[i]] = i;
  if (o.num_ops >= o.p->max_ops) {
    o.overflow = true;
    return;
  }
  gbsv_plan_op_t* op = &o.p->ops[o.num_ops++];
  memset(op, 0, sizeof(*op));
  op->contiguous = cc;
  for (int i = 0; i < c.m; ++i) op->positions[i] = order[i];
  if (!layouts) {
    op->type = 1;
    op->first = o.num_records;
    for (int gi : gates) plain_record(o, c, gi, local);
    op->count = o.num_records - op->first;
    return;
  }
  op->type = 2;
  op->first = o.num_layouts;
  // group into register layouts
  std::vector<std::pair<uint64_t, std::vector<int>>> groups;
  uint64_t need_all = 0;
  std::vector<int> cur;
  for (int gi : gates) {
    const gbsv_gate_desc_t& d = c.g[gi];
    uint64_t need = 0;
    if (d.kind == K_DIAG) {
      need = 0;
    } else if (d.kind == K_CTRL && d.nq == 2) {
      need = uint64_t(1) << local[pos_of(c, d.q1)];
    } else {
      need = uint64_t(1) << local[pos_of(c, d.q0)];
      if (d.nq == 2) need |= uint64_t(1) << local[pos_of(c, d.q1)];
    }
    if (popc(need_all | need) <= c.rb) {
      need_all |= need;
      cur.push_back(gi);
    } else {
      groups.emplace_back(need_all, cur);
      need_all = need;
      cur.assign(1, gi);
    }
  }
  groups.emplace_back(need_all, cur);
  for (auto& grp : groups) {
    if (o.num_layouts >= o.p->max_layouts) {
      o.overflow = true;
      return;
    }
    int bits[8], nb = 0;
    for (int b = 0; b < c.m; ++b)
      if ((grp.first >> b) & 1) bits[nb++] = b;
    for (int b = c.m - 1; nb < c.rb; --b)
      if (!((grp.first >> b) & 1)) bits[nb++] = b;
    int kreg[64];
    for (int i = 0; i < 64; ++i) kreg[i] = -1;
    for (int k = 0; k < c.rb; ++k) kreg[bits[k]] = k;
    gbsv_layout_t* L = &o.p->layouts[o.num_layouts++];
    memset(L, 0, sizeof(*L));
    for (int k = 0; k < c.rb; ++k) L->rb[k] = bits[k];
    L->first_gate = o.num_records;
    for (int gi : grp.second) layout_record(o, c, gi, local, kreg);
    L->num_gates = o.num_records - L->first_gate;
  }
  op->count = o.num_layouts - op->first;
}

}  // namespace

extern "C" int gbsv_plan(const gbsv_gate_desc_t* gates, int num_gates,
                         const void* matrices, int num_qubits,
                         int tile_qubits, int min_contiguous,
                         int register_bits, int fuse, gbsv_plan_t* plan) {
  if (!plan || (num_gates > 0 && (!gates || !matrices)))
    return GBSV_ERR_INVALID_ARG;
  const int n = num_qubits, m = tile_qubits;
  if (n < 1 || n > 62 || m < 1 || m > n || m > 14 || min_contiguous < 0 ||
      register_bits < 0 || register_bits > 5 ||
      (plan->dtype != GBSV_C64 && plan->dtype != GBSV_C128))
    return GBSV_ERR_INVALID_ARG;
  for (int i = 0; i < num_gates; ++i) {
    const gbsv_gate_desc_t& d = gates[i];
    if (d.nq < 1 || d.nq > 12 || d.q0 < 0 || d.q0 >= n ||
        (d.nq == 2 && (d.q1 < 0 || d.q1 >= n || d.q1 == d.q0)) ||
        d.kind < 0 || d.kind > 2 || d.mat < 0 || d.mat_bstride < 0)
      return GBSV_ERR_INVALID_ARG;
  }
  Ctx c{gates, static_cast<const cd*>(matrices), n, m,
        std::min(min_contiguous, m), register_bits};
  Out o;
  o.p = plan;
  const bool layouts =
      register_bits >= 1 && register_bits <= m && m <= register_bits + 9;
  const uint64_t low = c.c_min >= 64 ? ~0ull : ((uint64_t(1) << c.c_min) - 1);
  bool have = false;
  uint64_t tile = 0;
  std::vector<int> cur;
  auto close = [&]() {
    if (have) emit_stage(o, c, tile, cur, layouts);
    have = false;
    cur.clear();
  };
  for (int gi = 0; gi < num_gates && !o.overflow; ++gi) {
    int64_t need = fuse ? needs(c, gi) : -1;
    if (need >= 0 && popc(low | (uint64_t)need) > m) need = -1;
    if (need < 0) {
      close();
      if (o.num_ops >= plan->max_ops) {
        o.overflow = true;
        break;
      }
      gbsv_plan_op_t* op = &plan->ops[o.num_ops++];
      memset(op, 0, sizeof(*op));
      op->type = 0;
      op->first = gi;
      op->count = 1;
      continue;
    }
    if (!have) {
      have = true;
      tile = low;
    }
    if (popc(tile | (uint64_t)need) <= m) {
      tile |= (uint64_t)need;
      cur.push_back(gi);
    } else {
      close();
      have = true;
      tile = low | (uint64_t)need;
      cur.push_back(gi);
    }
  }
  close();
  if (o.overflow) return GBSV_ERR_SCRATCH;
  plan->num_ops = o.num_ops;
  plan->num_records = o.num_records;
  plan->num_layouts = o.num_layouts;
  plan->pool_len = o.pool_len;
  plan->used_layouts = layouts ? 1 : 0;
  return GBSV_OK;
}

// ---- register layouts of backward stages ----------------------------------
namespace {

// gbsv_adjoint_op_t as the stage entry points lay it out
struct HostAdjOp {
  int32_t kind, gen, bit, slot, pidx, pad_;
  double scale;
  gbsv_fused_gate_t g;
};
static_assert(sizeof(HostAdjOp) == 80, "gbsv_adjoint_op_t is 80 bytes");

struct PoolView {
  const void* p;
  int dtype;
  cd at(int64_t i) const {
    if (dtype == GBSV_C64) {
      const float* f = static_cast<const float*>(p) + 2 * i;
      return cd(f[0], f[1]);
    }
    const double* f = static_cast<const double*>(p) + 2 * i;
    return cd(f[0], f[1]);
  }
};

// diag(I, U) on two qubits, the first controlling
bool controlled(const PoolView& v, int64_t mat) {
  if (!v.p) return false;
  for (int r = 0; r < 4; ++r)
    for (int c = 0; c < 4; ++c) {
      if (r >= 2 && c >= 2) continue;
      if (v.at(mat + 4 * r + c) != cd(r == c ? 1.0 : 0.0)) return false;
    }
  return true;
}

}  // namespace

extern "C" int gbsv_adjoint_layouts(const void* ops, int num_ops,
                                    int tile_qubits, int register_bits,
                                    const void* pool, int dtype,
                                    gbsv_adjoint_regop_t* regops,
                                    int* num_regops,
                                    gbsv_adjoint_layout_t* layouts,
                                    int max_layouts, int* num_layouts) {
  const int m = tile_qubits, rb = register_bits;
  if (num_ops < 0 || !num_layouts || !num_regops || rb < 2 || rb > 4 || m < rb ||
      m - rb > 12 || (dtype != GBSV_C64 && dtype != GBSV_C128) ||
      (num_ops > 0 && (!ops || !regops || !layouts)))
    return GBSV_ERR_INVALID_ARG;
  const HostAdjOp* in = static_cast<const HostAdjOp*>(ops);
  const PoolView view{pool, dtype};
  *num_layouts = *num_regops = 0;
  struct Info {
    uint32_t need;     // tile bits that must be register bits
    uint32_t touch;    // tile bits it acts on
    bool diag, ctrl;
  };
  std::vector<Info> info(num_ops);
  for (int i = 0; i < num_ops; ++i) {
    const HostAdjOp& o = in[i];
    Info& f = info[i];
    f = Info{0, 0, false, false};
    auto bit = [](int b) { return b >= 0 ? 1u << b : 0u; };
    if (o.kind == 0) {
      f.touch = bit(o.bit);
      f.diag = o.gen == 2;
      f.need = f.diag ? 0u : f.touch;
    } else if (o.g.mat_bstride != 0) {
      return GBSV_ERR_UNSUPPORTED;
    } else if (o.g.kind == 2) {
      f.touch = bit(o.g.b0) | (o.g.nq > 1 ? bit(o.g.b1) : 0u);
      f.diag = true;
    } else if (o.g.kind == 1) {
      f.touch = bit(o.g.b0) | bit(o.g.b1);
      f.ctrl = controlled(view, o.g.mat);
      f.need = f.ctrl ? bit(o.g.b1) : f.touch;
    } else if (o.g.kind == 0) {
      f.touch = f.need = bit(o.g.b0);
    } else {
      return GBSV_ERR_UNSUPPORTED;
    }
  }
  std::vector<char> done(num_ops, 0);
  int left = num_ops, out = 0;
  const int classes = dtype == GBSV_C64 ? 4 : 3;  // bank bits of a slot
  while (left > 0) {
    if (*num_layouts >= max_layouts) return GBSV_ERR_SCRATCH;
    gbsv_adjoint_layout_t& L = layouts[(*num_layouts)++];
    memset(&L, 0, sizeof(L));
    L.first = out;
    // take ops in order; one may pass the ops left behind if it shares no
    // tile bit with them, or only bits on which both are diagonal
    uint32_t regs = 0, behind = 0, behind_diag = 0;
    std::vector<int> taken;
    for (int i = 0; i < num_ops; ++i) {
      if (done[i]) continue;
      const Info& f = info[i];
      const bool free = f.diag ? !(f.touch & behind)
                               : !(f.touch & (behind | behind_diag));
      if (free && __builtin_popcount(regs | f.need) <= rb) {
        regs |= f.need;
        taken.push_back(i);
        done[i] = 1;
        --left;
      } else if (f.diag) {
        behind_diag |= f.touch;
      } else {
        behind |= f.touch;
      }
    }
    // fill up with tile bits of the most numerous bank classes
    while (__builtin_popcount(regs) < rb) {
      int best = -1, most = -1;
      for (int b = m - 1; b >= 0; --b) {
        if ((regs >> b) & 1) continue;
        int cnt = 0;
        for (int q = b % classes; q < m; q += classes)
          cnt += !((regs >> q) & 1);
        if (cnt > most) {
          most = cnt;
          best = b;
        }
      }
      regs |= 1u << best;
    }
    int reg_of[32], k = 0, t = 0;
    for (int b = 0; b < 32; ++b) reg_of[b] = -1;
    for (int b = 0; b < m; ++b)
      if ((regs >> b) & 1) {
        reg_of[b] = k;
        L.rb[k++] = (int8_t)b;
      }
    // thread bits: one of each bank class first, then the rest ascending
    uint32_t used = regs;
    for (int c = 0; c < classes; ++c)
      for (int b = c; b < m; b += classes)
        if (!((used >> b) & 1)) {
          used |= 1u << b;
          L.tb[t++] = (int8_t)b;
          break;
        }
    for (int b = 0; b < m; ++b)
      if (!((used >> b) & 1)) L.tb[t++] = (int8_t)b;
    for (int i : taken) {
      const HostAdjOp& o = in[i];
      gbsv_adjoint_regop_t r;
      memset(&r, 0, sizeof(r));
      r.nq = 1;
      auto place = [&](int j, int b) {
        r.k[j] = b >= 0 ? reg_of[b] : -1;
        r.t[j] = b >= 0 && reg_of[b] < 0 ? 1u << b : 0u;
        r.o[j] = b < 0 ? -1 - b : -1;
      };
      if (o.kind == 0) {
        place(0, o.bit);
        r.slot = o.slot;
        r.type = r.k[0] >= 0 ? 4 * o.gen + r.k[0] : o.bit >= 0 ? 12 : 13;
        regops[out++] = r;
        continue;
      }
      r.mat = o.g.mat;
      r.cmask = o.g.cmask;
      r.cval = o.g.cval;
      if (o.g.kind == 2) {
        r.nq = o.g.nq;
        place(0, o.g.b0);
        if (o.g.nq > 1) place(1, o.g.b1);
        int minus = 0;  // entries -1
        bool sign = pool != nullptr;
        for (int e = 0; sign && e < (1 << r.nq); ++e) {
          const cd v = view.at(r.mat + e);
          if (v == cd(-1.0)) minus |= 1 << e;
          else if (v != cd(1.0)) sign = false;
        }
        if (!sign) {
          r.type = 15;
          regops[out++] = r;
          continue;
        }
        // the sign as a XOR of products of bits: for each set of qubits
        // (bit 1 of `set`: qubit 0 where there are two), the parity of the
        // -1 entries whose index lies within the set
        for (int set = 0; set < (1 << r.nq); ++set) {
          int par = 0;
          for (int e = 0; e < (1 << r.nq); ++e)
            if ((e & ~set) == 0) par ^= (minus >> e) & 1;
          if (!par) continue;
          gbsv_adjoint_regop_t q;
          memset(&q, 0, sizeof(q));
          q.type = 14;
          q.cmask = r.cmask;
          q.cval = r.cval;
          uint32_t regsel = 0xFFFFu;
          static const uint32_t kRegs[4] = {0xAAAAu, 0xCCCCu, 0xF0F0u,
                                            0xFF00u};
          for (int j = 0; j < r.nq; ++j) {
            if (!((set >> (r.nq - 1 - j)) & 1)) continue;
            if (r.k[j] >= 0) {
              regsel &= kRegs[r.k[j]];
            } else if (r.t[j]) {
              q.t[0] |= r.t[j];
            } else {
              q.cmask |= uint64_t(1) << r.o[j];
              q.cval |= uint64_t(1) << r.o[j];
            }
          }
          q.signs = (int32_t)regsel;
          regops[out++] = q;
        }
        continue;
      }
      if (o.g.kind == 0) {
        r.type = 16;
        place(0, o.g.b0);
      } else if (info[i].ctrl) {
        r.type = 16;
        r.nq = 2;
        place(0, o.g.b1);
        place(1, o.g.b0);
      } else {
        r.type = 17;
        r.nq = 2;
        place(0, o.g.b0);
        place(1, o.g.b1);
      }
      regops[out++] = r;
    }
    L.count = out - L.first;
    if (L.count == 0) --*num_layouts;  // its gates came to nothing
  }
  *num_regops = out;
  return GBSV_OK;
}

// ---- tensor-core stages -----------------------------------------------------
namespace {

struct TcGate {
  uint64_t m;   // positions it acts on
  bool diag;
  int id;       // index in the caller's list
};

constexpr int TCP_BITS = 5, TCP_TILE = 12, TCP_BLOCKS = 64;
// Gates of a list that is looked through whole when blocks are compared.
constexpr size_t TCP_WHOLE = 512;

uint64_t tc_dense(const std::vector<TcGate>& g) {
  uint64_t m = 0;
  for (const TcGate& x : g) m |= x.diag ? 0 : x.m;
  return m;
}

// Walks the gates in order and reports what a block on positions B takes:
// gates inside B, and diagonals disjoint from B (which commute with the
// block and cost nothing).  A gate may pass those left behind when it shares
// no position with them, or when both are diagonal there.  f(index, post).
// Ends where the dense gates left behind touch all of `all`.
template <typename F>
void tc_scan(const std::vector<TcGate>& g, uint64_t B, uint64_t all, F f) {
  uint64_t dense = 0, diag = 0;  // positions of the gates left behind
  for (size_t i = 0; i < g.size() && (!all || (dense & all) != all); ++i) {
    const TcGate& x = g[i];
    if (!(x.m & (x.diag ? dense : dense | diag))) {
      if (!(x.m & ~B)) {
        f(i, false);
        continue;
      }
      if (x.diag && !(x.m & B)) {
        f(i, true);
        continue;
      }
    }
    (x.diag ? diag : dense) |= x.m;
  }
}

// Gates a block on B takes in, diagonals a little less (another block may
// take them along), tile positions it would add to the stage last.
double tc_value(const std::vector<TcGate>& g, uint64_t B, uint64_t all,
                uint64_t tile) {
  double v = 0;
  tc_scan(g, B, all, [&](size_t i, bool post) {
    if (!post) v += g[i].diag ? 0.9 : 1.0;
  });
  return v - 0.01 * __builtin_popcountll(B & ~tile);
}

// The best positions found for the next block within `tile` (grown to at
// most 12): from each gate that can run now, grown by whole gates while that
// takes more in, then improved by exchanging single positions.
uint64_t tc_best(const std::vector<TcGate>& g, uint64_t all, uint64_t tile,
                 double* value) {
  auto fits = [&](uint64_t B) {
    return __builtin_popcountll(B) <= TCP_BITS &&
           __builtin_popcountll(tile | B) <= TCP_TILE;
  };
  std::vector<uint64_t> seeds, grow;
  auto add = [](std::vector<uint64_t>& v, uint64_t m, size_t most) {
    if (v.size() < most && std::find(v.begin(), v.end(), m) == v.end())
      v.push_back(m);
  };
  uint64_t dense = 0, diag = 0;
  for (size_t i = 0; i < g.size() && (!all || (dense & all) != all); ++i) {
    if (!(g[i].m & (g[i].diag ? dense : dense | diag))) add(seeds, g[i].m, 24);
    add(grow, g[i].m, 48);
    (g[i].diag ? diag : dense) |= g[i].m;
  }
  uint64_t best = 0;
  *value = 0;
  for (uint64_t B : seeds) {
    if (!fits(B)) continue;
    double v = tc_value(g, B, all, tile);
    while (true) {
      uint64_t next = 0;
      double nv = 0, gain = 0;
      for (uint64_t m : grow) {
        const uint64_t nb = B | m;
        if (nb == B || !fits(nb)) continue;
        const double x = tc_value(g, nb, all, tile);
        const double per = (x - v) / __builtin_popcountll(nb & ~B);
        if (!next || per > gain || (per == gain && x > nv)) {
          next = nb;
          nv = x;
          gain = per;
        }
      }
      if (!next || nv <= v) break;
      B = next;
      v = nv;
    }
    if (v > *value) {
      *value = v;
      best = B;
    }
  }
  if (!best) return 0;
  uint64_t reach = 0;
  for (uint64_t m : grow) reach |= m;
  for (int round = 0; round < 3; ++round) {
    uint64_t next = best;
    double nv = *value;
    for (uint64_t out = best; out; out &= out - 1)
      for (uint64_t in = reach & ~best; in; in &= in - 1) {
        const uint64_t nb = (best & ~(out & -out)) | (in & -in);
        if (!fits(nb)) continue;
        const double x = tc_value(g, nb, all, tile);
        if (x > nv) {
          next = nb;
          nv = x;
        }
      }
    if (next == best) break;
    best = next;
    *value = nv;
  }
  return best;
}

}  // namespace

// A block costs about twice what a stage costs beside its blocks (0.15 and
// 0.08 ms on 26 qubits), so the next block stays in the stage's tile unless
// a new tile would take in half as much again.
extern "C" int gbsv_plan_tc(const uint64_t* masks, const uint8_t* diagonal,
                            int num_gates, int min_contiguous, int32_t* stage,
                            int32_t* block, uint8_t* post) {
  if (num_gates < 0 || min_contiguous < 0 || min_contiguous > TCP_TILE ||
      (num_gates > 0 && (!masks || !diagonal || !stage || !block || !post)))
    return GBSV_ERR_INVALID_ARG;
  const uint64_t low = (uint64_t(1) << min_contiguous) - 1;
  std::vector<TcGate> left;
  uint64_t touched = 0;
  for (int i = 0; i < num_gates; ++i) {
    const int k = __builtin_popcountll(masks[i]);
    if (k > TCP_BITS || __builtin_popcountll(low | masks[i]) > TCP_TILE)
      return GBSV_ERR_UNSUPPORTED;
    left.push_back(TcGate{masks[i], diagonal[i] != 0, i});
    touched |= masks[i];
  }
  uint64_t tile = low;
  int s = 0, b = 0;  // current stage and its number of blocks
  while (!left.empty()) {
    // A qubit without dense gates is never left behind, and a long list
    // would be looked through to its end for every candidate (quadratic:
    // 10,000 gates 6.6 s, of which a quarter of the gates diagonal on one
    // such qubit).  What its diagonals add is not counted there then; the
    // block takes them all the same, below.
    const uint64_t all = left.size() > TCP_WHOLE ? tc_dense(left) : touched;
    double v = 0, fresh = 0;
    uint64_t B = b < TCP_BLOCKS ? tc_best(left, all, tile, &v) : 0;
    if (b > 0) {
      const uint64_t F = tc_best(left, all, low, &fresh);
      if (!B || v < 0.65 * fresh) {
        ++s;
        b = 0;
        tile = low;
        B = F;
      }
    }
    if (!B) B = left[0].m;  // gates on no position, or none found
    std::vector<char> take(left.size(), 0);
    tc_scan(left, B, 0, [&](size_t i, bool p) {
      take[i] = 1;
      const int id = left[i].id;
      stage[id] = s;
      block[id] = b;
      post[id] = p;
    });
    std::vector<TcGate> rest;
    for (size_t i = 0; i < left.size(); ++i)
      if (!take[i]) rest.push_back(left[i]);
    if (rest.size() == left.size()) return GBSV_ERR_UNSUPPORTED;
    left.swap(rest);
    tile |= B;
    ++b;
  }
  return GBSV_OK;
}
