// fmm_b200 host runtime and C ABI (declared in include/fmm_b200.h).
//
// Reference interfaces replaced (fmm-gen):
//   bl_dgemm                       common/dgemm/my_dgemm.c:115-210
//   bl_dgemm_strassen_abc/ab/naive common/include/bl_dgemm.h:96-130 (generated bodies:
//                                  meta/abc_gen_mix.py:448-472, meta/ab_gen_mix.py:430-456,
//                                  meta/naive_gen_mix.py:412-429)
//   fringe split + peeling         meta/common_mix.py:124-171, common/dgemm/bl_dgemm_util.c:316-353
//   packing pool                   common/dgemm/bl_dgemm_util.c:375-394 (here: stream-ordered
//                                  device allocations, freed after each call)
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <iterator>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "../../include/fmm_b200.h"
#include "fmm_kernels.cuh"
#include "fmm_split_bf16.cuh"
#include "fmm_tile.cuh"

namespace {

constexpr int kMaxDevices = 64;
constexpr int kMR = 8;  // register-tile granularity of the FMM/fringe split (bl_config.h:16-17)
constexpr int kNR = 4;

std::atomic<long long> g_launches{0};
thread_local int t_last_error = FMM_OK;
// Byte written into every ticket before a launch (fmm_debug_set): 0 in normal operation.
int g_ticket_fill = 0;
// Cap on the pre-summed operand workspace of one call (fmm_set_workspace_limit), and the
// workspace bytes the last call on this thread used.
constexpr long long kDefaultWorkspaceLimit = 8LL << 30;
std::atomic<long long> g_ws_limit{kDefaultWorkspaceLimit};
thread_local long long t_last_ws = 0;

// Optional per-kernel timing: when enabled, every launch is bracketed by CUDA events on
// its own stream; fmm_profile_end() sums the durations per kernel kind.
enum KernelKind {
  K_PRODUCTS = 0,
  K_TILE_GEMM = 1,
  K_PRESUM = 2,
  K_SCATTER = 3,
  K_SPLIT_OPERANDS = 4,
  K_GEMM_SPLIT = 5,
  K_PRODUCTS_BATCH = 6,
  K_PRESUM_BATCH = 7,
  K_PITCH_COPY = 8,
  K_COMBINE = 9,
  K_NUM = 10
};
const char* const kKernelNames[K_NUM] = {"fmm_products_kernel",       "fmm_tile_gemm_kernel",    "fmm_presum_kernel",
                                         "fmm_scatter_kernel",        "fmm_split_operands_kernel", "fmm_split_gemm_kernel",
                                         "fmm_products_batch_kernel", "fmm_presum_batch_kernel", "fmm_pitch_copy_kernel",
                                         "fmm_combine_kernel"};
struct ProfRec {
  int kind;
  cudaEvent_t e0, e1;
};
std::mutex g_prof_mu;
bool g_prof_on = false;
std::vector<ProfRec> g_prof;

struct ProfScope {
  int kind;
  cudaStream_t st;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  ProfScope(int k, cudaStream_t s) : kind(k), st(s) {
    std::lock_guard<std::mutex> lk(g_prof_mu);
    if (!g_prof_on) return;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
      e0 = e1 = nullptr;
      return;
    }
    cudaEventRecord(e0, st);
  }
  ~ProfScope() {
    if (!e0) return;
    cudaEventRecord(e1, st);
    std::lock_guard<std::mutex> lk(g_prof_mu);
    g_prof.push_back(ProfRec{kind, e0, e1});
  }
};

struct DevTables {
  fmm::Prod* prods = nullptr;
  fmm::Term* terms = nullptr;
  int* cblk = nullptr;
  int* ent_r = nullptr;
  double* ent_w = nullptr;
  int* cg_desc = nullptr;  // grouped combine tables
  int* cg_r = nullptr;
  int* cg_m = nullptr;
  double* cg_c = nullptr;
  int* ch_r = nullptr;
  unsigned long long* ch_n = nullptr;
  fmm::CombineOp* ch_op = nullptr;
  fmm::Prod* prods_ps = nullptr;  // products over pre-summed operands (one A and one B term each)
  fmm::Term* terms_ps = nullptr;
  int* plistA = nullptr;          // products whose A operand is pre-summed, in slot order
  int* plistB = nullptr;
  fmm::Prod* prods_all = nullptr;  // every product over pre-summed slots (slot r = product r)
  fmm::Term* terms_all = nullptr;
  int* plist_all = nullptr;        // 0 .. R-1
  int* ps_first[2] = {nullptr, nullptr};         // presum tables of the A and B side
  fmm::PTerm* ps_terms[2] = {nullptr, nullptr};
  bool ready = false;
};

// Tables derived from a plan on first use: the classical plan's k split into S parts
// (ksplit_build) or the products [S, g1) of a workspace group (group_build).
enum TableBase : int { BASE_SPLIT = 0, BASE_GROUP = 1 };
struct KSplitTables {
  int base = 0, S = 0, g1 = 0, dev = -1;
  fmm::Prod* prods = nullptr;
  fmm::Term* terms = nullptr;
};

}  // namespace

struct fmm_plan {
  int dims[3];
  int rank;
  std::vector<fmm::Prod> prods;
  std::vector<fmm::Term> terms;
  // Per C block lists of (product, coefficient), products in order: used by the scatter.
  std::vector<int> cblk;     // 4 ints per block
  std::vector<int> ent_r;
  std::vector<double> ent_w;
  int n_cblk = 0;
  int n_cterms = 0;  // C terms over all products
  // The same lists with the blocks in groups that share products (fmm_combine_kernel's
  // tables: group descriptors, merged entries and their coefficients; see build_combine_groups).
  std::vector<int> cg_desc, cg_r, cg_m;
  std::vector<double> cg_c;
  int n_cgroup = 0;
  std::vector<int> ch_r;                 // staged kernel: CST_CHUNK products per chunk
  std::vector<unsigned long long> ch_n;  // one byte per member: its operations in the chunk
  std::vector<fmm::CombineOp> ch_op;     // the operations in the order they run
  // Pre-summed form: each product's A operand is either its single A block (src 0) or
  // slot j of the workspace S (src 1) that holds sum_i U[i,r] A_i; likewise for B / T.
  std::vector<fmm::Prod> prods_ps;
  std::vector<fmm::Term> terms_ps;
  std::vector<int> plistA, plistB;
  // Every product pre-summed (slot r = product r): used when ks is not a multiple of the
  // k step, so that zero-padded workspaces keep each k step inside its operand block.
  std::vector<fmm::Prod> prods_all;
  std::vector<fmm::Term> terms_all;
  // A (0) and B (1) terms of every product, product r's from ps_first[r] on.
  std::vector<int> ps_first[2];
  std::vector<fmm::PTerm> ps_terms[2];
  std::mutex mu;
  DevTables dev[kMaxDevices];
  std::vector<KSplitTables> ksplit;  // uploaded k-split tables (any device), built on first use
};

namespace {

fmm_plan* g_default_plan = nullptr;
std::mutex g_default_mu;

int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return FMM_OK;
  if (e == cudaErrorMemoryAllocation) return FMM_E_NOMEM;
  return FMM_E_CUDA;
}

#define FMM_CUDA_TRY(expr)                  \
  do {                                      \
    cudaError_t _e = (expr);                \
    if (_e != cudaSuccess) return cuda_status(_e); \
  } while (0)

int upload_tables(fmm_plan* p, DevTables& d) {
  std::lock_guard<std::mutex> lk(p->mu);
  if (d.ready) return FMM_OK;
  FMM_CUDA_TRY(cudaMalloc(&d.prods, sizeof(fmm::Prod) * p->prods.size()));
  FMM_CUDA_TRY(cudaMalloc(&d.terms, sizeof(fmm::Term) * p->terms.size()));
  FMM_CUDA_TRY(cudaMalloc(&d.cblk, sizeof(int) * (p->cblk.size() ? p->cblk.size() : 1)));
  FMM_CUDA_TRY(cudaMalloc(&d.ent_r, sizeof(int) * (p->ent_r.size() ? p->ent_r.size() : 1)));
  FMM_CUDA_TRY(cudaMalloc(&d.ent_w, sizeof(double) * (p->ent_w.size() ? p->ent_w.size() : 1)));
  FMM_CUDA_TRY(cudaMemcpy(d.prods, p->prods.data(), sizeof(fmm::Prod) * p->prods.size(), cudaMemcpyHostToDevice));
  FMM_CUDA_TRY(cudaMemcpy(d.terms, p->terms.data(), sizeof(fmm::Term) * p->terms.size(), cudaMemcpyHostToDevice));
  if (!p->cblk.empty())
    FMM_CUDA_TRY(cudaMemcpy(d.cblk, p->cblk.data(), sizeof(int) * p->cblk.size(), cudaMemcpyHostToDevice));
  if (!p->ent_r.empty()) {
    FMM_CUDA_TRY(cudaMemcpy(d.ent_r, p->ent_r.data(), sizeof(int) * p->ent_r.size(), cudaMemcpyHostToDevice));
    FMM_CUDA_TRY(cudaMemcpy(d.ent_w, p->ent_w.data(), sizeof(double) * p->ent_w.size(), cudaMemcpyHostToDevice));
  }
  {
    auto up = [](auto** dst, const auto& v) -> cudaError_t {
      using T = typename std::decay_t<decltype(v)>::value_type;
      cudaError_t e = cudaMalloc(dst, sizeof(T) * (v.size() ? v.size() : 1));
      if (e == cudaSuccess && !v.empty()) e = cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
      return e;
    };
    FMM_CUDA_TRY(up(&d.cg_desc, p->cg_desc));
    FMM_CUDA_TRY(up(&d.cg_r, p->cg_r));
    FMM_CUDA_TRY(up(&d.cg_m, p->cg_m));
    FMM_CUDA_TRY(up(&d.cg_c, p->cg_c));
    FMM_CUDA_TRY(up(&d.ch_r, p->ch_r));
    FMM_CUDA_TRY(up(&d.ch_n, p->ch_n));
    FMM_CUDA_TRY(up(&d.ch_op, p->ch_op));
    for (int side = 0; side < 2; ++side) {
      FMM_CUDA_TRY(up(&d.ps_first[side], p->ps_first[side]));
      FMM_CUDA_TRY(up(&d.ps_terms[side], p->ps_terms[side]));
    }
  }
  FMM_CUDA_TRY(cudaMalloc(&d.prods_ps, sizeof(fmm::Prod) * p->prods_ps.size()));
  FMM_CUDA_TRY(cudaMalloc(&d.terms_ps, sizeof(fmm::Term) * p->terms_ps.size()));
  FMM_CUDA_TRY(cudaMalloc(&d.plistA, sizeof(int) * (p->plistA.size() + 1)));
  FMM_CUDA_TRY(cudaMalloc(&d.plistB, sizeof(int) * (p->plistB.size() + 1)));
  FMM_CUDA_TRY(cudaMemcpy(d.prods_ps, p->prods_ps.data(), sizeof(fmm::Prod) * p->prods_ps.size(),
                          cudaMemcpyHostToDevice));
  FMM_CUDA_TRY(cudaMemcpy(d.terms_ps, p->terms_ps.data(), sizeof(fmm::Term) * p->terms_ps.size(),
                          cudaMemcpyHostToDevice));
  if (!p->plistA.empty())
    FMM_CUDA_TRY(cudaMemcpy(d.plistA, p->plistA.data(), sizeof(int) * p->plistA.size(), cudaMemcpyHostToDevice));
  if (!p->plistB.empty())
    FMM_CUDA_TRY(cudaMemcpy(d.plistB, p->plistB.data(), sizeof(int) * p->plistB.size(), cudaMemcpyHostToDevice));
  std::vector<int> all(p->rank);
  for (int r = 0; r < p->rank; ++r) all[r] = r;
  FMM_CUDA_TRY(cudaMalloc(&d.prods_all, sizeof(fmm::Prod) * p->prods_all.size()));
  FMM_CUDA_TRY(cudaMalloc(&d.terms_all, sizeof(fmm::Term) * p->terms_all.size()));
  FMM_CUDA_TRY(cudaMalloc(&d.plist_all, sizeof(int) * all.size()));
  FMM_CUDA_TRY(cudaMemcpy(d.prods_all, p->prods_all.data(), sizeof(fmm::Prod) * p->prods_all.size(),
                          cudaMemcpyHostToDevice));
  FMM_CUDA_TRY(cudaMemcpy(d.terms_all, p->terms_all.data(), sizeof(fmm::Term) * p->terms_all.size(),
                          cudaMemcpyHostToDevice));
  FMM_CUDA_TRY(cudaMemcpy(d.plist_all, all.data(), sizeof(int) * all.size(), cudaMemcpyHostToDevice));
  d.ready = true;
  return FMM_OK;
}

int device_tables(const fmm_plan* cp, DevTables** out) {
  fmm_plan* p = const_cast<fmm_plan*>(cp);
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return FMM_E_UNSUPPORTED;
  DevTables& d = p->dev[dev];
  if (!d.ready) {
    int rc = upload_tables(p, d);
    if (rc != FMM_OK) return rc;
  }
  *out = &d;
  return FMM_OK;
}

// k split of the classical plan: S products over k parts of depth d, part q at block
// coordinate q (the products kernel addresses operand blocks by multiples of the product's k
// depth, so part q starts at q d), all added to the one C block in order.
void ksplit_build(int S, std::vector<fmm::Prod>* op, std::vector<fmm::Term>* ot) {
  for (int q = 0; q < S; ++q) {
    const int t = (int)ot->size();
    ot->push_back(fmm::Term{0, q, 1.0, 0, 0});
    ot->push_back(fmm::Term{q, 0, 1.0, 0, 0});
    ot->push_back(fmm::Term{0, 0, 1.0, 0, q});
    op->push_back(fmm::Prod{t, 1, t + 1, 1, t + 2, 1});
  }
}

// Tables of products [g0, g1) over the slots of a group workspace: product r reads slot
// r - g0 of S and of T (src 1), keeps its C terms, and counts its per-block ticket positions
// within the group (each group is a launch of its own).
void group_build(const fmm_plan* p, int g0, int g1, std::vector<fmm::Prod>* op, std::vector<fmm::Term>* ot) {
  std::vector<int> cnt((size_t)p->dims[0] * p->dims[2], 0);
  for (int r = g0; r < g1; ++r) {
    const fmm::Prod& pr = p->prods[r];
    fmm::Prod v{};
    v.a0 = (int)ot->size();
    v.na = 1;
    ot->push_back(fmm::Term{0, r - g0, 1.0, 1, 0});
    v.b0 = (int)ot->size();
    v.nb = 1;
    ot->push_back(fmm::Term{0, r - g0, 1.0, 1, 0});
    v.c0 = (int)ot->size();
    v.nc = pr.nc;
    for (int t = 0; t < pr.nc; ++t) {
      fmm::Term x = p->terms[pr.c0 + t];
      x.pad = cnt[(size_t)x.row * p->dims[2] + x.col]++;
      ot->push_back(x);
    }
    op->push_back(v);
  }
}

// Derived tables of a plan on the current device (uploaded on first use): the classical plan's
// k split into S parts, or with base == BASE_GROUP the group [S, g1) (group_build).
int ksplit_tables(const fmm_plan* cp, int base, int S, const fmm::Prod** prods, const fmm::Term** terms,
                  int g1 = 0) {
  fmm_plan* p = const_cast<fmm_plan*>(cp);
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(p->mu);
  for (const auto& t : p->ksplit)
    if (t.base == base && t.S == S && t.g1 == g1 && t.dev == dev) {
      *prods = t.prods;
      *terms = t.terms;
      return FMM_OK;
    }
  std::vector<fmm::Prod> vp;
  std::vector<fmm::Term> vt;
  if (base == BASE_GROUP)
    group_build(p, S, g1, &vp, &vt);
  else
    ksplit_build(S, &vp, &vt);
  KSplitTables t;
  t.base = base;
  t.S = S;
  t.g1 = g1;
  t.dev = dev;
  FMM_CUDA_TRY(cudaMalloc(&t.prods, sizeof(fmm::Prod) * vp.size()));
  cudaError_t e = cudaMalloc(&t.terms, sizeof(fmm::Term) * vt.size());
  if (e == cudaSuccess) e = cudaMemcpy(t.prods, vp.data(), sizeof(fmm::Prod) * vp.size(), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(t.terms, vt.data(), sizeof(fmm::Term) * vt.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(t.prods);
    if (t.terms) cudaFree(t.terms);
    return cuda_status(e);
  }
  p->ksplit.push_back(t);
  *prods = t.prods;
  *terms = t.terms;
  return FMM_OK;
}

// Blocks of the C grid in groups of up to fmm::COMBINE_GROUP that share products, for
// fmm_combine_kernel: greedily merge the two groups whose product sets overlap most (while
// the merged group fits), up to 64 blocks; beyond that, consecutive blocks.  Then one merged
// entry per product of a group's union (increasing r) with the mask of the members it
// updates and their coefficients in member order.
void build_combine_groups(fmm_plan* p) {
  const int nb = p->n_cblk;
  std::vector<std::vector<int>> mem(nb), uni(nb);
  for (int b = 0; b < nb; ++b) {
    mem[b] = {b};
    const int e0 = p->cblk[4 * b + 2], ne = p->cblk[4 * b + 3];
    uni[b].assign(p->ent_r.begin() + e0, p->ent_r.begin() + e0 + ne);  // increasing r
  }
  auto overlap = [](const std::vector<int>& x, const std::vector<int>& y) {
    size_t i = 0, j = 0;
    int n = 0;
    while (i < x.size() && j < y.size()) {
      if (x[i] == y[j]) ++n, ++i, ++j;
      else if (x[i] < y[j]) ++i;
      else ++j;
    }
    return n;
  };
  if (nb <= 64) {
    for (;;) {
      int best = 0, bi = -1, bj = -1;
      for (int i = 0; i < (int)mem.size(); ++i)
        for (int j = i + 1; j < (int)mem.size(); ++j) {
          if ((int)(mem[i].size() + mem[j].size()) > fmm::COMBINE_GROUP) continue;
          const int ov = overlap(uni[i], uni[j]);
          if (ov > best) best = ov, bi = i, bj = j;
        }
      if (bi < 0) break;
      mem[bi].insert(mem[bi].end(), mem[bj].begin(), mem[bj].end());
      std::vector<int> u;
      std::set_union(uni[bi].begin(), uni[bi].end(), uni[bj].begin(), uni[bj].end(), std::back_inserter(u));
      uni[bi] = u;
      mem.erase(mem.begin() + bj);
      uni.erase(uni.begin() + bj);
    }
  } else {
    std::vector<std::vector<int>> m2, u2;
    for (int b = 0; b < nb; b += fmm::COMBINE_GROUP) {
      std::vector<int> g, u;
      for (int q = b; q < std::min(nb, b + fmm::COMBINE_GROUP); ++q) {
        g.push_back(q);
        std::vector<int> t;
        std::set_union(u.begin(), u.end(), uni[q].begin(), uni[q].end(), std::back_inserter(t));
        u = t;
      }
      m2.push_back(g);
      u2.push_back(u);
    }
    mem = m2;
    uni = u2;
  }
  p->cg_desc.clear();
  p->ch_r.clear();
  p->ch_n.clear();
  p->ch_op.clear();
  p->cg_r.clear();
  p->cg_m.clear();
  p->cg_c.clear();
  for (size_t g = 0; g < mem.size(); ++g) {
    const int first = (int)p->cg_r.size();
    std::vector<size_t> pos(mem[g].size(), 0);  // cursor into each member's (increasing r) list
    for (int r : uni[g]) {
      int mask = 0;
      const int k0 = (int)p->cg_c.size();
      for (size_t q = 0; q < mem[g].size(); ++q) {
        const int b = mem[g][q];
        const int e0 = p->cblk[4 * b + 2], ne = p->cblk[4 * b + 3];
        if (pos[q] < (size_t)ne && p->ent_r[e0 + pos[q]] == r) {
          mask |= 1 << q;
          p->cg_c.push_back(p->ent_w[e0 + pos[q]]);
          ++pos[q];
        }
      }
      p->cg_r.push_back(r);
      p->cg_m.push_back(mask | (k0 << 8));
    }
    // the group's entries in chunks of CST_CHUNK (the staged kernel's stage): per chunk the
    // products, and per member the operations on it, slots in increasing product order
    const int first_chunk = (int)(p->ch_r.size() / fmm::CST_CHUNK), first_op = (int)p->ch_op.size();
    {
      const int ne = (int)p->cg_r.size() - first;
      for (int q0 = 0; q0 < ne; q0 += fmm::CST_CHUNK) {
        std::vector<fmm::CombineOp> ops[fmm::COMBINE_GROUP];
        for (int t = 0; t < fmm::CST_CHUNK; ++t) {
          const int e = first + std::min(q0 + t, ne - 1);
          p->ch_r.push_back(p->cg_r[e]);
          if (q0 + t >= ne) continue;
          const int mk = p->cg_m[e];
          int kc = mk >> 8;
          for (int q = 0; q < fmm::COMBINE_GROUP; ++q)
            if (mk & (1 << q))
              ops[q].push_back(fmm::CombineOp{p->cg_c[kc++], (int)(t * fmm::CST_TILE * sizeof(double)), 0});
        }
        unsigned long long n = 0;
        for (int q = 0; q < fmm::COMBINE_GROUP; ++q) {
          n |= (unsigned long long)ops[q].size() << (8 * q);
          p->ch_op.insert(p->ch_op.end(), ops[q].begin(), ops[q].end());
        }
        p->ch_n.push_back(n);
      }
    }
    p->cg_desc.push_back(first);
    p->cg_desc.push_back((int)p->cg_r.size() - first);
    p->cg_desc.push_back((int)mem[g].size());
    p->cg_desc.push_back(first_chunk);
    p->cg_desc.push_back(first_op);
    for (int q = 0; q < fmm::COMBINE_GROUP; ++q) {
      const int b = q < (int)mem[g].size() ? mem[g][q] : mem[g][0];
      p->cg_desc.push_back(p->cblk[4 * b] * p->dims[2] + p->cblk[4 * b + 1]);
    }
  }
  p->n_cgroup = (int)mem.size();
  // the kernels index their tables with these values: check them here (a plan whose tables
  // fail falls back to the per-block scatter)
  size_t nop = 0;
  for (unsigned long long n : p->ch_n)
    for (int q = 0; q < fmm::COMBINE_GROUP; ++q) nop += (n >> (8 * q)) & 0xff;
  bool ok = p->ch_r.size() == (size_t)fmm::CST_CHUNK * p->ch_n.size() && nop == p->ch_op.size();
  for (const auto& o : p->ch_op) ok = ok && o.off >= 0 && o.off < (int)(fmm::CST_STAGE_DOUBLES * sizeof(double));
  for (int r : p->ch_r) ok = ok && r >= 0 && r < p->rank;
  for (int r : p->cg_r) ok = ok && r >= 0 && r < p->rank;
  for (int g = 0; ok && g < p->n_cgroup; ++g) {
    const int* gd = p->cg_desc.data() + (size_t)g * fmm::GDESC;
    const int nch = (gd[1] + fmm::CST_CHUNK - 1) / fmm::CST_CHUNK;
    ok = gd[1] > 0 && gd[0] + gd[1] <= (int)p->cg_r.size() && gd[2] >= 1 && gd[2] <= fmm::COMBINE_GROUP &&
         gd[3] >= 0 && gd[3] + nch <= (int)p->ch_n.size() && gd[4] >= 0 && gd[4] <= (int)p->ch_op.size();
    for (int q = 0; ok && q < fmm::COMBINE_GROUP; ++q) ok = gd[fmm::GD_MEMBERS + q] >= 0 && gd[fmm::GD_MEMBERS + q] < p->dims[0] * p->dims[2];
  }
  if (!ok) p->n_cgroup = 0;
}

int build_plan(const int dims[3], int rank, const int* nterms, const int* rows, const int* cols,
               const double* coefs, fmm_plan** out) {
  if (!dims || !nterms || !rows || !cols || !coefs || !out || rank <= 0) return FMM_E_INVALID;
  if (dims[0] <= 0 || dims[1] <= 0 || dims[2] <= 0) return FMM_E_PLAN;
  fmm_plan* p = new (std::nothrow) fmm_plan();
  if (!p) return FMM_E_NOMEM;
  std::memcpy(p->dims, dims, sizeof(p->dims));
  p->rank = rank;
  int pos = 0;
  const int lim[3][2] = {{dims[0], dims[1]}, {dims[1], dims[2]}, {dims[0], dims[2]}};
  for (int r = 0; r < rank; ++r) {
    fmm::Prod pr{};
    int* first[3] = {&pr.a0, &pr.b0, &pr.c0};
    int* count[3] = {&pr.na, &pr.nb, &pr.nc};
    for (int s = 0; s < 3; ++s) {
      const int n = nterms[3 * r + s];
      if (n <= 0) {
        delete p;
        return FMM_E_PLAN;
      }
      *first[s] = (int)p->terms.size();
      *count[s] = n;
      for (int q = 0; q < n; ++q, ++pos) {
        if (rows[pos] < 0 || rows[pos] >= lim[s][0] || cols[pos] < 0 || cols[pos] >= lim[s][1]) {
          delete p;
          return FMM_E_PLAN;
        }
        p->terms.push_back(fmm::Term{rows[pos], cols[pos], coefs[pos], 0, 0});
      }
    }
    // A single operand term whose coefficient is a power of two moves its coefficient
    // into the product's W coefficients (exact), so the operand can be staged as is.
    for (int side = 0; side < 2; ++side) {
      const int n = side == 0 ? pr.na : pr.nb;
      fmm::Term& t = p->terms[side == 0 ? pr.a0 : pr.b0];
      int e2 = 0;
      if (n == 1 && t.coef != 1.0 && t.coef != 0.0 && std::frexp(std::fabs(t.coef), &e2) == 0.5) {
        for (int q = 0; q < pr.nc; ++q) p->terms[pr.c0 + q].coef *= t.coef;
        t.coef = 1.0;
      }
    }
    p->prods.push_back(pr);
  }
  for (const auto& pr : p->prods) p->n_cterms += pr.nc;
  // C block lists for the scatter (products in increasing order per block).
  const int nblk = dims[0] * dims[2];
  std::vector<std::vector<std::pair<int, double>>> lists(nblk);
  for (int r = 0; r < rank; ++r) {
    const fmm::Prod& pr = p->prods[r];
    for (int q = 0; q < pr.nc; ++q) {
      fmm::Term& t = p->terms[pr.c0 + q];
      auto& list = lists[t.row * dims[2] + t.col];
      t.pad = (int)list.size();  // position among the block's products (per-block tickets)
      list.push_back({r, t.coef});
    }
  }
  for (int b = 0; b < nblk; ++b) {
    if (lists[b].empty()) continue;
    p->cblk.push_back(b / dims[2]);
    p->cblk.push_back(b % dims[2]);
    p->cblk.push_back((int)p->ent_r.size());
    p->cblk.push_back((int)lists[b].size());
    for (auto& e : lists[b]) {
      p->ent_r.push_back(e.first);
      p->ent_w.push_back(e.second);
    }
    ++p->n_cblk;
  }
  build_combine_groups(p);
  for (int r = 0; r < rank; ++r) {
    const fmm::Prod& pr = p->prods[r];
    fmm::Prod q{};
    q.a0 = (int)p->terms_ps.size();
    q.na = 1;
    const fmm::Term& ta = p->terms[pr.a0];
    if (pr.na == 1 && ta.coef == 1.0) {
      p->terms_ps.push_back(ta);
    } else {
      p->terms_ps.push_back(fmm::Term{0, (int)p->plistA.size(), 1.0, 1, 0});
      p->plistA.push_back(r);
    }
    q.b0 = (int)p->terms_ps.size();
    q.nb = 1;
    const fmm::Term& tb = p->terms[pr.b0];
    if (pr.nb == 1 && tb.coef == 1.0) {
      p->terms_ps.push_back(tb);
    } else {
      p->terms_ps.push_back(fmm::Term{0, (int)p->plistB.size(), 1.0, 1, 0});
      p->plistB.push_back(r);
    }
    q.c0 = (int)p->terms_ps.size();
    q.nc = pr.nc;
    for (int c = 0; c < pr.nc; ++c) p->terms_ps.push_back(p->terms[pr.c0 + c]);
    p->prods_ps.push_back(q);
    fmm::Prod qa{};
    qa.a0 = (int)p->terms_all.size();
    qa.na = 1;
    p->terms_all.push_back(fmm::Term{0, r, 1.0, 1, 0});
    qa.b0 = (int)p->terms_all.size();
    qa.nb = 1;
    p->terms_all.push_back(fmm::Term{0, r, 1.0, 1, 0});
    qa.c0 = (int)p->terms_all.size();
    qa.nc = pr.nc;
    for (int c = 0; c < pr.nc; ++c) p->terms_all.push_back(p->terms[pr.c0 + c]);
    p->prods_all.push_back(qa);
    for (int side = 0; side < 2; ++side) {
      const int t0 = side == 0 ? pr.a0 : pr.b0, nt = side == 0 ? pr.na : pr.nb;
      p->ps_first[side].push_back((int)p->ps_terms[side].size());
      for (int t = 0; t < nt; ++t) {
        const fmm::Term& tm = p->terms[t0 + t];
        p->ps_terms[side].push_back(fmm::PTerm{tm.row, tm.col, tm.coef});
      }
    }
  }
  for (int side = 0; side < 2; ++side) p->ps_first[side].push_back((int)p->ps_terms[side].size());
  *out = p;
  return FMM_OK;
}

fmm_plan* classical_plan() {
  static fmm_plan* p = [] {
    const int dims[3] = {1, 1, 1};
    const int nt[3] = {1, 1, 1};
    const int rows[3] = {0, 0, 0}, cols[3] = {0, 0, 0};
    const double coefs[3] = {1.0, 1.0, 1.0};
    fmm_plan* q = nullptr;
    build_plan(dims, 1, nt, rows, cols, coefs, &q);
    return q;
  }();
  return p;
}

bool smem_configured[kMaxDevices];
int sm_count[kMaxDevices];
unsigned* dev_status[kMaxDevices];
std::mutex g_attr_mu;

PFN_cuTensorMapEncodeTiled_v12000 g_encode_tiled = nullptr;

// Dynamic shared memory of a launch of `ctas` CTAs that need `smem` each, so that no SM takes more
// than its share of them (at least two: calls on other streams find room).  A dependent launch's
// CTAs start as the previous kernel's leave, and an SM that empties early would otherwise be
// filled up: 148 CTAs of the products kernel ran three each on 50 SMs.  Measured on B200 without /
// with, whole calls: 222-1 240^3 17.9 / 14.4 us, 400^3 26.3 / 22.3, 512^3 32.6 / 29.1, 2000 x 100 x
// 2000 94 / 83, plain 100 x 3000 x 100 7.8 / 6.5; on four streams 240^3 6.1 / 5.5 us a call, 400^3
// 12.3 / 13.4.  Clusters are spread as it is (plain 256^3, four parts: 5.6 / 5.8).  Starting the
// dependents at the end of the operand sums instead did as much for the products but took 0.3 to 1.3 us
// more per call at other sizes.
constexpr size_t kSmSmem = 228 * 1024, kCtaReserve = 1024;  // shared memory of an SM; the system's part of a CTA
constexpr size_t kPsStagedSmem = kSmSmem / 2 - kCtaReserve;  // fmm_presum_staged_kernel: two CTAs per SM
constexpr size_t kSpreadSmem = kSmSmem / 3;                 // the most that spread_smem asks for
size_t spread_smem(size_t smem, long long ctas, int nsm) {
  const long long per = std::max<long long>(2, (ctas + nsm - 1) / nsm);
  if (per > 4) return smem;  // more than any of these kernels runs on an SM, or its own limit
  return std::max<size_t>(smem, kSmSmem / (size_t)(per + 1) / 256 * 256 - kCtaReserve + 256);  // per + 1 do not fit
}

int configure_kernel(int* dev_out) {
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return FMM_E_UNSUPPORTED;
  std::lock_guard<std::mutex> lk(g_attr_mu);
  if (!smem_configured[dev]) {
    auto smem = [](auto kernel, size_t bytes) {
      return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::max(bytes, kSpreadSmem));
    };
    for (auto kernel : {fmmt::fmm_tile_gemm_kernel<64, 64, false>, fmmt::fmm_tile_gemm_kernel<64, 64, true>,
                        fmmt::fmm_tile_gemm_kernel<64, 64, false, true>})
      FMM_CUDA_TRY(smem(kernel, fmmt::TileShape<64, 64>::SMEM));
    for (auto kernel : {fmmt::fmm_tile_gemm_kernel<32, 32, false>, fmmt::fmm_tile_gemm_kernel<32, 32, true>,
                        fmmt::fmm_tile_gemm_kernel<32, 32, false, true>})
      FMM_CUDA_TRY(smem(kernel, fmmt::TileShape<32, 32>::SMEM));
    FMM_CUDA_TRY(smem(fmm::fmm_presum_staged_kernel, kPsStagedSmem));
    for (auto kernel : {fmmt::fmm_products_kernel<64, false, false>, fmmt::fmm_products_kernel<64, false, true>,
                        fmmt::fmm_products_kernel<64, true, false>, fmmt::fmm_products_kernel<64, true, true>})
      FMM_CUDA_TRY(smem(kernel, fmmt::ProdShape<64>::SMEM));
    for (auto kernel : {fmmt::fmm_products_kernel<32, false, false>, fmmt::fmm_products_kernel<32, false, true>})
      FMM_CUDA_TRY(smem(kernel, fmmt::ProdShape<32>::SMEM));
    for (auto kernel : {fmmt::fmm_products_batch_kernel<false, false>, fmmt::fmm_products_batch_kernel<false, true>,
                        fmmt::fmm_products_batch_kernel<true, false>, fmmt::fmm_products_batch_kernel<true, true>})
      FMM_CUDA_TRY(smem(kernel, fmmt::ProdShape<64>::SMEM));
    if (!g_encode_tiled) {
      cudaDriverEntryPointQueryResult q;
      void* fn = nullptr;
      if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
        g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    FMM_CUDA_TRY(cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev));
    // Workspaces come from the device's stream-ordered pool; keep freed blocks mapped
    // instead of returning them to the driver at every synchronisation, so repeated
    // calls do not pay for mapping gigabytes of workspace again.
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
      cuuint64_t keep = ~0ULL;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    FMM_CUDA_TRY(cudaMalloc(&dev_status[dev], sizeof(unsigned)));
    FMM_CUDA_TRY(cudaMemset(dev_status[dev], 0, sizeof(unsigned)));
    smem_configured[dev] = true;
  }
  *dev_out = dev;
  return FMM_OK;
}

// Column-major FP64 matrix (rows x cols, leading dimension ld) as a 2-D tensor map with
// the given box.  Returns false when TMA cannot address it (then cp.async staging runs).
bool make_tensor_map(CUtensorMap* map, const double* base, long long rows, long long cols, long long ld,
                     unsigned box_rows, unsigned box_cols, bool swizzle = false) {
  if (!g_encode_tiled) return false;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld & 1) != 0) return false;
  if (rows <= 0 || cols <= 0 || rows >= (1LL << 31) || cols >= (1LL << 31) || ld * 8 >= (1LL << 40)) return false;
  cuuint64_t dims[2] = {(cuuint64_t)rows, (cuuint64_t)cols};
  cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(double)};
  cuuint32_t box[2] = {box_rows, box_cols};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double*>(base), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// The maps the tile kernels read their operands with (see fmm_tile.cuh's stage layout).
bool make_a_map(CUtensorMap* map, const double* A, long long m, long long k, long long lda) {
  return make_tensor_map(map, A, m, k, lda, 16, fmmt::BK, true);
}
bool make_b_map(CUtensorMap* map, const double* B, long long k, long long n, long long ldb, int tile) {
  return make_tensor_map(map, B, k, n, ldb, 8, tile);
}

// Launch with programmatic stream serialization (the kernel waits for its predecessors itself,
// griddepcontrol.wait, so its set-up overlaps their end) and an optional cluster.
template <class... Params, class... Args>
int launch_dependent(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t st, int cluster,
                     Args... args) {
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 1;
  if (cluster > 1) {
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cuda_status(e);
}

std::atomic<int> g_split_form{0};    // fmm_debug_set FMM_DEBUG_SPLIT_OPERANDS: 1 = one product per CTA
std::atomic<int> g_force_ksplit{0};  // fmm_debug_set FMM_DEBUG_KSPLIT: S for every classical launch (0: the rule)

long long tiles_of(int m, int n, int t) { return (long long)((m + t - 1) / t) * ((n + t - 1) / t); }

constexpr int kResident64 = fmmt::TileShape<64, 64>::CTAS;  // 64 x 64 CTAs per SM

// Tile side of a plain update with u64 units of 64 x 64 or u32 of 32 x 32: the modelled time,
// SM-seconds over the SMs plus half a unit for the last, partly filled round, the small tile at
// 6 % lower rate (more shared-memory reads per DMMA, twice the operand bytes).  Measured us with
// 64 / 32: 1024^3 77.1 / 75.8, 1200^3 139 / 124, 2048^3 503 / 528, 4096^3 3857 / 4022.  Two or three units an SM
// run at the same time and end together: 1088 x 1088 x 1200 90.6 / 99.4, 1344 x 1280 x 3936 431 / 454 (one alone does
// not reach the rate: 768 x 768 x 1200 58.8 / 55.0).
int tile_side(long long u64, long long u32, int nsm) {
  const double n64 = (double)u64 / nsm;
  const double c64 = (n64 > 1 && n64 <= kResident64 ? std::ceil(n64) : n64 + 0.5) * 4096;
  const double c32 = ((double)u32 / nsm + 0.5) * 1024 * 1.06;
  return c64 <= c32 ? 64 : 32;
}

// Units at the end of a launch of 64 x 64 products that are cut into row strips: those past the
// last whole number per SM, when their strips are fewer per SM than the unit they replace (up to
// 0.7 of the SMs; at three to four units per SM always, where an SM's last unit would run alone).
// Below three per SM all run at once, from twelve on the last round is a small share.  Measured us
// without / with: products of 222-1 1024^3 (448 units) 83.7 / 70.1, 1100^3 (567) 107 / 93, 1488 x 1200 x
// 998 (840) 136 / 116, 1900 x 1800 x 2200 (1575) 452 / 415; past the lines 1280^3 (700) 123 / 125,
// 2500^3 (2800) 827 / 836, 2048^3 (1792) 464 / 466.  Strips for one whole unit per SM more took 1488 x
// 1200 x 998 to 123; plain updates gained at some sizes and lost as much at others.
constexpr int kTailDepth = 128;  // k steps of a product worth cutting
bool cut_tail(double units_per_sm) {
  const double whole = std::floor(units_per_sm);
  return whole >= 3 && whole < 12 && (whole < 4 || units_per_sm - whole <= 0.7);
}

// Tile side for nprod products of m x n: SM-seconds of the 16 x 8 fragments over the SMs, the last,
// partly filled round in quarters where it runs as strips (half a unit for 32 x 32), the small
// tile at 6 % lower rate.  Measured us with 64 / 32: products of 222-1 1024^3 70 / 76, 1100^3 93 / 95,
// 1488 x 1200 x 998 116 / 124, 1900 x 1800 x 2200 415 / 444, 2500^3 827 / 872, of 222-1 x 333-1 1200^3
// 116 / 116, 2016^3 406 / 431 (blocks of 336: partial tiles cost their fragments, not whole tiles).  Launches
// without strips (k below kTailDepth, updates of C) are priced alike: their last round in whole units instead
// chose better at 222-1 1088^2 x 200 (40.5 / 36.8 us a call) and worse at 1600^2 x 200 (59.0 / 63.7), 333-1 1100^2 x 200
// (52.5 / 57.3), 222-2 1000^2 x 192 (55.0 / 58.6).
int product_tile(long long m, long long n, int nprod, int nsm) {
  const double work = (double)((m + 15) / 16 * 16) * (double)((n + 7) / 8 * 8) * nprod / nsm;
  const double u64 = work / 4096, whole = std::floor(u64), f = u64 - whole;
  const double c64 = 4096 * (whole >= 12 ? u64 + 0.5 : whole + (cut_tail(u64) ? std::ceil(4 * f) / 4 : std::ceil(f)));
  const double c32 = 1024 * 1.06 * (work / 1024 + 0.5);
  return c64 <= c32 ? 64 : 32;
}

// k parts of a classical update: S parts of depth d (a multiple of 8), part s covering
// [s d, min(k, (s + 1) d)).  The result of an update depends on S (each part is summed on its
// own and added to C in order), so S is a function of the sizes alone and batches use the
// same one.
// Launches that fill the SMs a few times run deep k in two parts all the same: half as long units, whose last round
// costs half as much (us with 1 / 2 parts: 1408 x 1408 x 3936 524 / 502, 1280 x 1216 x 8000 844 / 788, 2112 x 2112
// x 2048 567 / 560; 1600 x 1600 x 1504 246 / 251, and 1344 x 1344 x 3936 431 / 449, whose 64 x 64 units
// end together).  The lines are those of a 148-SM chip.
constexpr int kMinPartDepth = 64;
constexpr int kPartCtas = 460;
constexpr int kTwoPartDepth = 2048, kTwoPartSms = 148;
void classical_parts(int m, int n, int k, int* S, int* d) {
  auto depth = [&](int s) { return ((k + s - 1) / s + 7) / 8 * 8; };
  const long long t32 = tiles_of(m, n, 32);
  int s = 1;
  while (2 * s <= fmmt::MAX_SPLIT && t32 * 2 * s <= kPartCtas && k >= 2 * s * kMinPartDepth) s *= 2;
  if (s == 1 && k >= kTwoPartDepth) {
    const long long t64 = tiles_of(m, n, 64);
    const bool together = t64 <= kResident64 * kTwoPartSms && tile_side(t64, t32, kTwoPartSms) == 64;
    if (t64 <= 8 * kTwoPartSms && !together) s = 2;
  }
  const int forced = g_force_ksplit.load();
  if (forced > 0 && (long long)(forced - 1) * depth(forced) < k) s = forced;
  *S = s;
  *d = s == 1 ? k : depth(s);
}

// Depth of the parts in which a sum over k is formed (consume_k) for nprod products of m x n x k:
// k / S for the S below, in whole stages.  On random operands one chain over k has a relative error of about
// 0.3 * 2^-53 sqrt(k), S parts have 1 / sqrt(S) of that.  S is the k split that launches of few 128 x 128 units
// had when splitting was what filled the SMs (waves of 148 units, parts of at least 16 steps of eight k, four
// steps of overhead per unit): results of those sizes are as accurate as they were.  Measured relative
// error against 80-bit sums, one chain / parts: plain 2048^3 1.51e-15 / 7.6e-16, 1024 x 2048 x 4096
// 2.13e-15 / 7.6e-16, 222-1 2048^3 2.13e-15 / 1.52e-15, 1501 x 1203 x 999 1.47e-15 / 8.5e-16; us: plain 2048^3 497 /
// 525 (D = 448 506), 1024 x 2048 x 4096 536 / 545, 222-1 2048^3 510 / 519, 1501 x 1203 x 999 168 / 172, the
// 512-problem batch 0.4 % more.  Parts of an eighth of k at every size cost 2 to 5 %.
int sum_depth(int m, int n, int k, int nprod) {
  constexpr int kWave = 148, kStepOverhead = 4, kMinSteps = 16;
  const long long units = tiles_of(m, n, 128) * nprod;
  const int steps = k / 8;
  if (k % 8 != 0 || units >= 8LL * kWave) return k;
  auto cost = [&](int S) { return (double)((units * S + kWave - 1) / kWave) * (steps / S + kStepOverhead); };
  int best = 1;
  for (int S = 2; S <= 8; ++S)
    if (steps % S == 0 && steps / S >= kMinSteps && cost(S) < 0.97 * cost(best)) best = S;
  return best == 1 ? k : (k / best + fmmt::BK - 1) / fmmt::BK * fmmt::BK;
}
int product_depth(const fmm_plan* plan, int ms, int ns, int ks) {
  const int kk = (ks + 7) / 8 * 8;  // of the slots; the same whether or not the products read slots
  return (long long)ms * ns >= (1LL << 17) || plan->rank == 1 ? sum_depth(ms, ns, kk, plan->rank) : kk;
}

// Plain updates up to this deep are bound by their C traffic and run the kernel's SHALLOW form; in columns that do
// not all start on 16 bytes (two accesses a row pair) up to the second.  Measured us without / with: 12000 x
// 12000 x 8 634 / 456, x 40 734 / 633, x 64 853 / 869; 4000 x 4000 x 16 75 / 59; odd 12001 x 12001 x 8 830 / 600,
// x 96 1192 / 1088, x 256 2328 / 2335.
constexpr int kShallowDepth = 48, kShallowDepthOdd = 128;

// One classical update of a tile_gemm launch.
struct GemmJob {
  int m, n, k;
  const double* A;
  long long lda;
  const double* B;
  long long ldb;
  double* C;
  long long ldc;
};

template <int T>
int launch_tile_gemm(const GemmJob* jobs, int njob, int nsm, unsigned* status, cudaStream_t st) {
  fmmt::TileArgs g{};
  int cluster = 1;
  bool parts = false;
  for (int q = 0; q < njob; ++q) {
    fmmt::TileJob& J = g.job[q];
    classical_parts(jobs[q].m, jobs[q].n, jobs[q].k, &J.S, &J.d);
    cluster = std::max(cluster, J.S);
  }
  // parts of a tile are neighbours in a cluster, so every part count has to divide its size: they
  // are powers of two, but for the test hook's, whose jobs then go one by one
  for (int q = 0; q < njob; ++q)
    if (cluster % g.job[q].S != 0) {
      int rc = FMM_OK;
      for (int j = 0; j < njob && rc == FMM_OK; ++j) rc = launch_tile_gemm<T>(jobs + j, 1, nsm, status, st);
      return rc;
    }
  long long first = 0;
  for (int q = 0; q < njob; ++q) {
    const GemmJob& b = jobs[q];
    fmmt::TileJob& J = g.job[q];
    J.A = b.A;
    J.lda = b.lda;
    J.B = b.B;
    J.ldb = b.ldb;
    J.C = b.C;
    J.ldc = b.ldc;
    J.m = b.m;
    J.n = b.n;
    J.k = b.k;
    J.depth = sum_depth(b.m, b.n, b.k, 1);
    parts = parts || J.depth < J.d;
    J.tiles_m = (b.m + T - 1) / T;
    J.tiles_n = (b.n + T - 1) / T;
    J.a_tma = make_a_map(&J.tmA, b.A, b.m, b.k, b.lda);
    J.b_tma = make_b_map(&J.tmB, b.B, b.k, b.n, b.ldb, T);
    const long long units = (long long)J.tiles_m * J.tiles_n * J.S;
    if (first + units > INT32_MAX - fmmt::MAX_SPLIT) return FMM_E_UNSUPPORTED;
    J.first = (int)first;
    J.units = (int)units;
    first += (units + cluster - 1) / cluster * cluster;
  }
  g.njob = njob;
  g.status = status;
  bool shallow = cluster == 1 && !parts;
  for (int q = 0; q < njob; ++q) {
    const bool vec = (reinterpret_cast<uintptr_t>(jobs[q].C) & 15) == 0 && (jobs[q].ldc & 1) == 0;
    shallow = shallow && jobs[q].k <= (vec ? kShallowDepth : kShallowDepthOdd);
  }
  g.ahead = nsm;  // half a round to two rounds of the CTAs took 1 to 5 % longer
  ProfScope ps(K_TILE_GEMM, st);
  auto kernel = shallow ? fmmt::fmm_tile_gemm_kernel<T, T, false, true>
                : parts ? fmmt::fmm_tile_gemm_kernel<T, T, true>
                        : fmmt::fmm_tile_gemm_kernel<T, T, false>;
  return launch_dependent(kernel, dim3((unsigned)first), fmmt::NT,
                          cluster > 1 ? fmmt::TileShape<T, T>::SMEM : spread_smem(fmmt::TileShape<T, T>::SMEM, first, nsm),
                          st, cluster, g);
}

int tile_gemm(const GemmJob* jobs, int njob, cudaStream_t st) {
  int dev = 0;
  const int rc = configure_kernel(&dev);
  if (rc != FMM_OK) return rc;
  GemmJob todo[fmmt::MAX_JOBS];
  int n = 0, S = 1;
  for (int q = 0; q < njob; ++q) {
    if (jobs[q].m <= 0 || jobs[q].n <= 0 || jobs[q].k <= 0) continue;
    int s, d;
    classical_parts(jobs[q].m, jobs[q].n, jobs[q].k, &s, &d);
    S = std::max(S, s);
    todo[n++] = jobs[q];
  }
  if (n == 0) return FMM_OK;
  // a strip that fills the SMs several times (the k strip of a large C) has a launch of its own shape: with the thin
  // strips' 32 x 32 tiles, 222-1 12000 x 12000 x 17 took 2987 us instead of 2860
  for (int q = 0; n > 1 && q < n; ++q)
    if (tiles_of(todo[q].m, todo[q].n, 64) >= 8LL * fmmt::TileShape<64, 64>::CTAS * sm_count[dev]) {
      const GemmJob big = todo[q];
      const int r = tile_gemm(&big, 1, st);
      if (r != FMM_OK) return r;
      todo[q] = todo[n - 1];
      return tile_gemm(todo, n - 1, st);
    }
  if (n == 1 && S == 1 && tile_side(tiles_of(todo[0].m, todo[0].n, 64), tiles_of(todo[0].m, todo[0].n, 32), sm_count[dev]) == 64)
    return launch_tile_gemm<64>(todo, n, sm_count[dev], dev_status[dev], st);
  return launch_tile_gemm<32>(todo, n, sm_count[dev], dev_status[dev], st);
}

// Workspaces of pre-summed operands: slot j of S is ms x kslot, of T kslot x ns (block
// columns), kslot the products' depth; nslot = 0: every operand of that side is a block of A / B.
struct PresumOps {
  const int* plistA = nullptr;  // products of the slots (device)
  const int* plistB = nullptr;
  double* S = nullptr;
  long long ldS = 0;
  int nslotA = 0;
  double* T = nullptr;
  long long ldT = 0;
  int nslotB = 0;
};

// Every k group of a product reads only its own operand blocks: ks is a multiple of eight, or
// the plan is one product of whole operands, where the tensor maps end at their last k column
// / row and a partial last group reads TMA's zero fill.
bool whole_k_steps(const fmm_plan* plan, int ks) {
  return ks % 8 == 0 || (plan->rank == 1 && plan->dims[0] == 1 && plan->dims[1] == 1 && plan->dims[2] == 1);
}

// Tile side of a products launch and its tickets: per (tile, C block) where a product has no
// more tiles than CTAs run at a time (the units of one tile then run together, and one ticket
// per tile would chain all R updates), else per tile.
struct ProdLaunch {
  int tile = 64;
  size_t tickets = 0;
  int nbt = 0, nbc = 0;
  bool by_tiles = false;  // a unit per tile with all its products (no tickets)
};

ProdLaunch plan_products(const int grid_dims[3], int nprod, int mode, int ms, int ns, int nsm, bool by_tiles = false) {
  ProdLaunch L;
  L.tile = by_tiles ? 64 : product_tile(ms, ns, nprod, nsm);
  L.by_tiles = by_tiles;
  if (mode == fmm::MODE_ACCUM_C && nprod > 1 && !by_tiles) {
    const long long ntiles = tiles_of(ms, ns, L.tile);
    if (ntiles <= kResident64 * (long long)nsm) {
      L.nbt = grid_dims[0] * grid_dims[2];
      L.nbc = grid_dims[2];
    }
    L.tickets = 4 * (size_t)ntiles * (L.nbt > 0 ? L.nbt : 1);
  }
  return L;
}

// The products of a plan over sub-blocks ms x ns with k depth kk (kk: the slots' depth, ks:
// the operands' own); counter: the launch's work-unit counter and then its tickets, zeroed.
int launch_products(const fmm::Prod* prods, const fmm::Term* terms, const int grid_dims[3], int nprod, int mode,
                    const double* A, long long lda, const double* B, long long ldb, const PresumOps& ps, double* C,
                    long long ldc, double* M, int ms, int ns, int ks, int kk, int depth, const ProdLaunch& L,
                    int* counter, cudaStream_t st) {
  int dev = 0;
  int rc = configure_kernel(&dev);
  if (rc != FMM_OK) return rc;
  fmmt::ProdArgs a{};
  a.A = A;
  a.lda = lda;
  a.B = B;
  a.ldb = ldb;
  a.C = C;
  a.ldc = ldc;
  a.M = M;
  a.m_stride = (long long)ms * ns;
  a.prods = prods;
  a.terms = terms;
  a.ms = ms;
  a.ns = ns;
  a.ks = kk;
  a.depth = depth;
  a.nprod = nprod;
  a.tiles_m = (ms + L.tile - 1) / L.tile;
  a.tiles_n = (ns + L.tile - 1) / L.tile;
  a.chunks = L.by_tiles ? 1 : nprod;
  a.mode = mode;
  a.status = dev_status[dev];
  a.counter = counter;
  a.tickets = L.tickets ? counter + 1 : nullptr;
  a.nbt = L.nbt;
  a.nbc = L.nbc;
  a.a_tma = a.b_tma = 1;
  const long long units = (long long)a.tiles_m * a.tiles_n * a.chunks;
  const int nsm = sm_count[dev];
  const bool cut = !L.by_tiles && L.tile == 64 && L.tickets == 0 && kk >= kTailDepth && cut_tail((double)units / nsm);
  const long long tail = cut ? units % nsm : 0;
  const long long claims = units + (64 / fmmt::TAIL_ROWS - 1) * tail;
  if (claims > INT32_MAX) return FMM_E_UNSUPPORTED;
  a.tail = (int)(units - tail);
  a.claims = (int)claims;
  const long long am = (long long)grid_dims[0] * ms, ak = (long long)grid_dims[1] * ks, bn = (long long)grid_dims[2] * ns;
  bool ok = true;
  if (ps.nslotA < nprod) ok = ok && make_a_map(&a.tmA, A, am, ak, lda);
  if (ps.nslotB < nprod) ok = ok && make_b_map(&a.tmB, B, ak, bn, ldb, L.tile);
  if (ps.nslotA > 0) ok = ok && make_a_map(&a.tmAw, ps.S, ms, (long long)ps.nslotA * kk, ps.ldS);
  if (ps.nslotB > 0) ok = ok && make_b_map(&a.tmBw, ps.T, kk, (long long)ps.nslotB * ns, ps.ldT, L.tile);
  if (!ok) return FMM_E_UNSUPPORTED;
  const int per_sm = L.tile == 64 ? fmmt::TileShape<64, 64>::CTAS : fmmt::TileShape<32, 32>::CTAS;
  const unsigned grid = (unsigned)std::min<long long>(claims, (long long)nsm * per_sm);
  ProfScope pf(K_PRODUCTS, st);
  const bool parts = depth < kk;
  if (L.tile == 64) {
    auto kernel = tail > 0 ? (parts ? fmmt::fmm_products_kernel<64, true, true> : fmmt::fmm_products_kernel<64, true, false>)
                           : (parts ? fmmt::fmm_products_kernel<64, false, true> : fmmt::fmm_products_kernel<64, false, false>);
    return launch_dependent(kernel, dim3(grid), fmmt::NT, spread_smem(fmmt::ProdShape<64>::SMEM, grid, nsm), st, 1, a);
  }
  return launch_dependent(parts ? fmmt::fmm_products_kernel<32, false, true> : fmmt::fmm_products_kernel<32, false, false>,
                          dim3(grid), fmmt::NT, spread_smem(fmmt::ProdShape<32>::SMEM, grid, nsm), st, 1, a);
}

const int kUnitGrid[3] = {1, 1, 1};

int sm_count_current() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  return sm_count[dev];
}

// A classical update.  Operands with an odd leading dimension cannot be read by tensor copies;
// the per-lane copies that read them in place cost about 14 % of a large update (3001^3 1790 us
// against 1535 us at 3008^3), copying the operand once to an even pitch 16 bytes an element at
// about 4.6 TB/s.
int plain_gemm(int m, int n, int k, const double* A, long long lda, const double* B, long long ldb, double* C,
               long long ldc, cudaStream_t st) {
  if (m <= 0 || n <= 0 || k <= 0) return FMM_OK;
  const bool odd_a = (lda & 1) != 0, odd_b = (ldb & 1) != 0;
  const double gain = 0.14 * 2.0 * m * n * k / 35e12;
  const double cost = 16.0 * ((odd_a ? (double)m * k : 0.0) + (odd_b ? (double)k * n : 0.0)) / 4.6e12 + 8e-6;
  if ((!odd_a && !odd_b) || gain < cost || (odd_a && (reinterpret_cast<uintptr_t>(B) & 15) != 0 && !odd_b) ||
      (odd_b && (reinterpret_cast<uintptr_t>(A) & 15) != 0 && !odd_a)) {
    const GemmJob j{m, n, k, A, lda, B, ldb, C, ldc};
    return tile_gemm(&j, 1, st);
  }
  const long long pa = m + (m & 1), pb = k + (k & 1);
  const size_t sa = odd_a ? (sizeof(double) * (size_t)pa * k + 255) & ~(size_t)255 : 0;
  const size_t sb = odd_b ? sizeof(double) * (size_t)pb * n : 0;
  char* ws = nullptr;
  FMM_CUDA_TRY(cudaMallocAsync((void**)&ws, sa + sb, st));
  GemmJob j{m, n, k, A, lda, B, ldb, C, ldc};
  {
    ProfScope pf(K_PITCH_COPY, st);
    if (odd_a) {
      j.A = reinterpret_cast<double*>(ws);
      j.lda = pa;
      fmm::fmm_pitch_copy1_kernel<<<2048, 256, 0, st>>>(fmm::PitchCopy{A, lda, reinterpret_cast<double*>(ws), pa, m, k});
      g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    if (odd_b) {
      j.B = reinterpret_cast<double*>(ws + sa);
      j.ldb = pb;
      fmm::fmm_pitch_copy1_kernel<<<2048, 256, 0, st>>>(fmm::PitchCopy{B, ldb, reinterpret_cast<double*>(ws + sa), pb, k, n});
      g_launches.fetch_add(1, std::memory_order_relaxed);
    }
  }
  int rc = cuda_status(cudaGetLastError());
  if (rc == FMM_OK) rc = tile_gemm(&j, 1, st);
  cudaError_t fe = cudaFreeAsync(ws, st);
  return rc == FMM_OK ? cuda_status(fe) : rc;
}

int grid_for(long long total, int threads) {
  long long b = (total + threads - 1) / threads;
  if (b > 148LL * 16) b = 148LL * 16;
  if (b < 1) b = 1;
  return (int)b;
}

// Fringe GEMMs, the regions of the reference's dynamic peeling: the k strip updates the core's
// C, the n strip the last columns, the m strip the last rows; the three are disjoint in C, so
// one launch covers them.
int peel(int m, int n, int k, const double* A, long long lda, const double* B, long long ldb, double* C,
         long long ldc, int dim1, int dim2, int dim3, cudaStream_t st) {
  const int mr = m % dim1, kr = k % dim2, nr = n % dim3;
  const int ms = m - mr, ns = n - nr, ks = k - kr;
  const GemmJob jobs[3] = {{m, nr, k, A, lda, B + (long long)ns * ldb, ldb, C + (long long)ns * ldc, ldc},
                           {mr, ns, k, A + ms, lda, B, ldb, C + ms, ldc},
                           {ms, ns, kr, A + (long long)ks * lda, lda, B + ks, ldb, C, ldc}};
  return tile_gemm(jobs, 3, st);
}

// C_l += sum_r W[l,r] * M_r for every C block at once (fmm_combine_kernel); false when the
// plan's grouped tables do not fit the kernel's shared memory (the caller then uses the
// per-block scatter).
bool combine_fits(const fmm_plan* plan) {
  return plan->n_cgroup > 0 &&
         fmm::combine_group_smem_bytes(plan->n_cgroup, (int)plan->cg_r.size(), (int)plan->cg_c.size()) <= 200 * 1024;
}

bool combine_configured[kMaxDevices];
// element positions per thread of the combine (fmm_debug_set FMM_DEBUG_COMBINE_POSITIONS; 0: 1)
std::atomic<int> g_combine_positions{0};

int launch_combine(const fmm_plan* plan, const DevTables& d, double* C, long long ldc, int ms, int ns,
                   const double* M, long long ldm, long long m_stride, cudaStream_t st) {
  int dev = 0;
  int rc0 = configure_kernel(&dev);
  if (rc0 != FMM_OK) return rc0;
  {
    std::lock_guard<std::mutex> lk(g_attr_mu);
    if (!combine_configured[dev]) {
      FMM_CUDA_TRY(cudaFuncSetAttribute(fmm::fmm_combine_staged_kernel<false>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
      FMM_CUDA_TRY(cudaFuncSetAttribute(fmm::fmm_combine_staged_kernel<true>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
      FMM_CUDA_TRY(cudaFuncSetAttribute(fmm::fmm_combine_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        200 * 1024));
      FMM_CUDA_TRY(cudaFuncSetAttribute(fmm::fmm_combine_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        200 * 1024));
      combine_configured[dev] = true;
    }
  }
  fmm::CombineGroupArgs ga{};
  ga.C = C;
  ga.ldc = ldc;
  ga.ms = ms;
  ga.ns = ns;
  ga.M = M;
  ga.ldm = ldm;
  ga.m_stride = m_stride;
  ga.grid_n = plan->dims[2];
  ga.ngroup = plan->n_cgroup;
  ga.nent = (int)plan->cg_r.size();
  ga.ncoef = (int)plan->cg_c.size();
  ga.gdesc = d.cg_desc;
  ga.er = d.cg_r;
  ga.em = d.cg_m;
  ga.ec = d.cg_c;
  ga.nprod = plan->rank;
  const long long total = (long long)ms * ns;
  ga.nchunk = (int)plan->ch_n.size();
  ga.nop = (int)plan->ch_op.size();
  ga.chr = d.ch_r;
  ga.chn = d.ch_n;
  ga.op = d.ch_op;
  const size_t ssm = fmm::combine_staged_smem_bytes(ga.ngroup, ga.nchunk, ga.nop);
  // staged form: the M tiles of a position range are contiguous 16-byte-aligned runs
  const bool staged = g_combine_positions.load() == 0 && ldm == ms && m_stride % 2 == 0 && ms % 2 == 0 &&
                      ((uintptr_t)M & 15) == 0 && ssm <= 200 * 1024 && total > 0;
  if (staged) {
    const long long tiles = (total + fmm::CST_TILE - 1) / fmm::CST_TILE;
    const bool split = tiles < 3LL * sm_count[dev];  // too few tiles to fill the chip: a unit per group
    const long long ntile = tiles * (split ? ga.ngroup : 1);
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(ntile, (long long)sm_count[dev] * 3));
    {
      ProfScope pf(K_COMBINE, st);
      return launch_dependent(split ? fmm::fmm_combine_staged_kernel<true> : fmm::fmm_combine_staged_kernel<false>,
                              dim3(grid), fmm::CST_THREADS + 32, spread_smem(ssm, grid, sm_count[dev]), st, 1, ga,
                              dev_status[dev]);
    }
  }
  const int P = g_combine_positions.load() == 2 ? 2 : 1;
  const size_t smem = fmm::combine_group_smem_bytes(ga.ngroup, ga.nent, ga.ncoef);
  const long long per = (long long)fmm::COMBINE_G_THREADS * P;
  const long long blocks = ((long long)ms * ns + per - 1) / per;
  const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(blocks, (long long)sm_count_current() * 8));
  {
    ProfScope pf(K_COMBINE, st);
    if (P == 2)
      fmm::fmm_combine_kernel<2><<<grid, fmm::COMBINE_G_THREADS, smem, st>>>(ga);
    else
      fmm::fmm_combine_kernel<1><<<grid, fmm::COMBINE_G_THREADS, smem, st>>>(ga);
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cuda_status(cudaGetLastError());
}

// ABC schedule of a call (all give the same bits).
//   STORED: the products stored to a workspace and one combine pass (every M_r and C element crossing HBM once).
//   DIRECT: the multi-destination epilogue, C_l += W[l,r] M_r straight from each product tile, a unit per tile and
//     product, ordered by tickets.
//   DIRECT_TILES: the same, a unit per tile with all its products: its C tiles stay in L2 from update to update.
// The lines between them, measured on B200 (us stored / direct / direct by tiles):
//   * Few tiles: when a product has no more tiles than CTAs run at a time, the units of one tile run together
//     and their ordered C updates form a chain: stored.  222-1 1024^3 97 / 119; 222-2 1024^3 112 / 189;
//     222-1 x 333-1 2016^3 673 / 1165.
//   * C traffic: the epilogue moves 16 nnz(W) ms ns bytes of C, at 3 TB/s where nothing else bounds it, the stored
//     schedule 8 R ms ns and, after the products, 8 (R + 2 blocks) ms ns.  The model below (products at 35
//     TFLOP/s) picks the faster of the two at all of 204 sizes from 4000^2 to 14400^2, block depth 4 to 2048,
//     five plans: 222-1 12000^2 x 128 1825 / 2562, x 512 4484 / 4494, x 1024 8092 / 7836; 222-1 x 333-1 12000^2 x
//     1008 8269 / 13900.
//   * By tiles, where the tiles fill the SMs eight times and the C tiles of a CTA's few blocks stay in L2, up to
//     2.5 times as long for the products as for C (222-1 12000^2: x 128 1833, x 512 4293, x 1024 7776, x 2048
//     15011 against 14991; 4000^2 x 512, 1024 tiles, 578; 222-2, 16 blocks, 12000^2 x 512 7557 against 4644), and
//     against stored with at most four blocks and products that take at least 0.6 of its C updates' time (222-1 x 64
//     1532 against 1448, 232-1 x 504 4618 against 4848), in aligned columns (222-1 8001^2 x 128 1002 against 880).
// The product workspace (8 R ms ns bytes) must fit the workspace cap, and so must the operand sums
// (run_core: deep k makes them large where the products are few and small).  It is the reference's
// own trade between its ABC and AB variants (meta/model_gen.py:87-95 counts the C memory
// operations of each).
enum AbcSchedule : int { ABC_STORED = 0, ABC_DIRECT = 1, ABC_DIRECT_TILES = 2 };
AbcSchedule abc_schedule(const fmm_plan* plan, int ms, int ns, int ks, bool vec, int nsm) {
  const double mn = (double)ms * ns;
  const int nblk = plan->dims[0] * plan->dims[2];
  const long long ntiles = tiles_of(ms, ns, 64), resident = kResident64 * (long long)nsm;
  const bool room = plan->rank > 1 && combine_fits(plan) && 8.0 * plan->rank * mn <= (double)g_ws_limit.load();
  if (room && ntiles <= resident) return ABC_STORED;
  const double t_mma = 2.0 * plan->rank * mn * ks / 35e12;
  const double t_epi = 16.0 * plan->n_cterms * mn / 3e12;
  const double t_store = 8.0 * plan->rank * mn / 5e12;
  const double t_comb = 8.0 * (plan->rank + 2.0 * nblk) * mn / 4e12;
  const bool by_tiles = plan->rank > 1 && nblk <= 9 && ntiles >= 8 * resident && t_mma < 2.5 * t_epi;
  if (by_tiles && nblk <= 4 && vec && t_mma > 0.35 * t_epi) return ABC_DIRECT_TILES;  // C updates by tiles: 5.2 TB/s
  const double hi = std::max(t_mma, t_epi), lo = std::min(t_mma, t_epi);
  if (room && 0.98 * std::max(t_mma, t_store) + t_comb < hi + 0.7 * lo * lo / hi) return ABC_STORED;
  return by_tiles ? ABC_DIRECT_TILES : ABC_DIRECT;
}

// The pre-summed form of one call: which operands get slots, the tables the products kernel
// reads them with, and the workspace.  With k per product a whole number of k groups and both
// operands readable by tensor copies, single-block operands are read in place and only sums
// get slots; otherwise (or when every sum is wanted) every product gets a slot of its own,
// whose k extent is rounded up with zeros.
struct PresumPlan {
  bool all = false;
  int kk = 0;                // k depth of the products
  int nA = 0, nB = 0;        // slots
  long long ldS = 0, ldT = 0;
  size_t s_bytes = 0, t_bytes = 0;
};

PresumPlan presum_plan(const fmm_plan* plan, int ms, int ns, int ks, bool all) {
  PresumPlan pp;
  pp.all = all || !whole_k_steps(plan, ks);
  pp.kk = pp.all ? (ks + 7) / 8 * 8 : ks;
  pp.nA = pp.all ? plan->rank : (int)plan->plistA.size();
  pp.nB = pp.all ? plan->rank : (int)plan->plistB.size();
  pp.ldS = (ms + 1) / 2 * 2;
  pp.ldT = (pp.kk + 1) / 2 * 2;
  pp.s_bytes = (sizeof(double) * (size_t)pp.ldS * pp.kk * pp.nA + 255) & ~(size_t)255;
  pp.t_bytes = (sizeof(double) * (size_t)pp.ldT * ns * pp.nB + 255) & ~(size_t)255;
  return pp;
}

// One side's sums of products plist[0 .. n) into `out`.
fmm::PresumSide presum_side(const DevTables& d, int side, const double* X, long long ldx, int ms, int ns, int ks, int kk,
                            double* out, long long ldo, const int* plist, int n) {
  fmm::PresumSide p{};
  p.X = X;
  p.ldx = ldx;
  p.rows = side == 0 ? ms : ks;
  p.cols = side == 0 ? ks : ns;
  p.orows = (int)ldo;  // even; the pitch element of an odd row count is a zero
  p.ocols = side == 0 ? kk : ns;
  p.blk_row_stride = p.rows;
  p.blk_col_stride = p.cols;
  p.out = out;
  p.ldo = ldo;
  p.out_stride = ldo * p.ocols;
  p.plist = plist;
  p.first = d.ps_first[side];
  p.terms = d.ps_terms[side];
  p.nout = n;
  return p;
}

// Terms of the larger side and the output ranges per position chunk: enough CTAs to fill the
// SMs several times, else one CTA walks all its outputs so that they share its input values.
constexpr int kPsChunk = fmm::PS_THREADS;  // positions of a presum CTA
int presum_cap(const fmm_plan* plan) {
  return (int)std::min<size_t>(fmm::PS_TERMS, std::max(plan->ps_terms[0].size(), plan->ps_terms[1].size()));
}
unsigned presum_ranges(long long chunks, int nout, int nsm) {
  long long y = (8LL * nsm + chunks - 1) / std::max<long long>(1, chunks);
  return (unsigned)std::max<long long>(1, std::min<long long>(y, nout));
}

// Both sides' sums; zero[0 .. nzero) is cleared too (with no sums to make, by a memset).
int launch_presum(const fmm_plan* plan, const fmm::PresumSide& a, const fmm::PresumSide& b, int* zero, long long nzero,
                  int nsm, cudaStream_t st) {
  if (a.nout == 0 && b.nout == 0)
    return nzero > 0 ? cuda_status(cudaMemsetAsync(zero, 0, sizeof(int) * nzero, st)) : FMM_OK;
  if (nzero > INT32_MAX) return FMM_E_UNSUPPORTED;
  fmm::PresumArgs g{};
  g.s[0] = a;
  g.s[1] = b;
  g.zero = zero;
  g.nzero = (int)nzero;
  g.cap = presum_cap(plan);
  g.s[0].brows = plan->dims[0];
  g.s[0].bcols = g.s[1].brows = plan->dims[1];
  g.s[1].bcols = plan->dims[2];
  const int nblk = std::max(plan->dims[0] * plan->dims[1], plan->dims[1] * plan->dims[2]);
  const size_t staged = fmm::presum_staged_smem(nblk, g.cap);
  auto staged_chunks = [](const fmm::PresumSide& x) {
    return x.nout ? ((long long)(x.orows / 2) * x.ocols + fmm::PSS_THREADS - 1) / fmm::PSS_THREADS : 0;
  };
  const long long nsc = staged_chunks(a) + staged_chunks(b);
  // the staged form where two CTAs fit an SM and every SM has a chunk (below: 222-1 x 333-1 528^3
  // 20.7 us staged, 19.0 gathered)
  if (staged <= kPsStagedSmem && nsc >= nsm &&
      std::max(plan->ps_terms[0].size(), plan->ps_terms[1].size()) <= fmm::PS_TERMS) {
    const long long per = std::min<long long>(8, kSmSmem / (staged + kCtaReserve));
    const unsigned gx = (unsigned)std::min<long long>(nsc, per * nsm);
    const long long y = (per * nsm + nsc - 1) / nsc;
    ProfScope pf(K_PRESUM, st);
    return launch_dependent(fmm::fmm_presum_staged_kernel,
                            dim3(gx, (unsigned)std::min<long long>(y, std::max(a.nout, b.nout))), fmm::PSS_THREADS,
                            staged, st, 1, g);
  }
  const long long ca = (long long)(a.orows / 2) * a.ocols, cb = (long long)(b.orows / 2) * b.ocols;
  const long long nca = a.nout ? (ca + kPsChunk - 1) / kPsChunk : 0, ncb = b.nout ? (cb + kPsChunk - 1) / kPsChunk : 0;
  const long long nc = nca + ncb;
  const unsigned gx = (unsigned)std::max<long long>(1, std::min<long long>(nc, 4LL * nsm));
  ProfScope pf(K_PRESUM, st);
  return launch_dependent(fmm::fmm_presum_kernel, dim3(gx, presum_ranges(nc, std::max(a.nout, b.nout), nsm)),
                          fmm::PS_THREADS, fmm::presum_smem_bytes(g.cap), st, 1, g);
}

// Bytes of the pre-summed workspace of one call.
size_t presum_bytes(const PresumPlan& pp) { return pp.s_bytes + pp.t_bytes; }

// C_l += sum_r W[l,r] M_r for stored products (product r at M + r ms ns).
int apply_stored(const fmm_plan* plan, const DevTables& d, double* C, long long ldc, int ms, int ns, const double* M,
                 cudaStream_t st) {
  if (combine_fits(plan)) return launch_combine(plan, d, C, ldc, ms, ns, M, ms, (long long)ms * ns, st);
  fmm::ScatterArgs sa{};
  sa.C = C;
  sa.ldc = ldc;
  sa.ms = ms;
  sa.ns = ns;
  sa.M = M;
  sa.ldm = ms;
  sa.m_stride = (long long)ms * ns;
  sa.cblk = d.cblk;
  sa.ent_r = d.ent_r;
  sa.ent_w = d.ent_w;
  const dim3 gs((unsigned)grid_for(sa.m_stride, 256), (unsigned)plan->n_cblk);
  ProfScope pf(K_SCATTER, st);
  fmm::fmm_scatter_kernel<<<gs, 256, 0, st>>>(sa);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cuda_status(cudaGetLastError());
}

// Pre-summed products in groups, when one call's whole operand workspace would exceed the
// workspace limit: the R products run as groups of G consecutive products, each group's
// operand sums (one slot per product, k extent padded to whole k groups) formed in the one
// workspace before its products run.  (Two half-size buffers with the next group's sums on a
// second stream measured slower: the products' CTAs fill the SMs, so the sums ran between the
// products launches all the same, and twice the groups read A and B twice as often: 16384^3
// 222-1 x 333-1 200.6 ms.)  Groups run in product order, so every C element still receives its
// products' updates in order r = 0..R-1 (results are those of the ungrouped call).  Workspace
// G (ms + ns) kk 8 bytes, within the limit for G >= 1, and less where it cannot be allocated.  stored (the
// ab pack type): the products go to a workspace of their own and W is applied at the end.
int run_presum_groups(const fmm_plan* plan, const DevTables& d, const double* A, long long lda, const double* B,
                      long long ldb, double* C, long long ldc, int ms, int ns, int ks, int nsm, bool stored,
                      cudaStream_t st) {
  const int R = plan->rank;
  const int kk = (ks + 7) / 8 * 8;
  const long long ldS = (ms + 1) / 2 * 2;
  const size_t sb = sizeof(double) * (size_t)ldS * kk, tb = sizeof(double) * (size_t)kk * ns;
  long long G = g_ws_limit.load() / (long long)(sb + tb);
  G = std::max<long long>(1, std::min<long long>(G, R));
  const int mode = stored ? fmm::MODE_STORE_M : fmm::MODE_ACCUM_C;
  const size_t mb = stored ? sizeof(double) * (size_t)ms * ns * R : 0;
  ProdLaunch L;
  size_t tk = 0;
  char* ws = nullptr;
  for (;;) {
    const int ng = (int)((R + G - 1) / G);
    G = (R + ng - 1) / ng;  // even groups
    L = plan_products(plan->dims, (int)G, mode, ms, ns, nsm);
    tk = (sizeof(int) * (1 + L.tickets) + 255) & ~(size_t)255;
    const size_t sums = ((size_t)G * (sb + tb) + 255) & ~(size_t)255;
    const cudaError_t e = cudaMallocAsync((void**)&ws, tk + sums + mb, st);
    if (e == cudaSuccess) break;
    if (e != cudaErrorMemoryAllocation || G == 1) return cuda_status(e);
    cudaGetLastError();
    G = G / 2;
  }
  t_last_ws = (long long)(G * (sb + tb));
  double* M = stored ? reinterpret_cast<double*>(ws + tk + (((size_t)G * (sb + tb) + 255) & ~(size_t)255)) : nullptr;
  int* counter = reinterpret_cast<int*>(ws);
  int rc = FMM_OK;
  for (int g0 = 0; g0 < R && rc == FMM_OK; g0 += (int)G) {
    const int g1 = (int)std::min<long long>(R, g0 + G), n = g1 - g0;
    PresumOps ps;
    ps.S = reinterpret_cast<double*>(ws + tk);
    ps.ldS = ldS;
    ps.nslotA = n;
    ps.T = reinterpret_cast<double*>(ws + tk + G * sb);
    ps.ldT = kk;
    ps.nslotB = n;
    rc = launch_presum(plan, presum_side(d, 0, A, lda, ms, ns, ks, kk, ps.S, ps.ldS, d.plist_all + g0, n),
                       presum_side(d, 1, B, ldb, ms, ns, ks, kk, ps.T, ps.ldT, d.plist_all + g0, n), counter,
                       1 + (long long)L.tickets, nsm, st);
    const fmm::Prod* gp = nullptr;
    const fmm::Term* gt = nullptr;
    if (rc == FMM_OK) rc = ksplit_tables(plan, BASE_GROUP, g0, &gp, &gt, g1);
    if (rc == FMM_OK)
      rc = launch_products(gp, gt, plan->dims, n, mode, A, lda, B, ldb, ps, C, ldc,
                           stored ? M + (long long)g0 * ms * ns : nullptr, ms, ns, ks, kk, product_depth(plan, ms, ns, ks),
                           L, counter, st);
  }
  if (rc == FMM_OK && stored) rc = apply_stored(plan, d, C, ldc, ms, ns, M, st);
  cudaError_t fe = cudaFreeAsync(ws, st);
  return rc == FMM_OK ? cuda_status(fe) : rc;
}

int check_args(int m, int n, int k, const void* A, long long lda, const void* B, long long ldb, const void* C,
               long long ldc) {
  if (m < 0 || n < 0 || k < 0) return FMM_E_INVALID;
  if (m == 0 || n == 0 || k == 0) return FMM_OK;
  if (!A || !B || !C) return FMM_E_INVALID;
  if (lda < m || ldb < k || ldc < m) return FMM_E_INVALID;
  return FMM_OK;
}

bool is_classical(const fmm_plan* p) {
  return p->rank == 1 && p->dims[0] == 1 && p->dims[1] == 1 && p->dims[2] == 1 && p->plistA.empty() &&
         p->plistB.empty() && p->prods[0].nc == 1 && p->terms[p->prods[0].c0].coef == 1.0;
}

// The FMM core: sub-blocks ms x ks x ns, every dimension a whole number of them.
//   abc: operand sums in HBM, then every product either added to its C blocks as it is made
//        (tickets keep each C element's updates in product order) or, where that C traffic or
//        the launch's few units dominate, stored and applied by one combine pass;
//   ab, naive: the products stored, W applied by the combine pass (naive makes a temporary
//        of every operand).
int run_core(const fmm_plan* plan, int pack, const double* A, long long lda, const double* B, long long ldb, double* C,
             long long ldc, int ms, int ns, int ks, cudaStream_t st) {
  DevTables* d = nullptr;
  int rc = device_tables(plan, &d);
  if (rc != FMM_OK) return rc;
  int dev = 0;
  rc = configure_kernel(&dev);
  if (rc != FMM_OK) return rc;
  const int R = plan->rank, nsm = sm_count[dev];
  // operands a tensor copy cannot read in place (odd leading dimension, unaligned base) all get slots
  CUtensorMap probe;
  const bool in_place = make_a_map(&probe, A, (long long)plan->dims[0] * ms, (long long)plan->dims[1] * ks, lda) &&
                        make_b_map(&probe, B, (long long)plan->dims[1] * ks, (long long)plan->dims[2] * ns, ldb, 64);
  const PresumPlan pp = presum_plan(plan, ms, ns, ks, pack == FMM_PACK_NAIVE || !in_place);
  // an ABC call whose operand sums exceed the workspace cap runs in groups, whatever its C traffic
  const bool capped = pack == FMM_PACK_ABC && (long long)presum_bytes(pp) > g_ws_limit.load();
  const bool vec = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && (ldc & 1) == 0;
  AbcSchedule sched = pack != FMM_PACK_ABC ? ABC_STORED : abc_schedule(plan, ms, ns, ks, vec, nsm);
  if (pack == FMM_PACK_ABC && g_ticket_fill != 0) sched = ABC_DIRECT;  // the schedule with tickets
  const bool stored = sched == ABC_STORED;
  if (capped) return run_presum_groups(plan, *d, A, lda, B, ldb, C, ldc, ms, ns, ks, nsm, false, st);
  const int mode = stored ? fmm::MODE_STORE_M : fmm::MODE_ACCUM_C;
  const ProdLaunch L = plan_products(plan->dims, R, mode, ms, ns, nsm, sched == ABC_DIRECT_TILES);
  const size_t tk = (sizeof(int) * (1 + L.tickets) + 255) & ~(size_t)255;
  const size_t mb = stored ? sizeof(double) * (size_t)ms * ns * R : 0;
  char* ws = nullptr;
  const cudaError_t ae = cudaMallocAsync((void**)&ws, tk + presum_bytes(pp) + mb, st);
  if (ae == cudaErrorMemoryAllocation && pack != FMM_PACK_NAIVE) {  // no room: a group's sums at a time
    cudaGetLastError();
    return run_presum_groups(plan, *d, A, lda, B, ldb, C, ldc, ms, ns, ks, nsm, pack == FMM_PACK_AB, st);
  }
  FMM_CUDA_TRY(ae);
  t_last_ws = (long long)presum_bytes(pp);
  int* counter = reinterpret_cast<int*>(ws);
  double* M = stored ? reinterpret_cast<double*>(ws + tk + presum_bytes(pp)) : nullptr;
  PresumOps ps;
  ps.plistA = pp.all ? d->plist_all : d->plistA;
  ps.plistB = pp.all ? d->plist_all : d->plistB;
  ps.S = reinterpret_cast<double*>(ws + tk);
  ps.ldS = pp.ldS;
  ps.nslotA = pp.nA;
  ps.T = reinterpret_cast<double*>(ws + tk + pp.s_bytes);
  ps.ldT = pp.ldT;
  ps.nslotB = pp.nB;
  rc = launch_presum(plan, presum_side(*d, 0, A, lda, ms, ns, ks, pp.kk, ps.S, ps.ldS, ps.plistA, ps.nslotA),
                     presum_side(*d, 1, B, ldb, ms, ns, ks, pp.kk, ps.T, ps.ldT, ps.plistB, ps.nslotB), counter,
                     1 + (long long)L.tickets, nsm, st);
  if (rc == FMM_OK && g_ticket_fill != 0 && L.tickets > 0)
    rc = cuda_status(cudaMemsetAsync(counter + 1, g_ticket_fill, sizeof(int) * L.tickets, st));
  if (rc == FMM_OK)
    rc = launch_products(pp.all ? d->prods_all : d->prods_ps, pp.all ? d->terms_all : d->terms_ps, plan->dims, R, mode, A,
                         lda, B, ldb, ps, C, ldc, M, ms, ns, ks, pp.kk, product_depth(plan, ms, ns, ks), L, counter, st);
  if (rc == FMM_OK && stored) rc = apply_stored(plan, *d, C, ldc, ms, ns, M, st);
  cudaError_t fe = cudaFreeAsync(ws, st);
  return rc == FMM_OK ? cuda_status(fe) : rc;
}

int run_fmm(const fmm_plan* plan, int pack, int m, int n, int k, const double* A, long long lda, const double* B,
            long long ldb, double* C, long long ldc, cudaStream_t st) {
  if (!plan) return FMM_E_NOPLAN;
  if (pack != FMM_PACK_ABC && pack != FMM_PACK_AB && pack != FMM_PACK_NAIVE) return FMM_E_UNSUPPORTED;
  int rc = check_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != FMM_OK) return rc;
  if (m == 0 || n == 0 || k == 0) return FMM_OK;
  t_last_ws = 0;
  if (is_classical(plan)) return plain_gemm(m, n, k, A, lda, B, ldb, C, ldc, st);
  const int pm = plan->dims[0] * kMR, pk = plan->dims[1], pn = plan->dims[2] * kNR;
  const int md = m - m % pm, kd = k - k % pk, nd = n - n % pn;
  if (md > 0 && kd > 0 && nd > 0) {
    rc = run_core(plan, pack, A, lda, B, ldb, C, ldc, md / plan->dims[0], nd / plan->dims[2], kd / plan->dims[1], st);
    if (rc != FMM_OK) return rc;
  }
  return peel(m, n, k, A, lda, B, ldb, C, ldc, pm, pk, pn, st);
}

int noalloc_status(int dev, bool clear);  // the no-allocation entry point's status word (below)
bool noalloc_used(int dev);

int device_status(bool clear) {
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return FMM_E_UNSUPPORTED;
  unsigned v = 0;
  if (smem_configured[dev]) {
    FMM_CUDA_TRY(cudaMemcpy(&v, dev_status[dev], sizeof(unsigned), cudaMemcpyDeviceToHost));
    if (clear && v) FMM_CUDA_TRY(cudaMemset(dev_status[dev], 0, sizeof(unsigned)));
  }
  const int rn = noalloc_status(dev, clear);
  if (rn != FMM_OK && rn != FMM_E_TIMEOUT) return rn;
  if (v & fmm::STATUS_TABLE) return FMM_E_PLAN;
  return (v || rn == FMM_E_TIMEOUT) ? FMM_E_TIMEOUT : FMM_OK;
}

// Host-pointer execution: stage A, B, C into device memory, run, copy C back.
//
// Large problems run as a grid of R row panels x P column panels of C, each block
// C[I, J] += A[I, :] * B[:, J] a GEMM of its own (partitioned like any |I| x |J| x k call), so
// that the copies overlap the compute.  Blocks run column panel by column panel, the row
// panels inside: the copy-in stream brings, in that order, each block's operands that are not
// on the device yet (A[I, :] at its first use, B[:, J] at its first use, C[I, J]); the
// calling thread's stream computes block b once its copies have landed while the next
// blocks' operands come in; a copy-out stream returns C[I, J] after its block (host-to-
// device and device-to-host copies run at the same time).  Before the first kernel only
// A[I_0, :], B[:, J_0] and C[I_0, J_0] are copied: with two row panels half of A instead of
// all of it (16384^3: 1.8 instead of 3.2 GB).  Row and column edges fall on multiples of 128 x
// (block rows / columns of the plan), so every block's sub-blocks are whole tiles where the
// size allows.
#ifndef FMM_HOST_PANELS
#define FMM_HOST_PANELS 4
#endif
constexpr int kHostPanelMinCols = 512;               // column panels at least this wide
constexpr long long kHostPanelMinElems = 1LL << 20;  // C of at least 8 MB
constexpr long long kHostRowSplitMinA = 1LL << 26;   // two row panels once A has 2^26 elements (512 MB)
constexpr int kHostRowPanelMinRows = 4096;

void split_edges(int total, int parts, int unit, std::vector<int>* edges) {
  edges->assign(1, 0);
  for (int j = 1; j < parts; ++j) {
    long long e = (long long)total * j / parts;
    if (total / parts >= unit) e -= e % unit;
    if (e > edges->back() && e < total) edges->push_back((int)e);
  }
  edges->push_back(total);
}

int host_panels(const fmm_plan* plan, bool plain, int m, int n, int k, std::vector<int>* rows,
                std::vector<int>* cols) {
  int P = 1, R = 1;
  if ((long long)m * n >= kHostPanelMinElems) P = std::max(1, std::min(FMM_HOST_PANELS, n / kHostPanelMinCols));
  if (P > 1 && (long long)m * k >= kHostRowSplitMinA && m >= 2 * kHostRowPanelMinRows) R = 2;
  split_edges(m, R, 128 * ((plain || !plan) ? 1 : plan->dims[0]), rows);
  split_edges(n, P, 128 * ((plain || !plan) ? 1 : plan->dims[2]), cols);
  return (int)(rows->size() - 1) * (int)(cols->size() - 1);
}

// What a host call needs beside its buffers, kept for the next call: the two copy streams, the
// events that order blocks, and a pinned word for the device status.  A call takes one and
// gives it back; at most kHostLanes stay per device.
constexpr int kHostBlocks = 2 * FMM_HOST_PANELS;
constexpr size_t kHostLanes = 8;
struct HostLane {
  cudaStream_t in = nullptr, out = nullptr;
  cudaEvent_t ev[1 + 2 * kHostBlocks] = {};  // [0]: allocations made; [1 + b]: block b copied in; then: block b done
  unsigned* status = nullptr;
};
std::mutex g_lane_mu;
std::vector<HostLane*> g_lanes[kMaxDevices];

void lane_free(HostLane* l) {
  if (!l) return;
  for (auto e : l->ev)
    if (e) cudaEventDestroy(e);
  if (l->in) cudaStreamDestroy(l->in);
  if (l->out) cudaStreamDestroy(l->out);
  if (l->status) cudaFreeHost(l->status);
  delete l;
}

int lane_take(int dev, HostLane** out) {
  {
    std::lock_guard<std::mutex> lk(g_lane_mu);
    if (!g_lanes[dev].empty()) {
      *out = g_lanes[dev].back();
      g_lanes[dev].pop_back();
      return FMM_OK;
    }
  }
  HostLane* l = new (std::nothrow) HostLane();
  if (!l) return FMM_E_NOMEM;
  cudaError_t e = cudaStreamCreateWithFlags(&l->in, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&l->out, cudaStreamNonBlocking);
  for (auto& v : l->ev)
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&l->status, sizeof(unsigned));
  if (e != cudaSuccess) {
    lane_free(l);
    return cuda_status(e);
  }
  *out = l;
  return FMM_OK;
}

void lane_give(int dev, HostLane* l) {
  {
    std::lock_guard<std::mutex> lk(g_lane_mu);
    if (g_lanes[dev].size() < kHostLanes) {
      g_lanes[dev].push_back(l);
      return;
    }
  }
  lane_free(l);
}

// rows x cols doubles between column-major matrices; dense ones as one run (short columns
// otherwise cost the copy engine more than their bytes).
cudaError_t copy_matrix(double* dst, size_t ldd, const double* src, size_t lds, int rows, int cols, cudaMemcpyKind kind,
                        cudaStream_t st) {
  if ((ldd == (size_t)rows && lds == (size_t)rows) || cols == 1)
    return cudaMemcpyAsync(dst, src, sizeof(double) * (size_t)rows * cols, kind, st);
  return cudaMemcpy2DAsync(dst, sizeof(double) * ldd, src, sizeof(double) * lds, sizeof(double) * rows, cols, kind, st);
}

int run_host(const fmm_plan* plan, int pack, bool plain, int m, int n, int k, const double* A, int lda,
             const double* B, int ldb, double* C, int ldc) {
  int rc = check_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != FMM_OK) return rc;
  if (m == 0 || n == 0 || k == 0) return FMM_OK;
  if (!plain && !plan) return FMM_E_NOPLAN;
  int dev = 0;
  rc = configure_kernel(&dev);
  if (rc != FMM_OK) return rc;
  HostLane* lane = nullptr;
  rc = lane_take(dev, &lane);
  if (rc != FMM_OK) return rc;
  cudaStream_t st = cudaStreamPerThread;
  std::vector<int> re, ce;
  const int NB = host_panels(plan, plain, m, n, k, &re, &ce);
  const int R = (int)re.size() - 1;
  double *dA = nullptr, *dB = nullptr, *dC = nullptr;
  auto ok = [&](cudaError_t e) {
    if (rc == FMM_OK && e != cudaSuccess) rc = cuda_status(e);
    return rc == FMM_OK;
  };
  ok(cudaMallocAsync((void**)&dA, sizeof(double) * (size_t)m * k, st)) &&
      ok(cudaMallocAsync((void**)&dB, sizeof(double) * (size_t)k * n, st)) &&
      ok(cudaMallocAsync((void**)&dC, sizeof(double) * (size_t)m * n, st));
  cudaStream_t cin = NB > 1 ? lane->in : st, cout = NB > 1 ? lane->out : st;
  cudaEvent_t* ev = lane->ev;
  if (rc == FMM_OK && NB > 1) ok(cudaEventRecord(ev[0], st)) && ok(cudaStreamWaitEvent(cin, ev[0], 0));
  // block b = column panel b / R, row panel b % R
  for (int b = 0; b < NB && rc == FMM_OK; ++b) {
    const int i = b % R, j = b / R;
    const int r0 = re[i], mi = re[i + 1] - re[i], c0 = ce[j], nj = ce[j + 1] - ce[j];
    if (j == 0)  // A[I, :] at its first use
      ok(copy_matrix(dA + r0, m, A + r0, lda, mi, k, cudaMemcpyHostToDevice, cin));
    if (i == 0 && rc == FMM_OK)  // B[:, J] at its first use
      ok(copy_matrix(dB + (size_t)c0 * k, k, B + (size_t)c0 * ldb, ldb, k, nj, cudaMemcpyHostToDevice, cin));
    if (rc == FMM_OK)
      ok(copy_matrix(dC + r0 + (size_t)c0 * m, m, C + r0 + (size_t)c0 * ldc, ldc, mi, nj, cudaMemcpyHostToDevice, cin));
    if (NB > 1 && rc == FMM_OK) ok(cudaEventRecord(ev[1 + b], cin));
  }
  for (int b = 0; b < NB && rc == FMM_OK; ++b) {
    const int i = b % R, j = b / R;
    const int r0 = re[i], mi = re[i + 1] - re[i], c0 = ce[j], nj = ce[j + 1] - ce[j];
    if (NB > 1 && !ok(cudaStreamWaitEvent(st, ev[1 + b], 0))) break;
    double* Cb = dC + r0 + (size_t)c0 * m;
    rc = plain ? plain_gemm(mi, nj, k, dA + r0, m, dB + (size_t)c0 * k, k, Cb, m, st)
               : run_fmm(plan, pack, mi, nj, k, dA + r0, m, dB + (size_t)c0 * k, k, Cb, m, st);
    if (rc != FMM_OK) break;
    if (NB > 1) ok(cudaEventRecord(ev[1 + kHostBlocks + b], st)) && ok(cudaStreamWaitEvent(cout, ev[1 + kHostBlocks + b], 0));
    if (rc == FMM_OK)
      ok(copy_matrix(C + r0 + (size_t)c0 * ldc, ldc, Cb, m, mi, nj, cudaMemcpyDeviceToHost, cout));
  }
  *lane->status = 0;
  ok(cudaMemcpyAsync(lane->status, dev_status[dev], sizeof(unsigned), cudaMemcpyDeviceToHost, st));
  // join: every copy has finished before the buffers go back to the pool
  if (NB > 1) {
    ok(cudaStreamSynchronize(lane->in));
    ok(cudaStreamSynchronize(lane->out));
  }
  if (dA) cudaFreeAsync(dA, st);
  if (dB) cudaFreeAsync(dB, st);
  if (dC) cudaFreeAsync(dC, st);
  ok(cudaStreamSynchronize(st));
  if (rc == FMM_OK && (*lane->status != 0 || noalloc_used(dev))) rc = device_status(true);
  lane_give(dev, lane);
  return rc;
}

}  // namespace

extern "C" {

int fmm_plan_create(const int dims[3], int rank, const int* nterms, const int* rows, const int* cols,
                    const double* coefs, fmm_plan** out) {
  return build_plan(dims, rank, nterms, rows, cols, coefs, out);
}

int fmm_plan_destroy(fmm_plan* plan) {
  if (!plan) return FMM_E_INVALID;
  {
    std::lock_guard<std::mutex> lk(g_default_mu);
    if (g_default_plan == plan) g_default_plan = nullptr;
  }
  for (auto& d : plan->dev) {
    if (!d.ready) continue;
    cudaFree(d.prods);
    cudaFree(d.terms);
    cudaFree(d.cblk);
    cudaFree(d.ent_r);
    cudaFree(d.ent_w);
    cudaFree(d.cg_desc);
    cudaFree(d.cg_r);
    cudaFree(d.cg_m);
    cudaFree(d.cg_c);
    cudaFree(d.ch_r);
    cudaFree(d.ch_n);
    cudaFree(d.ch_op);
    cudaFree(d.prods_ps);
    cudaFree(d.terms_ps);
    cudaFree(d.plistA);
    cudaFree(d.plistB);
    cudaFree(d.prods_all);
    cudaFree(d.terms_all);
    cudaFree(d.plist_all);
    for (int side = 0; side < 2; ++side) {
      cudaFree(d.ps_first[side]);
      cudaFree(d.ps_terms[side]);
    }
  }
  for (auto& t : plan->ksplit) {
    cudaFree(t.prods);
    cudaFree(t.terms);
  }
  delete plan;
  return FMM_OK;
}

int fmm_plan_rank(const fmm_plan* plan) { return plan ? plan->rank : FMM_E_INVALID; }

int fmm_plan_combine_info(const fmm_plan* plan, int* groups, int* entries, int* chunks) {
  if (!plan) return FMM_E_INVALID;
  if (groups) *groups = plan->n_cgroup;
  if (entries) *entries = plan->n_cgroup ? (int)plan->cg_r.size() : 0;
  if (chunks) *chunks = plan->n_cgroup ? (int)plan->ch_n.size() : 0;
  return FMM_OK;
}

int fmm_bind_default_plan(fmm_plan* plan) {
  std::lock_guard<std::mutex> lk(g_default_mu);
  g_default_plan = plan;
  return FMM_OK;
}

fmm_plan* fmm_default_plan(void) {
  std::lock_guard<std::mutex> lk(g_default_mu);
  return g_default_plan;
}

int fmm_dgemm_dev(const fmm_plan* plan, int pack_type, int m, int n, int k, const double* A, long lda,
                  const double* B, long ldb, double* C, long ldc, void* stream) {
  return run_fmm(plan, pack_type, m, n, k, A, lda, B, ldb, C, ldc, static_cast<cudaStream_t>(stream));
}

int fmm_plain_dgemm_dev(int m, int n, int k, const double* A, long lda, const double* B, long ldb, double* C,
                        long ldc, void* stream) {
  int rc = check_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != FMM_OK || m == 0 || n == 0 || k == 0) return rc;
  return plain_gemm(m, n, k, A, lda, B, ldb, C, ldc, static_cast<cudaStream_t>(stream));
}

int fmm_dgemm_host(const fmm_plan* plan, int pack_type, int m, int n, int k, const double* A, int lda,
                   const double* B, int ldb, double* C, int ldc) {
  return run_host(plan, pack_type, false, m, n, k, A, lda, B, ldb, C, ldc);
}

void bl_dgemm(int m, int n, int k, double* A, int lda, double* B, int ldb, double* C, int ldc) {
  t_last_error = run_host(nullptr, 0, true, m, n, k, A, lda, B, ldb, C, ldc);
}

void bl_dgemm_strassen_abc(int m, int n, int k, double* A, int lda, double* B, int ldb, double* C, int ldc) {
  t_last_error = run_host(fmm_default_plan(), FMM_PACK_ABC, false, m, n, k, A, lda, B, ldb, C, ldc);
}

void bl_dgemm_strassen_ab(int m, int n, int k, double* A, int lda, double* B, int ldb, double* C, int ldc) {
  t_last_error = run_host(fmm_default_plan(), FMM_PACK_AB, false, m, n, k, A, lda, B, ldb, C, ldc);
}

void bl_dgemm_strassen_naive(int m, int n, int k, double* A, int lda, double* B, int ldb, double* C, int ldc) {
  t_last_error = run_host(fmm_default_plan(), FMM_PACK_NAIVE, false, m, n, k, A, lda, B, ldb, C, ldc);
}

void bl_dynamic_peeling(int m, int n, int k, double* A, int lda, double* B, int ldb, double* C, int ldc, int dim1,
                        int dim2, int dim3) {
  if (dim1 <= 0 || dim2 <= 0 || dim3 <= 0) {
    t_last_error = FMM_E_INVALID;
    return;
  }
  int rc = check_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != FMM_OK || m == 0 || n == 0 || k == 0) {
    t_last_error = rc;
    return;
  }
  cudaStream_t st = cudaStreamPerThread;
  double *dA = nullptr, *dB = nullptr, *dC = nullptr;
  const int pa = m + (m & 1), pb = k + (k & 1);  // even device pitches (16-byte column starts)
  const size_t szA = sizeof(double) * (size_t)pa * k, szB = sizeof(double) * (size_t)pb * n,
               szC = sizeof(double) * (size_t)m * n;
  rc = cuda_status(cudaMallocAsync((void**)&dA, szA, st));
  if (rc == FMM_OK) rc = cuda_status(cudaMallocAsync((void**)&dB, szB, st));
  if (rc == FMM_OK) rc = cuda_status(cudaMallocAsync((void**)&dC, szC, st));
  if (rc == FMM_OK)
    rc = cuda_status(cudaMemcpy2DAsync(dA, sizeof(double) * pa, A, sizeof(double) * lda, sizeof(double) * m, k,
                                       cudaMemcpyHostToDevice, st));
  if (rc == FMM_OK)
    rc = cuda_status(cudaMemcpy2DAsync(dB, sizeof(double) * pb, B, sizeof(double) * ldb, sizeof(double) * k, n,
                                       cudaMemcpyHostToDevice, st));
  if (rc == FMM_OK)
    rc = cuda_status(cudaMemcpy2DAsync(dC, sizeof(double) * m, C, sizeof(double) * ldc, sizeof(double) * m, n,
                                       cudaMemcpyHostToDevice, st));
  if (rc == FMM_OK) rc = peel(m, n, k, dA, pa, dB, pb, dC, m, dim1, dim2, dim3, st);
  if (rc == FMM_OK)
    rc = cuda_status(cudaMemcpy2DAsync(C, sizeof(double) * ldc, dC, sizeof(double) * m, sizeof(double) * m, n,
                                       cudaMemcpyDeviceToHost, st));
  if (dA) cudaFreeAsync(dA, st);
  if (dB) cudaFreeAsync(dB, st);
  if (dC) cudaFreeAsync(dC, st);
  cudaError_t se = cudaStreamSynchronize(st);
  if (rc == FMM_OK) rc = cuda_status(se);
  if (rc == FMM_OK) rc = device_status(true);
  t_last_error = rc;
}

int fmm_last_error(void) { return t_last_error; }

const char* fmm_error_string(int code) {
  switch (code) {
    case FMM_OK: return "ok";
    case FMM_E_INVALID: return "invalid argument (dimension, leading dimension or pointer)";
    case FMM_E_NOPLAN: return "no FMM plan bound";
    case FMM_E_CUDA: return "CUDA runtime error";
    case FMM_E_NOMEM: return "out of memory";
    case FMM_E_PLAN: return "malformed plan tables";
    case FMM_E_UNSUPPORTED: return "unsupported pack type or option";
    case FMM_E_TIMEOUT: return "device-side wait timed out";
    case FMM_E_TOO_LARGE: return "problem exceeds the no-allocation scratch limits";
    default: return "unknown error";
  }
}

long long fmm_kernel_launch_count(void) { return g_launches.load(); }

int fmm_device_status(int clear) { return device_status(clear != 0); }

long long fmm_set_workspace_limit(long long bytes) {
  return g_ws_limit.exchange(bytes > 0 ? bytes : kDefaultWorkspaceLimit);
}

long long fmm_last_workspace_bytes(void) { return t_last_ws; }

int fmm_debug_set(int what, long long value) {
  switch (what) {
    case FMM_DEBUG_WAIT_LIMIT_NS: {
      const unsigned long long v = value > 0 ? (unsigned long long)value : fmm::WAIT_LIMIT_NS;
      FMM_CUDA_TRY(cudaMemcpyToSymbol(fmm::g_wait_limit_ns, &v, sizeof(v)));
      return FMM_OK;
    }
    case FMM_DEBUG_TICKET_FILL:
      if (value < 0 || value > 255) return FMM_E_INVALID;
      g_ticket_fill = (int)value;
      return FMM_OK;
    case FMM_DEBUG_SPLIT_OPERANDS:
      if (value < 0 || value > 1) return FMM_E_INVALID;
      g_split_form = (int)value;
      return FMM_OK;
    case FMM_DEBUG_KSPLIT:
      if (value < 0 || value > 8) return FMM_E_INVALID;
      g_force_ksplit = (int)value;
      return FMM_OK;
    case FMM_DEBUG_COMBINE_POSITIONS:
      if (value < 0 || value > 2) return FMM_E_INVALID;
      g_combine_positions = (int)value;
      return FMM_OK;
    default:
      return FMM_E_INVALID;
  }
}

int fmm_profile_begin(void) {
  std::lock_guard<std::mutex> lk(g_prof_mu);
  for (auto& r : g_prof) {
    cudaEventDestroy(r.e0);
    cudaEventDestroy(r.e1);
  }
  g_prof.clear();
  g_prof_on = true;
  return FMM_OK;
}

int fmm_profile_end(double* ms_out, long long* count_out) {
  std::vector<ProfRec> recs;
  {
    std::lock_guard<std::mutex> lk(g_prof_mu);
    g_prof_on = false;
    recs.swap(g_prof);
  }
  for (int k = 0; k < K_NUM; ++k) {
    if (ms_out) ms_out[k] = 0.0;
    if (count_out) count_out[k] = 0;
  }
  int rc = FMM_OK;
  for (auto& r : recs) {
    float ms = 0.f;
    cudaError_t e = cudaEventSynchronize(r.e1);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, r.e0, r.e1);
    if (e != cudaSuccess) rc = cuda_status(e);
    if (ms_out) ms_out[r.kind] += ms;
    if (count_out) count_out[r.kind] += 1;
    cudaEventDestroy(r.e0);
    cudaEventDestroy(r.e1);
  }
  return rc;
}

int fmm_profile_num_kinds(void) { return K_NUM; }

const char* fmm_profile_kind_name(int kind) { return (kind >= 0 && kind < K_NUM) ? kKernelNames[kind] : ""; }

}  // extern "C"

// ------------------------------------------------------------------------------------
// No-allocation entry point.
//
// Some callers cannot allocate device memory when they call us: frameworks that own the
// whole device memory through their own arena or caching allocator and forbid foreign
// cudaMalloc calls (an allocation behind their back can fail or fragment their pool),
// and code on latency-critical paths where an allocation (or the synchronisation a
// cudaFree implies) is not acceptable.  fmm_dgemm_dev_noalloc() serves them: it runs the
// ABC FMM with the operand sums folded during staging (no pre-summed workspace), and
// keeps the only scratch the kernel needs -- per-tile tickets, a work-unit counter, the status word --
// and the plan tables in one statically allocated device array.
// ------------------------------------------------------------------------------------
namespace {

constexpr int kNoAllocMaxTiles = 16384;   // tile positions (128 x 128) of one call
constexpr int kNoAllocMaxProds = 1024;    // products of a plan
constexpr int kNoAllocMaxTerms = 12288;   // A, B and C terms of a plan
constexpr size_t kNoAllocTicketsOff = 0;
constexpr size_t kNoAllocStatusOff = kNoAllocTicketsOff + sizeof(int) * kNoAllocMaxTiles;
constexpr size_t kNoAllocCounterOff = kNoAllocStatusOff + 128;  // a launch's work-unit counter
constexpr size_t kNoAllocProdsOff = kNoAllocStatusOff + 256;
constexpr size_t kNoAllocTermsOff = kNoAllocProdsOff + sizeof(fmm::Prod) * (kNoAllocMaxProds + 1);
constexpr size_t kNoAllocBytes = kNoAllocTermsOff + sizeof(fmm::Term) * (kNoAllocMaxTerms + 3);

}  // namespace

// Every GPU that loads this library holds this array (about 384 KB) until the process exits.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

namespace {

std::mutex g_noalloc_mu;
unsigned char* g_noalloc_ptr[kMaxDevices];  // device address of g_noalloc_scratch, per device
bool g_noalloc_ready[kMaxDevices];

// Once per device, with that device current: resolve the array's device address (in host
// code the symbol is only a host-side stand-in) and configure the kernels.  Nothing here
// allocates device memory.
int noalloc_setup(int dev) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (g_noalloc_ready[dev]) return FMM_OK;
  void* p = nullptr;
  FMM_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  if (p == nullptr) return FMM_E_CUDA;
  FMM_CUDA_TRY(cudaFuncSetAttribute(fmm::fmm_gemm_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)fmm::smem_bytes(false)));
  FMM_CUDA_TRY(cudaFuncSetAttribute(fmm::fmm_gemm_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)fmm::smem_bytes(true)));
  int nsm = 0;
  FMM_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  {
    std::lock_guard<std::mutex> lk2(g_attr_mu);
    if (sm_count[dev] == 0) sm_count[dev] = nsm;
    if (!g_encode_tiled) {
      cudaDriverEntryPointQueryResult q;
      void* fn = nullptr;
      if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
          q == cudaDriverEntryPointSuccess)
        g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
  }
  // The classical product used by the fringe strips never changes: its tables (product
  // index kNoAllocMaxProds, terms after the plan's) are written here once, and the status
  // word starts at zero.  Both copies are blocking, from memory that outlives them.
  static const fmm::Prod classic{kNoAllocMaxTerms, 1, kNoAllocMaxTerms + 1, 1, kNoAllocMaxTerms + 2, 1};
  static const fmm::Term classic_terms[3] = {{0, 0, 1.0, 0, 0}, {0, 0, 1.0, 0, 0}, {0, 0, 1.0, 0, 0}};
  unsigned char* base = static_cast<unsigned char*>(p);
  FMM_CUDA_TRY(cudaMemcpy(base + kNoAllocProdsOff + sizeof(fmm::Prod) * kNoAllocMaxProds, &classic, sizeof(classic),
                          cudaMemcpyHostToDevice));
  FMM_CUDA_TRY(cudaMemcpy(base + kNoAllocTermsOff + sizeof(fmm::Term) * kNoAllocMaxTerms, classic_terms,
                          sizeof(classic_terms), cudaMemcpyHostToDevice));
  FMM_CUDA_TRY(cudaMemset(base + kNoAllocStatusOff, 0, sizeof(unsigned)));
  g_noalloc_ptr[dev] = base;
  g_noalloc_ready[dev] = true;
  return FMM_OK;
}

bool noalloc_used(int dev) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  return g_noalloc_ready[dev];
}

int noalloc_status(int dev, bool clear) {
  unsigned char* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ready[dev]) return FMM_OK;
    base = g_noalloc_ptr[dev];
  }
  unsigned v = 0;
  FMM_CUDA_TRY(cudaMemcpy(&v, base + kNoAllocStatusOff, sizeof(unsigned), cudaMemcpyDeviceToHost));
  if (clear && v) FMM_CUDA_TRY(cudaMemset(base + kNoAllocStatusOff, 0, sizeof(unsigned)));
  return v ? FMM_E_TIMEOUT : FMM_OK;
}

// One launch of fmm_gemm_kernel in MODE_ACCUM_C with caller-provided tables, tickets and
// status word (nothing allocated).
int noalloc_launch(const fmm::Prod* prods, const fmm::Term* terms, const int grid_dims[3], int nprod,
                   const double* A, long long lda, const double* B, long long ldb, double* C, long long ldc,
                   int ms, int ns, int ks, int* tickets, unsigned* status, int* counter, int nsm, cudaStream_t st) {
  if (ms <= 0 || ns <= 0 || ks <= 0 || nprod <= 0) return FMM_OK;
  fmm::GemmArgs a{};
  a.A = A;
  a.lda = lda;
  a.B = B;
  a.ldb = ldb;
  a.C = C;
  a.ldc = ldc;
  a.ms = ms;
  a.ns = ns;
  a.ks = ks;
  a.prods = prods;
  a.terms = terms;
  a.nprod = nprod;
  a.tiles_m = (ms + fmm::BM - 1) / fmm::BM;
  a.tiles_n = (ns + fmm::BN - 1) / fmm::BN;
  a.status = status;
  const int ntiles = a.tiles_m * a.tiles_n;
  a.tickets = tickets;
  if (nprod > 1 && ntiles > kNoAllocMaxTiles) return FMM_E_TOO_LARGE;  // tickets of one launch must fit
  if (nprod > 1) FMM_CUDA_TRY(cudaMemsetAsync(tickets, 0, sizeof(int) * ntiles, st));
  a.counter = counter;
  FMM_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(int), st));
  const long long units = (long long)ntiles * nprod;
  const unsigned grid = (unsigned)(units < nsm ? units : nsm);
  const long long am = (long long)grid_dims[0] * ms, ak = (long long)grid_dims[1] * ks,
                  bn = (long long)grid_dims[2] * ns;
  const bool tma = make_tensor_map(&a.tmA, A, am, ak, lda, fmm::BM, fmm::BK) &&
                   make_tensor_map(&a.tmB, B, ak, bn, ldb, fmm::BK, fmm::BN) &&
                   make_tensor_map(&a.tmB2, B, ak, bn, ldb, fmm::TB_K, fmm::BN);
  if (tma)
    fmm::fmm_gemm_kernel<true><<<grid, fmm::NTHREADS, fmm::smem_bytes(true), st>>>(a);
  else
    fmm::fmm_gemm_kernel<false><<<grid, fmm::NTHREADS, fmm::smem_bytes(false), st>>>(a);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return cuda_status(cudaGetLastError());
}

}  // namespace

extern "C" int fmm_dgemm_dev_noalloc(const fmm_plan* plan, int m, int n, int k, const double* A, long lda,
                                     const double* B, long ldb, double* C, long ldc, void* stream, int sync) {
  if (!plan) return FMM_E_NOPLAN;
  int rc = check_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != FMM_OK) return rc;
  if (m == 0 || n == 0 || k == 0) return FMM_OK;
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return FMM_E_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // size limits of the static scratch
  const int pm = plan->dims[0] * kMR, pk = plan->dims[1], pn = plan->dims[2] * kNR;
  const int md = m - m % pm, kd = k - k % pk, nd = n - n % pn;
  const int ms = md / plan->dims[0], ks = kd / plan->dims[1], ns = nd / plan->dims[2];
  const long long tiles_fmm = (long long)((ms + fmm::BM - 1) / fmm::BM) * ((ns + fmm::BN - 1) / fmm::BN);
  if ((int)plan->prods.size() > kNoAllocMaxProds || (int)plan->terms.size() > kNoAllocMaxTerms ||
      tiles_fmm > kNoAllocMaxTiles)
    return FMM_E_TOO_LARGE;
  rc = noalloc_setup(dev);
  if (rc != FMM_OK) return rc;
  unsigned char* base = g_noalloc_ptr[dev];
  int* tickets = reinterpret_cast<int*>(base + kNoAllocTicketsOff);
  unsigned* status = reinterpret_cast<unsigned*>(base + kNoAllocStatusOff);
  int* counter = reinterpret_cast<int*>(base + kNoAllocCounterOff);
  fmm::Prod* prods = reinterpret_cast<fmm::Prod*>(base + kNoAllocProdsOff);
  fmm::Term* terms = reinterpret_cast<fmm::Term*>(base + kNoAllocTermsOff);
  // the plan's tables (from the plan's own storage, which outlives the copy); the classical
  // product of the fringe strips was written at set-up
  FMM_CUDA_TRY(cudaMemcpyAsync(prods, plan->prods.data(), sizeof(fmm::Prod) * plan->prods.size(),
                               cudaMemcpyHostToDevice, st));
  FMM_CUDA_TRY(cudaMemcpyAsync(terms, plan->terms.data(), sizeof(fmm::Term) * plan->terms.size(),
                               cudaMemcpyHostToDevice, st));
  const int nsm = sm_count[dev] > 0 ? sm_count[dev] : 148;
  rc = noalloc_launch(prods, terms, plan->dims, plan->rank, A, lda, B, ldb, C, ldc, ms, ns, ks, tickets, status,
                      counter, nsm, st);
  // fringe GEMMs (same regions and order as the reference's dynamic peeling)
  const int mr = m - md, kr = k - kd, nr = n - nd;
  const fmm::Prod* cp = prods + kNoAllocMaxProds;
  if (rc == FMM_OK && kr > 0 && md > 0 && nd > 0)
    rc = noalloc_launch(cp, terms, kUnitGrid, 1, A + (long long)kd * lda, lda, B + kd, ldb, C, ldc, md, nd, kr,
                        tickets, status, counter, nsm, st);
  if (rc == FMM_OK && nr > 0)
    rc = noalloc_launch(cp, terms, kUnitGrid, 1, A, lda, B + (long long)nd * ldb, ldb, C + (long long)nd * ldc, ldc, m,
                        nr, k, tickets, status, counter, nsm, st);
  if (rc == FMM_OK && mr > 0 && nd > 0)
    rc = noalloc_launch(cp, terms, kUnitGrid, 1, A + md, lda, B, ldb, C + md, ldc, mr, nd, k, tickets, status,
                        counter, nsm, st);
  // The status word is not cleared per call: a timeout recorded by a sync = 0 call stays
  // until a sync = 1 call or fmm_device_status() reports (and clears) it.
  if (rc == FMM_OK && sync) {
    unsigned v = 0;
    FMM_CUDA_TRY(cudaMemcpyAsync(&v, status, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    if (v) {
      FMM_CUDA_TRY(cudaMemsetAsync(status, 0, sizeof(unsigned), st));
      FMM_CUDA_TRY(cudaStreamSynchronize(st));
      rc = FMM_E_TIMEOUT;
    }
  }
  return rc;
}

// ---------------------------------------------------------------------------------------
// Split-BF16 FMM (tcgen05 tensor cores): FP32 A and B, FP64 C.  Same partition, product
// order and fringe peeling as the FP64 path; every GEMM (FMM core and fringe strips) runs
// as bf16 plane products with FP64 accumulation across 64-deep k chunks.
// ---------------------------------------------------------------------------------------
namespace {

bool split_configured[kMaxDevices];
constexpr int kPlaneSmem = 200 * 1024;

int split_configure(int* dev_out) {
  int rc = configure_kernel(dev_out);
  if (rc != FMM_OK) return rc;
  std::lock_guard<std::mutex> lk(g_attr_mu);
  if (!split_configured[*dev_out]) {
    FMM_CUDA_TRY(cudaFuncSetAttribute(fmms::fmm_split_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)fmms::SMEM_BYTES));
    for (auto kernel : {fmms::fmm_split_planes_kernel<16, 2>, fmms::fmm_split_planes_kernel<16, 1>,
                        fmms::fmm_split_planes_kernel<8, 1>})
      FMM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPlaneSmem));
    split_configured[*dev_out] = true;
  }
  return g_encode_tiled ? FMM_OK : FMM_E_UNSUPPORTED;
}

// bf16 planes (rows x kpad, row-major, pitch kpad) as a tensor map with box 64 x 128 and
// the 128-byte swizzle the UMMA descriptors expect.
bool make_plane_map(CUtensorMap* map, const __nv_bfloat16* base, long long rows, long long kpad) {
  if (rows <= 0 || rows >= (1LL << 32) || kpad % fmms::KPAD != 0) return false;
  cuuint64_t dims[2] = {(cuuint64_t)kpad, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)kpad * sizeof(__nv_bfloat16)};
  cuuint32_t box[2] = {(cuuint32_t)fmms::BK, (cuuint32_t)fmms::BM};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims,
                              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// One GEMM of a split-BF16 call: sub-blocks ms x ks x ns of a plan (the classical plan: a fringe
// strip or the whole problem).
struct SplitPart {
  const fmm_plan* plan;
  const float* A;
  const float* B;
  double* C;
  int ms, ns, ks;
  // workspace of its planes, tickets (ints from the counter on) and stored products
  size_t off_a = 0, off_b = 0, off_m = 0;
  long long ticket = 0;
  long long kpad = 0;
  int parts = 1, part_stages = 0;
  bool use_m = false;
  bool planes_done = false;
};

// k parts of a single product: rounds of the SMs times chunks per unit (4.6 us each) against the
// parts' C updates, which follow one another (kPartUpdateUs each).  Measured us with 1 / as many
// parts as chunks: 512 x 512 x 2048 50 / 75, 512 x 512 x 8192 156 / 92, 258^3 21 / 29.
constexpr double kChunkUs = 4.6, kPartUpdateUs = 6.0;
void split_parts(SplitPart* p, int nsm) {
  const int nks = (int)(p->kpad / fmms::BK);
  const int chunks = (nks + fmms::DRAIN_STAGES - 1) / fmms::DRAIN_STAGES;
  const long long tiles = tiles_of(p->ms, p->ns, fmms::BM);
  int best = 1;
  double cost = 1e300;
  for (int s = 1; s <= std::min(chunks, 16); ++s) {
    const double c = (double)((tiles * s + nsm - 1) / nsm) * ((chunks + s - 1) / s) * kChunkUs + s * kPartUpdateUs;
    if (c < 0.97 * cost) {
      best = s;
      cost = c;
    }
  }
  p->part_stages = (chunks + best - 1) / best * fmms::DRAIN_STAGES;
  p->parts = (nks + p->part_stages - 1) / p->part_stages;
}

// The tile of a planes CTA by the operand's blocks: 16 rows x 64 k for few blocks (and several
// k tiles per CTA, so that a thread has at least 16 loads in flight), x 32 k beyond, 8 rows for
// more than 16.
struct PlaneTile {
  int tr, np, kts;
};
PlaneTile plane_tile(int maxblk, int nblk) {
  if (maxblk <= 4) return PlaneTile{16, 2, std::max(1, 4 / nblk)};
  return PlaneTile{maxblk <= 16 ? 16 : 8, 1, std::max(1, 8 / nblk)};
}

// The operand planes of several GEMMs (fmm_split_planes_kernel); zero[0 .. nzero) is cleared.
int launch_planes(SplitPart* ps, int np, char* ws, long long lda, long long ldb, int* zero, long long nzero,
                  cudaStream_t st) {
  fmms::PlaneArgs g{};
  int maxblk = 1;
  for (int q = 0; q < np; ++q)
    if (!ps[q].planes_done)
      maxblk = std::max({maxblk, ps[q].plan->dims[0] * ps[q].plan->dims[1], ps[q].plan->dims[1] * ps[q].plan->dims[2]});
  const int tr = plane_tile(maxblk, 1).tr, np2 = plane_tile(maxblk, 1).np;
  long long ctas = 0;
  size_t smem = 0;
  for (int q = 0; q < np; ++q) {
    SplitPart& p = ps[q];
    if (p.planes_done) continue;
    DevTables* d = nullptr;
    const int rc = device_tables(p.plan, &d);
    if (rc != FMM_OK) return rc;
    for (int side = 0; side < 2; ++side) {
      fmms::PlaneJob& j = g.job[g.njob++];
      j.X = side == 0 ? p.A : p.B;
      j.ldx = side == 0 ? lda : ldb;
      j.out = reinterpret_cast<__nv_bfloat16*>(ws + (side == 0 ? p.off_a : p.off_b));
      j.first = d->ps_first[side];
      j.terms = d->ps_terms[side];
      j.rows = side == 0 ? p.ms : p.ns;
      j.ks = p.ks;
      j.kpad = (int)p.kpad;
      j.blk_row_stride = side == 0 ? p.ms : p.ks;
      j.blk_col_stride = side == 0 ? p.ks : p.ns;
      j.nblk = side == 0 ? p.plan->dims[0] * p.plan->dims[1] : p.plan->dims[1] * p.plan->dims[2];
      j.block_cols = side == 0 ? p.plan->dims[1] : p.plan->dims[2];
      j.nprod = p.plan->rank;
      j.nterm = (int)p.plan->ps_terms[side].size();
      j.side = side;
      j.kt = (int)(p.kpad / (32 * np2));
      j.kts = plane_tile(maxblk, j.nblk).kts;
      j.cta0 = (int)ctas;
      ctas += (long long)((j.rows + tr - 1) / tr) * ((j.kt + j.kts - 1) / j.kts);
      smem = std::max(smem, fmms::plane_smem_bytes(tr, np2, j.nblk, j.kts, j.nprod, j.nterm));
    }
  }
  if (ctas > INT32_MAX || nzero > INT32_MAX) return FMM_E_UNSUPPORTED;
  if (g.njob == 0) return cuda_status(cudaMemsetAsync(zero, 0, sizeof(int) * nzero, st));
  g.zero = zero;
  g.nzero = (int)nzero;
  ProfScope pf(K_SPLIT_OPERANDS, st);
  return launch_dependent(np2 == 2   ? fmms::fmm_split_planes_kernel<16, 2>
                          : tr == 16 ? fmms::fmm_split_planes_kernel<16, 1>
                                     : fmms::fmm_split_planes_kernel<8, 1>,
                          dim3((unsigned)ctas), 16 * tr, smem, st, 1, g);
}

// A core whose staged tiles do not fit (or the test hook): one product per CTA.
int launch_operands(const SplitPart& p, char* ws, long long lda, long long ldb, cudaStream_t st) {
  DevTables* d = nullptr;
  const int rc = device_tables(p.plan, &d);
  if (rc != FMM_OK) return rc;
  for (int side = 0; side < 2; ++side) {
    fmms::SplitArgs a{};
    a.X = side == 0 ? p.A : p.B;
    a.ldx = side == 0 ? lda : ldb;
    a.rows = side == 0 ? p.ms : p.ns;
    a.ks = p.ks;
    a.kpad = (int)p.kpad;
    a.blk_row_stride = side == 0 ? p.ms : p.ks;
    a.blk_col_stride = side == 0 ? p.ks : p.ns;
    a.out = reinterpret_cast<__nv_bfloat16*>(ws + (side == 0 ? p.off_a : p.off_b));
    a.prods = d->prods;
    a.terms = d->terms;
    a.side = side;
    ProfScope pf(K_SPLIT_OPERANDS, st);
    fmms::fmm_split_operands_kernel<<<dim3((unsigned)p.plan->rank, (unsigned)(p.kpad / fmms::SPLIT_K),
                                           (unsigned)((a.rows + fmms::SPLIT_ROWS - 1) / fmms::SPLIT_ROWS)),
                                      dim3(32, 8), 0, st>>>(a);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    FMM_CUDA_TRY(cudaGetLastError());
  }
  return FMM_OK;
}

// The GEMMs [p0, p1) in one launch; `counter` is the launch's own.
int launch_split_gemm(const SplitPart* ps, int p0, int p1, char* ws, long long ldc, int* counter, int* tickets, int dev,
                      cudaStream_t st) {
  fmms::SplitGemmArgs g{};
  long long units = 0;
  for (int q = p1 - 1; q >= p0; --q) {  // the strips' long units first
    const SplitPart& p = ps[q];
    DevTables* d = nullptr;
    const int rc = device_tables(p.plan, &d);
    if (rc != FMM_OK) return rc;
    fmms::SplitJob& j = g.job[g.njob++];
    const int R = p.plan->rank;
    if (!make_plane_map(&j.tmA, reinterpret_cast<const __nv_bfloat16*>(ws + p.off_a), 3LL * R * p.ms, p.kpad) ||
        !make_plane_map(&j.tmB, reinterpret_cast<const __nv_bfloat16*>(ws + p.off_b), 3LL * R * p.ns, p.kpad))
      return FMM_E_UNSUPPORTED;
    j.C = p.C;
    j.ldc = ldc;
    j.prods = d->prods;
    j.terms = d->terms;
    j.tickets = tickets + p.ticket;
    j.M = p.use_m ? reinterpret_cast<double*>(ws + p.off_m) : nullptr;
    j.m_stride = (long long)p.ms * p.ns;
    j.ms = p.ms;
    j.ns = p.ns;
    j.nks = (int)(p.kpad / fmms::BK);
    j.nprod = R;
    j.parts = p.parts;
    j.part_stages = p.part_stages;
    j.tiles_m = (p.ms + fmms::BM - 1) / fmms::BM;
    j.tiles_n = (p.ns + fmms::BN - 1) / fmms::BN;
    j.first = (int)units;
    units += (long long)j.tiles_m * j.tiles_n * (p.parts > 1 ? p.parts : R);
    if (units > INT32_MAX) return FMM_E_UNSUPPORTED;
  }
  g.units = (int)units;
  g.status = dev_status[dev];
  g.counter = counter;
  const unsigned grid = (unsigned)std::min<long long>(units, sm_count[dev]);
  ProfScope pf(K_GEMM_SPLIT, st);
  return launch_dependent(fmms::fmm_split_gemm_kernel, dim3(grid), fmms::NTHREADS, fmms::SMEM_BYTES, st, 1, g);
}

// Same partition as the FP64 path: the FMM core, then the fringe strips (classical).  The n
// and m strips lie outside the core's C and run in its launch; the k strip updates the core's
// C and follows the combine pass.
int run_split(const fmm_plan* plan, int m, int n, int k, const float* A, long long lda, const float* B,
              long long ldb, double* C, long long ldc, cudaStream_t st) {
  int rc = check_args(m, n, k, A, lda, B, ldb, C, ldc);
  if (rc != FMM_OK || m == 0 || n == 0 || k == 0) return rc;
  const fmm_plan* cls = classical_plan();
  if (!plan || is_classical(plan)) plan = cls;
  int dev = 0;
  rc = split_configure(&dev);
  if (rc != FMM_OK) return rc;
  static_assert(fmms::BM == fmms::BN, "one box shape for both plane maps");
  SplitPart ps[4];
  int np = 0;
  auto add = [&](const fmm_plan* p, const float* a, const float* b, double* c, int ms, int ns, int ks) {
    if (ms <= 0 || ns <= 0 || ks <= 0) return;
    ps[np] = SplitPart{};
    ps[np].plan = p;
    ps[np].A = a;
    ps[np].B = b;
    ps[np].C = c;
    ps[np].ms = ms;
    ps[np].ns = ns;
    ps[np].ks = ks;
    ++np;
  };
  int last = 0;  // the k strip's index when it needs a launch of its own
  if (plan == cls) {
    add(cls, A, B, C, m, n, k);
    last = np;
  } else {
    const int pm = plan->dims[0] * kMR, pk = plan->dims[1], pn = plan->dims[2] * kNR;
    const int md = m - m % pm, kd = k - k % pk, nd = n - n % pn;
    const bool core = md > 0 && nd > 0 && kd > 0;
    if (core) add(plan, A, B, C, md / plan->dims[0], nd / plan->dims[2], kd / plan->dims[1]);
    add(cls, A, B + (long long)nd * ldb, C + (long long)nd * ldc, m, n - nd, k);
    add(cls, A + md, B, C + md, m - md, nd, k);
    last = np;
    add(cls, A + (long long)kd * lda, B + kd, C, md, nd, k - kd);
    if (!core) last = np;  // no core: the three strips are disjoint
  }
  // workspace: planes, stored products, the launches' counters (2) and the tickets
  size_t bytes = 0;
  long long tickets = 0;
  auto take = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) & ~(size_t)255;
    return at;
  };
  for (int q = 0; q < np; ++q) {
    SplitPart& p = ps[q];
    const int R = p.plan->rank;
    p.kpad = ((long long)p.ks + fmms::KPAD - 1) / fmms::KPAD * fmms::KPAD;
    const long long tiles = tiles_of(p.ms, p.ns, fmms::BM);
    if (tiles * R > INT32_MAX || (p.ms + fmms::SPLIT_ROWS - 1) / fmms::SPLIT_ROWS > 65535 ||
        (p.ns + fmms::SPLIT_ROWS - 1) / fmms::SPLIT_ROWS > 65535 || p.kpad / fmms::SPLIT_K > 65535)
      return FMM_E_UNSUPPORTED;
    // several products: store each M_r, then one combine pass applies W (no C loads in the
    // tensor-core kernel's epilogue); a single product goes straight into C
    p.use_m = R > 1 && combine_fits(p.plan);
    p.part_stages = (int)(p.kpad / fmms::BK);
    if (R == 1) split_parts(&p, sm_count[dev]);
    p.off_a = take(sizeof(__nv_bfloat16) * 3 * (size_t)R * p.ms * p.kpad);
    p.off_b = take(sizeof(__nv_bfloat16) * 3 * (size_t)R * p.ns * p.kpad);
    if (p.use_m) p.off_m = take(sizeof(double) * (size_t)R * p.ms * p.ns);
    p.ticket = tickets;
    if (!p.use_m && (R > 1 || p.parts > 1)) tickets += tiles * (fmms::NEPI / 32);
  }
  const size_t off_c = take(sizeof(int) * (2 + (size_t)tickets));
  char* ws = nullptr;
  FMM_CUDA_TRY(cudaMallocAsync((void**)&ws, bytes, st));
  int* counter = reinterpret_cast<int*>(ws + off_c);
  for (int q = 0; q < np && rc == FMM_OK; ++q) {  // cores whose staged tiles do not fit
    SplitPart& p = ps[q];
    const int na = p.plan->dims[0] * p.plan->dims[1], nb = p.plan->dims[1] * p.plan->dims[2];
    const PlaneTile t = plane_tile(std::max(na, nb), std::max(na, nb));
    const bool fits =
        fmms::plane_smem_bytes(t.tr, t.np, na, t.kts, p.plan->rank, (int)p.plan->ps_terms[0].size()) <= kPlaneSmem &&
        fmms::plane_smem_bytes(t.tr, t.np, nb, t.kts, p.plan->rank, (int)p.plan->ps_terms[1].size()) <= kPlaneSmem;
    if (fits && (g_split_form.load() == 0 || p.plan->rank == 1)) continue;
    rc = launch_operands(p, ws, lda, ldb, st);
    p.planes_done = true;
  }
  if (rc == FMM_OK) rc = launch_planes(ps, np, ws, lda, ldb, counter, 2 + tickets, st);
  if (rc == FMM_OK && last > 0) rc = launch_split_gemm(ps, 0, last, ws, ldc, counter, counter + 2, dev, st);
  if (rc == FMM_OK && ps[0].use_m) {
    DevTables* d = nullptr;
    rc = device_tables(ps[0].plan, &d);
    if (rc == FMM_OK)
      rc = launch_combine(ps[0].plan, *d, ps[0].C, ldc, ps[0].ms, ps[0].ns, reinterpret_cast<double*>(ws + ps[0].off_m),
                          ps[0].ms, (long long)ps[0].ms * ps[0].ns, st);
  }
  if (rc == FMM_OK && last < np) rc = launch_split_gemm(ps, last, np, ws, ldc, counter + 1, counter + 2, dev, st);
  cudaError_t fe = cudaFreeAsync(ws, st);
  return rc == FMM_OK ? cuda_status(fe) : rc;
}

}  // namespace

extern "C" int fmm_split_gemm_dev(const fmm_plan* plan, int m, int n, int k, const float* A, long lda,
                                  const float* B, long ldb, double* C, long ldc, void* stream) {
  return run_split(plan, m, n, k, A, lda, B, ldb, C, ldc, static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------
// Batches: many independent FP64 problems, each with its own plan (or classical), in one
// persistent launch.  The reference runs one generated entry point per call
// (meta/abc_gen_mix.py:448-472); a batch is the GPU form of calling it for many shapes.
// ---------------------------------------------------------------------------------------
struct fmm_batch {
  struct Job {
    int prob;                      // problem index
    const fmm_plan* plan;          // tables to run (the classical plan for strips)
    int grid[3];                   // plan dims (1,1,1 for classical)
    int ms, ns, ks;                // sub-block sizes
    int a_r, a_c, b_r, b_c, c_r, c_c;  // operand offsets (row, column) inside the problem
    PresumPlan pp;                 // its pre-summed operands (FMM jobs)
    size_t ws_off;                 // byte offset of S (then T) in the workspace
    int chunks, tiles_m, tiles_n, units;
    int S, d;                      // classical jobs: the k parts a single call makes (classical_parts)
    int depth;                     // of the parts of a product's sums (sum_depth)
    bool parts;                    // more than one of them
    const fmm::Prod* vprods;       // their tables when S > 1
    const fmm::Term* vterms;
    size_t ticket_off;             // int offset into the ticket array
    double cost;                   // estimated k steps per unit (scheduling order)
  };
  int count = 0;
  int dev = 0;
  std::vector<int> m, n, k;
  std::vector<const fmm_plan*> plans;
  // One products launch and, before it, the launch of its operand sums: usually one group of all FMM cores and
  // disjoint strips (several, which use the same workspace in turn, where their sums together are too
  // large), then the k strips.
  struct Group {
    int job0 = 0, njob = 0;        // its jobs
    int start0 = 0, units = 0;     // its njob + 1 entries of unit_start
    int ps0 = 0, nps = 0;          // its tasks of the operand sums
    bool parts = false;            // some job's products are summed in parts
    bool tma = true;               // this call's operands: all read by tensor copies
  };
  std::vector<Job> jobs;           // by group
  std::vector<Group> groups;
  bool k_strips = false;           // the last group holds the k strips
  std::vector<int> unit_start;
  int max_slots = 0, presum_cap = 1;
  long long max_presum_chunks = 1;
  int n_presum = 0;
  size_t n_tickets = 0, ws_bytes = 0, max_job_ws = 0;
  fmmt::ProdArgs* d_jobs = nullptr;
  int* d_start = nullptr;
  fmmt::ProdArgs* h_jobs = nullptr;  // pinned staging of the job tables
  fmm::PresumSide* d_ps = nullptr;
  fmm::PresumSide* h_ps = nullptr;
  int* d_tickets = nullptr;        // a work-unit counter per group, then the tickets
  char* d_ws = nullptr;
  // Even-pitch copies of A / B for problems whose row count is odd (a dense operand then
  // has an odd leading dimension, which tensor copies cannot stage): byte offsets into
  // d_pitch, or SIZE_MAX when the operand needs none.
  std::vector<size_t> pitch_a, pitch_b;
  size_t pitch_bytes = 0;
  char* d_pitch = nullptr;
  fmm::PitchCopy* d_pc = nullptr;
  fmm::PitchCopy* h_pc = nullptr;
  cudaEvent_t staged = nullptr;    // the staging buffers' last copies are done
};

namespace {

// Products per unit: units of about the work of a 64 x 64 x 4096 classical tile, so the
// persistent grid balances across problems of very different sizes.
int batch_chunks(int nprod, int ks) {
  const long long ksteps = (long long)nprod * ((ks + 7) / 8);
  long long c = (ksteps + 511) / 512;
  if (c < 1) c = 1;
  if (c > nprod) c = nprod;
  return (int)c;
}

void batch_add_job(fmm_batch* b, std::vector<fmm_batch::Job>& jobs, int prob, const fmm_plan* plan, int ms, int ns, int ks, int a_r, int a_c,
                   int b_r, int b_c, int c_r, int c_c) {
  if (ms <= 0 || ns <= 0 || ks <= 0) return;
  fmm_batch::Job j{};
  j.prob = prob;
  j.plan = plan;
  std::memcpy(j.grid, plan->dims, sizeof(j.grid));
  j.ms = ms;
  j.ns = ns;
  j.ks = ks;
  j.a_r = a_r;
  j.a_c = a_c;
  j.b_r = b_r;
  j.b_c = b_c;
  j.c_r = c_r;
  j.c_c = c_c;
  j.S = 1;
  j.d = ks;
  int nprod = plan->rank, depth = ks;
  if (is_classical(plan)) {
    classical_parts(ms, ns, ks, &j.S, &j.d);
    nprod = j.S;
    depth = j.d;
    j.depth = sum_depth(ms, ns, ks, 1);
    j.chunks = 1;  // one unit adds all its parts, in order
  } else {
    // operands with an odd row count or k get slots throughout, so that no pitch copy of them
    // is needed for the core
    j.pp = presum_plan(plan, ms, ns, ks, (b->m[prob] & 1) || (b->k[prob] & 1));
    b->max_slots = std::max(b->max_slots, std::max(j.pp.nA, j.pp.nB));
    b->presum_cap = std::max(b->presum_cap, presum_cap(plan));
    const long long ca = j.pp.nA ? (j.pp.ldS / 2) * j.pp.kk : 0, cb = j.pp.nB ? (j.pp.ldT / 2) * ns : 0;
    b->max_presum_chunks = std::max(b->max_presum_chunks, (std::max(ca, cb) + kPsChunk - 1) / kPsChunk);
    depth = j.pp.kk;
    j.depth = product_depth(plan, ms, ns, ks);
    j.chunks = batch_chunks(nprod, depth);
  }
  j.parts = j.depth < depth;
  j.tiles_m = (ms + 63) / 64;
  j.tiles_n = (ns + 63) / 64;
  j.units = j.tiles_m * j.tiles_n * j.chunks;
  j.ticket_off = b->n_tickets;
  if (j.chunks > 1) b->n_tickets += 4 * (size_t)j.tiles_m * j.tiles_n;
  j.cost = (double)nprod / j.chunks * ((depth + 7) / 8);
  jobs.push_back(j);
}

// Append `jobs` to the batch, longest units first (the persistent grid takes units in order, so the short
// ones fill in at the end), in groups whose operand sums take at most `budget` bytes (one job's at least).
// A group has at most kMaxPresumTasks tasks, the z extent of their launch.
constexpr int kMaxPresumTasks = 65535;
int batch_group(fmm_batch* b, std::vector<fmm_batch::Job>& jobs, long long budget) {
  std::stable_sort(jobs.begin(), jobs.end(),
                   [](const fmm_batch::Job& x, const fmm_batch::Job& y) { return x.cost > y.cost; });
  fmm_batch::Group g{};
  size_t ws = 0;
  long long units = 0;
  auto close = [&] {
    if (g.njob == 0) return;
    b->unit_start.push_back((int)units);
    g.units = (int)units;
    b->groups.push_back(g);
  };
  for (fmm_batch::Job& j : jobs) {
    const size_t need = presum_bytes(j.pp);
    const int tasks = (j.pp.nA > 0) + (j.pp.nB > 0);
    if (g.njob == 0 || (need > 0 && (long long)(ws + need) > budget) || g.nps + tasks > kMaxPresumTasks) {
      close();
      g = fmm_batch::Group{};
      g.job0 = (int)b->jobs.size();
      g.start0 = (int)b->unit_start.size();
      g.ps0 = b->n_presum;
      ws = 0;
      units = 0;
    }
    j.ws_off = ws;
    ws += need;
    b->ws_bytes = std::max(b->ws_bytes, ws);
    b->max_job_ws = std::max(b->max_job_ws, need);
    g.nps += tasks;
    b->n_presum += tasks;
    g.parts = g.parts || j.parts;
    ++g.njob;
    b->unit_start.push_back((int)units);
    units += j.units;
    if (units > INT32_MAX) return FMM_E_UNSUPPORTED;
    DevTables* d = nullptr;
    int rc = device_tables(j.plan, &d);
    if (rc == FMM_OK && j.S > 1) rc = ksplit_tables(j.plan, BASE_SPLIT, j.S, &j.vprods, &j.vterms);
    if (rc != FMM_OK) return rc;
    b->jobs.push_back(j);
  }
  close();
  return FMM_OK;
}

// Operand sums a batch holds at a time: four times a single call's cap.  A batch of large problems keeps the
// one launch that its balance rests on (the 512-problem batch has 7 GB of sums), one of many small two-level
// problems, whose sums are up to 4.5 times their operands, stays runnable.
long long batch_budget() { return 4 * g_ws_limit.load(); }

// After an allocation of the batch failed: a budget of half its sums, or 0 when they are one job's already.
long long batch_smaller(const fmm_batch* b) {
  cudaGetLastError();
  return b->ws_bytes > b->max_job_ws ? (long long)(b->ws_bytes / 2) : 0;
}

void batch_free(fmm_batch* b) {
  if (b->d_jobs) cudaFree(b->d_jobs);
  if (b->d_start) cudaFree(b->d_start);
  if (b->h_jobs) cudaFreeHost(b->h_jobs);
  if (b->d_ps) cudaFree(b->d_ps);
  if (b->h_ps) cudaFreeHost(b->h_ps);
  if (b->d_tickets) cudaFree(b->d_tickets);
  if (b->d_ws) cudaFree(b->d_ws);
  if (b->d_pitch) cudaFree(b->d_pitch);
  if (b->d_pc) cudaFree(b->d_pc);
  if (b->h_pc) cudaFreeHost(b->h_pc);
  if (b->staged) cudaEventDestroy(b->staged);
  delete b;
}

// The host side of a batch: jobs per group in scheduling order, unit ranges, and the sizes
// of the tickets and workspaces (operand sums of at most `budget` bytes).  Allocates no device memory (the plans' tables are
// uploaded on first use by device_tables).
int batch_build(int count, const fmm_plan* const* plans, const int* m, const int* n, const int* k, long long budget,
                fmm_batch** out, const int* tile_m = nullptr) {
  if (!out || count <= 0 || !m || !n || !k) return FMM_E_INVALID;
  for (int i = 0; i < count; ++i) {
    if (m[i] < 0 || n[i] < 0 || k[i] < 0) return FMM_E_INVALID;
    if (tile_m && tile_m[i] != 0 && tile_m[i] != 128 && tile_m[i] != 64) return FMM_E_INVALID;
  }
  int dev = 0;
  int rc = configure_kernel(&dev);
  if (rc != FMM_OK) return rc;
  fmm_batch* b = new (std::nothrow) fmm_batch();
  if (!b) return FMM_E_NOMEM;
  b->count = count;
  b->dev = dev;
  b->m.assign(m, m + count);
  b->n.assign(n, n + count);
  b->k.assign(k, k + count);
  const fmm_plan* cls = classical_plan();
  std::vector<fmm_batch::Job> main, strips;  // strips: the k strips, which update their core's C
  for (int i = 0; i < count; ++i) {
    const fmm_plan* p = (plans && plans[i]) ? plans[i] : nullptr;
    b->plans.push_back(p);
    const bool live = m[i] > 0 && n[i] > 0 && k[i] > 0;
    auto reserve = [&](int rows, int cols) {
      const size_t off = b->pitch_bytes;
      b->pitch_bytes += (sizeof(double) * (size_t)(rows + 1) * cols + 255) & ~(size_t)255;
      return off;
    };
    b->pitch_a.push_back(live && (m[i] & 1) ? reserve(m[i], k[i]) : SIZE_MAX);
    b->pitch_b.push_back(live && (k[i] & 1) ? reserve(k[i], n[i]) : SIZE_MAX);
    if (!live) continue;
    if (!p || is_classical(p)) {
      batch_add_job(b, main, i, cls, m[i], n[i], k[i], 0, 0, 0, 0, 0, 0);
      continue;
    }
    // same partition and fringe regions as the single-problem path (run_fmm + peel)
    const int pm = p->dims[0] * kMR, pk = p->dims[1], pn = p->dims[2] * kNR;
    const int mr = m[i] % pm, kr = k[i] % pk, nr = n[i] % pn;
    const int md = m[i] - mr, kd = k[i] - kr, nd = n[i] - nr;
    if (md > 0 && nd > 0 && kd > 0)
      batch_add_job(b, main, i, p, md / p->dims[0], nd / p->dims[2], kd / p->dims[1], 0, 0, 0, 0, 0, 0);
    if (kr > 0 && md > 0 && nd > 0) batch_add_job(b, strips, i, cls, md, nd, kr, 0, kd, kd, 0, 0, 0);
    if (nr > 0) batch_add_job(b, main, i, cls, m[i], nr, k[i], 0, 0, 0, nd, 0, nd);
    if (mr > 0 && nd > 0) batch_add_job(b, main, i, cls, mr, nd, k[i], md, 0, 0, 0, md, 0);
  }
  rc = batch_group(b, main, budget);
  if (rc == FMM_OK) rc = batch_group(b, strips, budget);
  b->k_strips = !strips.empty();
  if (rc != FMM_OK) {
    batch_free(b);
    return rc;
  }
  *out = b;
  return FMM_OK;
}

int batch_create(int count, const fmm_plan* const* plans, const int* m, const int* n, const int* k, fmm_batch** out,
                 const int* tile_m = nullptr) {
  for (long long budget = batch_budget(); budget > 0;) {
    fmm_batch* b = nullptr;
    const int rc = batch_build(count, plans, m, n, k, budget, &b, tile_m);
    if (rc != FMM_OK) return rc;
    cudaError_t e = cudaSuccess;
    const size_t nj = b->jobs.size(), ns = b->unit_start.size();
    if (nj > 0) {
      e = cudaMalloc((void**)&b->d_jobs, sizeof(fmmt::ProdArgs) * nj);
      if (e == cudaSuccess) e = cudaMalloc((void**)&b->d_start, sizeof(int) * ns);
      if (e == cudaSuccess) e = cudaMallocHost((void**)&b->h_jobs, sizeof(fmmt::ProdArgs) * nj);
      if (e == cudaSuccess) e = cudaMemcpy(b->d_start, b->unit_start.data(), sizeof(int) * ns, cudaMemcpyHostToDevice);
    }
    if (e == cudaSuccess && b->n_presum > 0) {
      e = cudaMalloc((void**)&b->d_ps, sizeof(fmm::PresumSide) * b->n_presum);
      if (e == cudaSuccess) e = cudaMallocHost((void**)&b->h_ps, sizeof(fmm::PresumSide) * b->n_presum);
    }
    if (e == cudaSuccess) e = cudaMalloc((void**)&b->d_tickets, sizeof(int) * (b->groups.size() + b->n_tickets + 1));
    if (e == cudaSuccess && b->pitch_bytes > 0) {
      e = cudaMalloc((void**)&b->d_pitch, b->pitch_bytes);
      if (e == cudaSuccess) e = cudaMalloc((void**)&b->d_pc, sizeof(fmm::PitchCopy) * 2 * count);
      if (e == cudaSuccess) e = cudaMallocHost((void**)&b->h_pc, sizeof(fmm::PitchCopy) * 2 * count);
    }
    if (e == cudaSuccess && b->ws_bytes > 0) e = cudaMalloc((void**)&b->d_ws, b->ws_bytes);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->staged, cudaEventDisableTiming);
    if (e == cudaSuccess) {
      *out = b;
      return FMM_OK;
    }
    budget = e == cudaErrorMemoryAllocation ? batch_smaller(b) : 0;
    batch_free(b);
    if (budget == 0) return cuda_status(e);
  }
  return FMM_E_NOMEM;
}

// Fill the job table of one group for this call's operands; false if some operand cannot be
// read by tensor copies (the launch then carries the per-lane copies).
bool batch_fill(fmm_batch* b, const fmm_batch::Group& g, const double* const* A, const long* lda, const double* const* B,
                const long* ldb, double* const* C, const long* ldc, int* n_ps) {
  bool tma = true;
  for (int q = g.job0; q < g.job0 + g.njob; ++q) {
    const fmm_batch::Job& j = b->jobs[q];
    const DevTables& d = j.plan->dev[b->dev];
    fmmt::ProdArgs a{};
    const long long la = lda[j.prob], lb = ldb[j.prob], lc = ldc[j.prob];
    a.A = A[j.prob] + j.a_r + (long long)j.a_c * la;
    a.lda = la;
    a.B = B[j.prob] + j.b_r + (long long)j.b_c * lb;
    a.ldb = lb;
    a.C = C[j.prob] + j.c_r + (long long)j.c_c * lc;
    a.ldc = lc;
    a.ms = j.ms;
    a.ns = j.ns;
    a.ks = j.d;
    a.depth = j.depth;
    a.kcap = j.grid[1] * j.ks;
    a.nprod = j.plan->rank;
    a.tiles_m = j.tiles_m;
    a.tiles_n = j.tiles_n;
    a.chunks = j.chunks;
    a.mode = fmm::MODE_ACCUM_C;
    a.tickets = j.chunks > 1 ? b->d_tickets + b->groups.size() + j.ticket_off : nullptr;
    a.status = dev_status[b->dev];
    const PresumPlan& pp = j.pp;
    double* S = reinterpret_cast<double*>(b->d_ws + j.ws_off);
    double* T = reinterpret_cast<double*>(b->d_ws + j.ws_off + pp.s_bytes);
    if (is_classical(j.plan)) {
      a.prods = j.S > 1 ? j.vprods : d.prods;
      a.terms = j.S > 1 ? j.vterms : d.terms;
      a.nprod = j.S;
    } else {
      a.ks = pp.kk;
      a.prods = pp.all ? d.prods_all : d.prods_ps;
      a.terms = pp.all ? d.terms_all : d.terms_ps;
      if (pp.nA > 0)
        b->h_ps[(*n_ps)++] = presum_side(d, 0, a.A, la, j.ms, j.ns, j.ks, pp.kk, S, pp.ldS,
                                         pp.all ? d.plist_all : d.plistA, pp.nA);
      if (pp.nB > 0)
        b->h_ps[(*n_ps)++] = presum_side(d, 1, a.B, lb, j.ms, j.ns, j.ks, pp.kk, T, pp.ldT,
                                         pp.all ? d.plist_all : d.plistB, pp.nB);
    }
    const long long am = (long long)j.grid[0] * j.ms, ak = (long long)j.grid[1] * j.ks,
                    bn = (long long)j.grid[2] * j.ns;
    // an operand with slots throughout is never read in place
    a.a_tma = pp.all || make_a_map(&a.tmA, a.A, am, ak, la);
    a.b_tma = pp.all || make_b_map(&a.tmB, a.B, ak, bn, lb, 64);
    bool ok = true;
    if (pp.nA > 0) ok = make_a_map(&a.tmAw, S, j.ms, (long long)pp.nA * pp.kk, pp.ldS);
    if (pp.nB > 0) ok = ok && make_b_map(&a.tmBw, T, pp.kk, (long long)pp.nB * j.ns, pp.ldT, 64);
    tma = tma && ok && a.a_tma && a.b_tma;
    b->h_jobs[q] = a;
  }
  return tma;
}

void batch_prepare(fmm_batch* b, const double* const* A, const long* lda, const double* const* B, const long* ldb,
                   double* const* C, const long* ldc, int* n_pc_out);
int batch_launch(fmm_batch* b, cudaStream_t st, int n_pc);

int batch_run(fmm_batch* b, const double* const* A, const long* lda, const double* const* B, const long* ldb,
              double* const* C, const long* ldc, cudaStream_t st) {
  if (!b || !A || !lda || !B || !ldb || !C || !ldc) return FMM_E_INVALID;
  int dev = 0;
  FMM_CUDA_TRY(cudaGetDevice(&dev));
  if (dev != b->dev) return FMM_E_INVALID;
  for (int i = 0; i < b->count; ++i) {
    int rc = check_args(b->m[i], b->n[i], b->k[i], A[i], lda[i], B[i], ldb[i], C[i], ldc[i]);
    if (rc != FMM_OK) return rc;
  }
  // The staging buffers are reused: the previous call's copies out of them must be done.
  // Inside a stream capture the copies become graph nodes that read the staging buffers
  // at every replay, so a graph replays with the most recent call's operands.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  FMM_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
  if (cap == cudaStreamCaptureStatusNone) FMM_CUDA_TRY(cudaEventSynchronize(b->staged));
  int n_pc = 0;
  batch_prepare(b, A, lda, B, ldb, C, ldc, &n_pc);
  if (!b->jobs.empty())
    FMM_CUDA_TRY(cudaMemcpyAsync(b->d_jobs, b->h_jobs, sizeof(fmmt::ProdArgs) * b->jobs.size(), cudaMemcpyHostToDevice,
                                 st));
  if (b->n_presum > 0)
    FMM_CUDA_TRY(cudaMemcpyAsync(b->d_ps, b->h_ps, sizeof(fmm::PresumSide) * b->n_presum, cudaMemcpyHostToDevice, st));
  if (n_pc > 0)
    FMM_CUDA_TRY(cudaMemcpyAsync(b->d_pc, b->h_pc, sizeof(fmm::PitchCopy) * n_pc, cudaMemcpyHostToDevice, st));
  if (cap == cudaStreamCaptureStatusNone) FMM_CUDA_TRY(cudaEventRecord(b->staged, st));
  return batch_launch(b, st, n_pc);
}

// This call's job tables (host staging): even-pitch copies for odd leading dimensions,
// per-job arguments and tensor maps, pre-sum tasks.
void batch_prepare(fmm_batch* b, const double* const* A, const long* lda, const double* const* B, const long* ldb,
                   double* const* C, const long* ldc, int* n_pc_out) {
  // Operands with an odd leading dimension and a reserved even-pitch copy are staged
  // through it (rows + 1 pitch); the others are used in place.
  std::vector<const double*> eA(A, A + b->count), eB(B, B + b->count);
  std::vector<long> elda(lda, lda + b->count), eldb(ldb, ldb + b->count);
  int n_pc = 0;
  for (int i = 0; i < b->count; ++i) {
    if ((lda[i] & 1) && b->pitch_a[i] != SIZE_MAX) {
      double* dst = reinterpret_cast<double*>(b->d_pitch + b->pitch_a[i]);
      b->h_pc[n_pc++] = fmm::PitchCopy{A[i], lda[i], dst, b->m[i] + 1LL, b->m[i], b->k[i]};
      eA[i] = dst;
      elda[i] = b->m[i] + 1;
    }
    if ((ldb[i] & 1) && b->pitch_b[i] != SIZE_MAX) {
      double* dst = reinterpret_cast<double*>(b->d_pitch + b->pitch_b[i]);
      b->h_pc[n_pc++] = fmm::PitchCopy{B[i], ldb[i], dst, b->k[i] + 1LL, b->k[i], b->n[i]};
      eB[i] = dst;
      eldb[i] = b->k[i] + 1;
    }
  }
  int n_ps = 0;
  for (fmm_batch::Group& g : b->groups) g.tma = batch_fill(b, g, eA.data(), elda.data(), eB.data(), eldb.data(), C, ldc, &n_ps);
  *n_pc_out = n_pc;
}

// Enqueue the launches of a prepared batch whose tables are (being) copied to the device.
int batch_launch(fmm_batch* b, cudaStream_t st, int n_pc) {
  // the groups' work-unit counters and every ticket start at zero
  FMM_CUDA_TRY(cudaMemsetAsync(b->d_tickets, 0, sizeof(int) * (b->groups.size() + b->n_tickets), st));
  if (n_pc > 0) {
    ProfScope pf(K_PITCH_COPY, st);
    fmm::fmm_pitch_copy_kernel<<<dim3(256, (unsigned)n_pc), 256, 0, st>>>(b->d_pc);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    FMM_CUDA_TRY(cudaGetLastError());
  }
  for (size_t q = 0; q < b->groups.size(); ++q) {
    const fmm_batch::Group& g = b->groups[q];
    if (g.nps > 0) {
      ProfScope pf(K_PRESUM_BATCH, st);
      const long long nc = std::min<long long>(b->max_presum_chunks, 1 << 16);
      fmm::fmm_presum_batch_kernel<<<dim3((unsigned)nc, presum_ranges(nc * g.nps, b->max_slots, sm_count[b->dev]),
                                          (unsigned)g.nps),
                                     fmm::PS_THREADS, fmm::presum_smem_bytes(b->presum_cap), st>>>(b->d_ps + g.ps0,
                                                                                                   b->presum_cap);
      g_launches.fetch_add(1, std::memory_order_relaxed);
      FMM_CUDA_TRY(cudaGetLastError());
    }
    fmmt::ProdBatchArgs ba{};
    ba.jobs = b->d_jobs + g.job0;
    ba.unit_start = b->d_start + g.start0;
    ba.njobs = g.njob;
    ba.units = g.units;
    ba.status = dev_status[b->dev];
    ba.counter = b->d_tickets + q;
    const unsigned grid =
        (unsigned)std::min<long long>(ba.units, (long long)sm_count[b->dev] * fmmt::TileShape<64, 64>::CTAS);
    ProfScope pf(K_PRODUCTS_BATCH, st);
    auto kernel = g.tma ? (g.parts ? fmmt::fmm_products_batch_kernel<false, true> : fmmt::fmm_products_batch_kernel<false, false>)
                        : (g.parts ? fmmt::fmm_products_batch_kernel<true, true> : fmmt::fmm_products_batch_kernel<true, false>);
    const int rc = launch_dependent(kernel, dim3(grid), fmmt::NT,
                                    spread_smem(fmmt::ProdShape<64>::SMEM, grid, sm_count[b->dev]), st, 1, ba);
    if (rc != FMM_OK) return rc;
  }
  return FMM_OK;
}

}  // namespace

extern "C" {

int fmm_batch_create(int count, const fmm_plan* const* plans, const int* m, const int* n, const int* k,
                     fmm_batch** out) {
  return batch_create(count, plans, m, n, k, out);
}

int fmm_batch_create_tiled(int count, const fmm_plan* const* plans, const int* m, const int* n, const int* k,
                           const int* tile_m, fmm_batch** out) {
  return batch_create(count, plans, m, n, k, out, tile_m);
}

int fmm_batch_dgemm(fmm_batch* batch, const double* const* A, const long* lda, const double* const* B,
                    const long* ldb, double* const* C, const long* ldc, void* stream) {
  return batch_run(batch, A, lda, B, ldb, C, ldc, static_cast<cudaStream_t>(stream));
}

int fmm_batch_units(const fmm_batch* batch, int phase) {
  if (!batch || phase < 0 || phase > 1) return FMM_E_INVALID;
  const size_t main = batch->groups.size() - (batch->k_strips ? 1 : 0);
  long long units = 0;
  for (size_t q = phase == 0 ? 0 : main; q < (phase == 0 ? main : batch->groups.size()); ++q) units += batch->groups[q].units;
  return (int)std::min<long long>(units, INT32_MAX);
}

int fmm_batch_destroy(fmm_batch* batch) {
  if (!batch) return FMM_E_INVALID;
  cudaEventSynchronize(batch->staged);
  batch_free(batch);
  return FMM_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// One-shot batches for request loops: the batch is formed, run and released per call with
// no cudaMalloc / cudaFree (those synchronise the device, which would stop the requests
// of a serving loop from overlapping).  Device buffers come from the stream-ordered pool;
// the job tables go through a ring of pinned host buffers, each reused only after the
// copy out of it has completed.
// ---------------------------------------------------------------------------------------
namespace {

struct PinnedRing {
  static constexpr int N = 8;
  char* buf[N] = {};
  size_t cap[N] = {};
  cudaEvent_t ev[N] = {};
  int next = 0;
  std::mutex mu;
};
PinnedRing g_ring[kMaxDevices];

int ring_acquire(int dev, size_t bytes, char** buf, cudaEvent_t* ev) {
  PinnedRing& r = g_ring[dev];
  std::lock_guard<std::mutex> lk(r.mu);
  const int s = r.next;
  r.next = (s + 1) % PinnedRing::N;
  if (!r.ev[s]) FMM_CUDA_TRY(cudaEventCreateWithFlags(&r.ev[s], cudaEventDisableTiming));
  FMM_CUDA_TRY(cudaEventSynchronize(r.ev[s]));  // the slot's previous copy is done
  if (r.cap[s] < bytes) {
    if (r.buf[s]) cudaFreeHost(r.buf[s]);
    r.buf[s] = nullptr;
    r.cap[s] = 0;
    const size_t cap = std::max<size_t>(bytes + bytes / 2, (size_t)1 << 20);
    FMM_CUDA_TRY(cudaMallocHost((void**)&r.buf[s], cap));
    r.cap[s] = cap;
  }
  *buf = r.buf[s];
  *ev = r.ev[s];
  return FMM_OK;
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

int batch_submit(int count, const fmm_plan* const* plans, const int* m, const int* n, const int* k,
                 const double* const* A, const long* lda, const double* const* B, const long* ldb, double* const* C,
                 const long* ldc, cudaStream_t st) {
  if (!A || !lda || !B || !ldb || !C || !ldc) return FMM_E_INVALID;
  for (int i = 0; i < count; ++i) {
    int rc = check_args(m[i], n[i], k[i], A[i], lda[i], B[i], ldb[i], C[i], ldc[i]);
    if (rc != FMM_OK) return rc;
  }
  fmm_batch* b = nullptr;
  size_t o_jobs = 0, o_start, o_ps, o_pc, table_bytes, o_tk, o_ws, o_pt;
  char *stage = nullptr, *blk = nullptr;
  cudaEvent_t stage_ev = nullptr;
  int rc = FMM_E_NOMEM;
  for (long long budget = batch_budget(); budget > 0;) {
    rc = batch_build(count, plans, m, n, k, budget, &b);
    if (rc != FMM_OK) return rc;
    // table block (identical layout in pinned staging and on the device)
    o_start = align_up(o_jobs + sizeof(fmmt::ProdArgs) * b->jobs.size(), 16);
    o_ps = align_up(o_start + sizeof(int) * b->unit_start.size(), 64);
    o_pc = align_up(o_ps + sizeof(fmm::PresumSide) * b->n_presum, 64);
    table_bytes = align_up(o_pc + sizeof(fmm::PitchCopy) * 2 * count, 256);
    o_tk = table_bytes;
    o_ws = align_up(o_tk + sizeof(int) * (b->groups.size() + b->n_tickets), 256);
    o_pt = align_up(o_ws + b->ws_bytes, 256);
    rc = cuda_status(cudaMallocAsync((void**)&blk, o_pt + b->pitch_bytes, st));
    if (rc == FMM_OK) break;
    budget = rc == FMM_E_NOMEM ? batch_smaller(b) : 0;
    batch_free(b);
    b = nullptr;
  }
  if (rc != FMM_OK) return rc;
  rc = ring_acquire(b->dev, table_bytes, &stage, &stage_ev);
  if (rc != FMM_OK) {
    cudaFreeAsync(blk, st);
    batch_free(b);
    return rc;
  }
  b->h_jobs = reinterpret_cast<fmmt::ProdArgs*>(stage + o_jobs);
  b->d_jobs = reinterpret_cast<fmmt::ProdArgs*>(blk + o_jobs);
  b->d_start = reinterpret_cast<int*>(blk + o_start);
  if (!b->unit_start.empty()) std::memcpy(stage + o_start, b->unit_start.data(), sizeof(int) * b->unit_start.size());
  b->h_ps = reinterpret_cast<fmm::PresumSide*>(stage + o_ps);
  b->d_ps = reinterpret_cast<fmm::PresumSide*>(blk + o_ps);
  b->h_pc = reinterpret_cast<fmm::PitchCopy*>(stage + o_pc);
  b->d_pc = reinterpret_cast<fmm::PitchCopy*>(blk + o_pc);
  b->d_tickets = reinterpret_cast<int*>(blk + o_tk);
  b->d_ws = b->ws_bytes ? blk + o_ws : nullptr;
  b->d_pitch = b->pitch_bytes ? blk + o_pt : nullptr;
  int n_pc = 0;
  batch_prepare(b, A, lda, B, ldb, C, ldc, &n_pc);
  rc = cuda_status(cudaMemcpyAsync(blk, stage, table_bytes, cudaMemcpyHostToDevice, st));
  if (rc == FMM_OK) rc = cuda_status(cudaEventRecord(stage_ev, st));
  if (rc == FMM_OK) rc = batch_launch(b, st, n_pc);
  cudaError_t fe = cudaFreeAsync(blk, st);
  if (rc == FMM_OK) rc = cuda_status(fe);
  // the buffers belong to the pool and the ring: detach them before freeing the host side
  b->h_jobs = nullptr, b->d_jobs = nullptr, b->d_start = nullptr;
  b->h_ps = nullptr, b->d_ps = nullptr, b->h_pc = nullptr, b->d_pc = nullptr;
  b->d_tickets = nullptr, b->d_ws = nullptr, b->d_pitch = nullptr;
  batch_free(b);
  return rc;
}

}  // namespace

extern "C" int fmm_batch_submit(int count, const fmm_plan* const* plans, const int* m, const int* n, const int* k,
                                const double* const* A, const long* lda, const double* const* B, const long* ldb,
                                double* const* C, const long* ldc, void* stream) {
  return batch_submit(count, plans, m, n, k, A, lda, B, ldb, C, ldc, static_cast<cudaStream_t>(stream));
}
