// fmm_b200 device code shared by the FP64 kernels (barriers, bounded waits, work-unit claims,
// DMMA), the operand sums and combine passes, and the folding GEMM of the no-allocation entry
// point: a persistent, warp-specialised FP64 DMMA GEMM whose producer warpgroup forms the U/V
// linear combinations of A and B sub-blocks while staging them into shared memory, and whose
// consumer warpgroups scatter each product into every C block with a nonzero W coefficient.
// The other FP64 launches run the tile kernels of fmm_tile.cuh.  sm_100a only.
//
// Mapping of the reference's CPU design (fmm-gen):
//   * BLIS packing with fused sums (meta/abc_gen_mix.py:171-251, packA/B_add_stra_abc<r>)
//     -> fmm_presum_staged_kernel, fmm_presum_kernel (operand sums formed in HBM; S_Add / T_Add of
//        meta/naive_gen_mix.py:60-137 too), or the folding GEMM's producer warps (cp.async /
//        TMA of every U/V term tile, folded into the operand stage).
//   * AVX 8x4 micro-kernel (common/kernels/bl_dgemm_asm_8x4.c)
//     -> mma.sync.m16n8k4 FP64 (DMMA) fragments.
//   * multi-destination C update (meta/abc_micro_kernel_gen.py:147-244)
//     -> epilogue C_l += W[l,r] * M_r for every nonzero W of product r.  A work unit owns one
//        tile position in all C blocks; tickets per tile (or per tile and C block) order the
//        units' C updates (bounded spin, error flag on timeout), so no two CTAs ever update
//        the same C element at once and every element receives its products in order
//        r = 0..R-1.
//   * M_Add (meta/ab_gen_mix.py:341-372)
//     -> fmm_combine_staged_kernel and fmm_combine_kernel (every C_l += W[l,r] M_r of the
//        stored products in one pass, the C blocks in groups that share products, running
//        values in registers; the staged form brings the M tiles in by bulk copies),
//        fmm_scatter_kernel (one C block per launch row, beyond the combine's tables).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace fmm {

constexpr int BM = 128;   // CTA tile rows (m)
constexpr int BN = 128;   // CTA tile columns (n)
constexpr int BK = 8;     // k depth of one operand stage
constexpr int NPROD = 256;               // producer threads (warpgroups 0, 1)
constexpr int NCONS = 256;               // consumer threads (warpgroups 2, 3)
constexpr int NTHREADS = NPROD + NCONS;  // 512
constexpr int LAUNCH_REGS = 65536 / NTHREADS;  // registers per thread at launch (128)
// Operand stages are dense: opA[k][m] (BK x BM) and opB[n][k] (BN x BK), exactly the
// layout a TMA box writes, so single-term operands are copied straight into a stage.
// (The consumers' FP64 fragment loads then see 4-way bank conflicts; shared-memory
// bandwidth has room for that: measured no loss against padded rows.)
constexpr int LDA_S = BM;      // opA[k][m]
constexpr int LDB_S = BK;      // opB[n][k]
constexpr int NSTAGE = 6;      // operand stages (producer -> consumers)
constexpr int NRAW = 6;        // cp.async path: thread-private raw term slots in flight
constexpr int EA = BM * BK / NPROD;  // A elements a producer thread stages per term (8)
constexpr int EB = BN * BK / NPROD;  // B elements a producer thread stages per term (8)
constexpr int OPA_SZ = BK * LDA_S;
constexpr int OPB_SZ = BN * LDB_S;
constexpr int STAGE_SZ = OPA_SZ + OPB_SZ;
constexpr int RAW_SZ = (EA + EB) * NPROD;
// TMA staging: one raw slot holds an A term box (BK x BM, m contiguous) and a B term box
// (BN columns of BK + 2 k values, k contiguous; two wider so that a box can start at the
// even k coordinate at or below an odd one).
constexpr int TB_K = BK + 2;
constexpr int TRAW_A = BK * BM;
constexpr int TRAW_SZ = TRAW_A + BN * TB_K;
constexpr int NRAW_TMA = 6;
constexpr int NFOLD = NPROD - 32;  // folding threads: producer warps 1..7 (warp 0 issues TMA)
constexpr int FPAIRS = (BM * BK / 2 + NFOLD - 1) / NFOLD;  // A element pairs per folding thread
constexpr int FELEMS = (BN * BK + NFOLD - 1) / NFOLD;      // B elements per folding thread
constexpr unsigned TMA_BYTES_A = TRAW_A * sizeof(double);
constexpr unsigned TMA_BYTES_B = BN * TB_K * sizeof(double);   // raw B box (k rounded down to even)
constexpr unsigned TMA_BYTES_B8 = BN * BK * sizeof(double);    // direct B box
static_assert((NSTAGE * STAGE_SZ * sizeof(double)) % 128 == 0, "raw slots must start 128-byte aligned");
static_assert((TRAW_SZ * sizeof(double)) % 128 == 0, "TMA raw slots must be 128-byte aligned");
static_assert((TRAW_A * sizeof(double)) % 128 == 0, "TMA B box must be 128-byte aligned");
constexpr int UQ_DEPTH = 16;  // work-unit ring entries (see UnitClaimer)
constexpr size_t RING_BYTES = 2 * UQ_DEPTH * sizeof(unsigned long long) + UQ_DEPTH * sizeof(int);
constexpr size_t SMEM_BYTES_CPASYNC = (size_t)(NSTAGE * STAGE_SZ + NRAW * RAW_SZ) * sizeof(double) +
                                      (2 * NSTAGE + 2 * NRAW_TMA) * sizeof(unsigned long long) + RING_BYTES;
// What the folding warps need to know about a raw slot, written by the issuer before
// the slot's TMA copies (published by the release of its arrive.expect_tx).
struct SlotMeta {
  double ca, cb;  // coefficients of the staged A and B terms
  int shift;      // B box starts one k before the term's first k
  int pad[3];
};
constexpr size_t SMEM_BYTES_TMA = (size_t)(NSTAGE * STAGE_SZ + NRAW_TMA * TRAW_SZ) * sizeof(double) +
                                  NRAW_TMA * sizeof(SlotMeta) +
                                  (2 * NSTAGE + 2 * NRAW_TMA) * sizeof(unsigned long long) + RING_BYTES;
constexpr size_t smem_bytes(bool tma) { return tma ? SMEM_BYTES_TMA : SMEM_BYTES_CPASYNC; }
constexpr int GROUP_M = 8;  // tile raster: groups of 8 tile rows for L2 reuse
constexpr int C_BATCH_J = 4;          // epilogue: 8-column groups per batch of C loads (4 elements each);
                                      // 4 (16 loads in flight per thread) measured 1-8 % faster than 2
constexpr int C_PREFETCH_STEPS = 24;  // k steps before a product's end at which its C tiles are prefetched
                                      // (at its first k step when it has fewer)
constexpr int PROD_REGS = 72;
constexpr int CONS_REGS = 184;
static_assert(NPROD * PROD_REGS + NCONS * CONS_REGS <= NTHREADS * LAUNCH_REGS,
              "register split exceeds the launch budget");
constexpr unsigned long long WAIT_LIMIT_NS = 4000000000ULL;  // bounded device-side waits give up after 4 s
// try_wait suspends the waiting thread until the phase completes or this many ns pass,
// so waiting warps do not take issue slots from the warps they wait for.
constexpr unsigned MBAR_SUSPEND_NS = 20000;

struct Term {
  int row;      // global block row in the composed grid
  int col;      // global block column
  double coef;  // coefficient
  int src;      // A/B terms: 0 = the operand matrix, 1 = the pre-summed workspace (S / T)
  int pad;      // C terms: this product's position among the products with a term in the
                // same C block (product order); the per-block tickets count up to it
};

struct Prod {
  int a0, na;   // A terms: terms[a0 .. a0+na)
  int b0, nb;   // B terms
  int c0, nc;   // C terms
};

enum Mode : int { MODE_ACCUM_C = 0, MODE_STORE_M = 1 };

// STATUS_TICKET_TIMEOUT: a wait for another CTA's C updates gave up (the kernel finishes,
// without the product order from then on); STATUS_WAIT_TIMEOUT: a wait inside a CTA's own
// pipeline gave up (every later wait returns at once and the kernel winds down).
// STATUS_TABLE: a kernel found an index outside its tables (clamped; the result is void)
enum StatusBits : unsigned { STATUS_TICKET_TIMEOUT = 1u, STATUS_WAIT_TIMEOUT = 2u, STATUS_TABLE = 4u };

// Time limit of the bounded device-side waits in ns: WAIT_LIMIT_NS unless a test lowers it
// (fmm_debug_set); read only on a wait's slow path.
__device__ unsigned long long g_wait_limit_ns = WAIT_LIMIT_NS;
__device__ __forceinline__ unsigned long long wait_limit_ns() {
  return *reinterpret_cast<volatile unsigned long long*>(&g_wait_limit_ns);
}

struct GemmArgs {
  CUtensorMap tmA;   // whole-matrix tensor maps (TMA path), FP64: A (m x k), box BM x BK
  CUtensorMap tmB;   // B (k x n), box BK x BN (direct loads)
  CUtensorMap tmB2;  // B (k x n), box (BK + 2) x BN (raw loads at even k)
  const double* A;
  long long lda;
  const double* B;
  long long ldb;
  double* C;        // C blocks receive C_l += w * M_r
  long long ldc;
  int ms, ns, ks;   // sub-block sizes
  const Prod* prods;
  const Term* terms;
  int nprod;
  int tiles_m, tiles_n;
  int* tickets;     // per tile: products whose C updates are done (zeroed before launch); used when nprod > 1
  unsigned* status; // device status word (StatusBits)
  int* counter;     // work units claimed so far in this launch (zeroed before launch)
};

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void cp_async8(unsigned dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile(
      "{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(bar),
      "r"(bytes)
      : "memory");
}

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile(
      "{\n .reg .b64 st;\n mbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n}\n" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2, %3;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(MBAR_SUSPEND_NS)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;\n" : "=l"(t));
  return t;
}

// Bounded wait for the phase with the given parity.  Every phase is completed by another
// role of the same CTA, so in a correct run the wait ends; if it has not after the wait
// limit, the status word gets STATUS_WAIT_TIMEOUT and every later such wait of every CTA
// returns at once, so the kernel still finishes and the host reports FMM_E_TIMEOUT.  A
// ticket timeout alone (STATUS_TICKET_TIMEOUT) does not cut these waits short: the
// pipeline keeps running and every issued copy is consumed before the kernel ends.
__device__ __forceinline__ void mbar_wait(unsigned bar, unsigned parity, unsigned* status) {
  if (mbar_try_wait(bar, parity)) return;
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if ((*(volatile unsigned*)status & STATUS_WAIT_TIMEOUT) != 0u) return;
    if (global_ns() - t0 > wait_limit_ns()) {
      atomicOr(status, STATUS_WAIT_TIMEOUT);
      return;
    }
  }
}

// Wait for a phase with a time limit only (no early exit on the status word): used at the
// end of a role for copies that may still be in flight (only on an error path, where
// other roles stopped consuming; in a normal run these phases have long completed).
__device__ __forceinline__ void mbar_wait_drain(unsigned bar, unsigned parity) {
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > wait_limit_ns()) return;
  }
}

__device__ __forceinline__ void named_bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(count) : "memory");
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;\n" ::"l"(p), "r"(v) : "memory");
}

// Bounded wait for a ticket written by another CTA: until *p >= target.  On timeout the
// status word gets STATUS_TICKET_TIMEOUT; once any status bit is set, ticket waits return
// at once.
__device__ __forceinline__ void ticket_spin(const int* p, int target, unsigned* status, unsigned sleep_ns) {
  if (ld_acquire(p) >= target) return;
  const unsigned long long t0 = global_ns();
  while (ld_acquire(p) < target) {
    if (*(volatile unsigned*)status != 0u) return;
    if (global_ns() - t0 > wait_limit_ns()) {
      atomicOr(status, STATUS_TICKET_TIMEOUT);
      return;
    }
    __nanosleep(sleep_ns);
  }
}

__device__ __forceinline__ void dmma_16x8x4(double (&d)[4], const double (&a)[2], double b) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a[0]), "d"(a[1]), "d"(b));
}

__device__ __forceinline__ int prod_T(const Prod& p) { return p.na > p.nb ? p.na : p.nb; }

// Work unit u -> (tile position, product).  Product-major order: the units of one tile are a
// whole tile grid apart, so a later product is claimed well after the earlier one.
struct Unit {
  int m0, n0, tile, r;
};

__device__ __forceinline__ Unit decode_unit(const GemmArgs& a, int u) {
  const int ntiles = a.tiles_m * a.tiles_n;
  Unit w;
  const int bid = u % ntiles;
  w.r = u / ntiles;
  const int per_group = GROUP_M * a.tiles_n;
  const int grp = bid / per_group;
  const int first_m = grp * GROUP_M;
  const int rows_here = min(a.tiles_m - first_m, GROUP_M);
  const int in_grp = bid % per_group;
  w.m0 = (first_m + in_grp % rows_here) * BM;
  w.n0 = (in_grp / rows_here) * BN;
  w.tile = bid;
  return w;
}

__device__ __forceinline__ int num_units(const GemmArgs& a) { return a.tiles_m * a.tiles_n * a.nprod; }

// ------------------------------------------------------------------------------------
// Work-unit claims.  One thread of each CTA (the operand issuer) claims the launch's units
// in increasing order from a launch-wide counter and publishes each claimed index through
// a shared-memory ring; every other role of the CTA reads the ring in the same order
// (index -1 ends the sequence).  A unit waits only on tickets of lower-numbered units,
// which running CTAs claimed before it, so the launch makes progress whether or not all of
// its CTAs are resident at once (another kernel may hold some SMs).
//
// Ring depth: the issuer runs at most one operand pipeline (<= 6 stages of at least one
// unit each) plus the product-tile hand-off ahead of the slowest reader, so 16 entries never
// make it wait; if they did, the wait would end as the readers move on.
// ------------------------------------------------------------------------------------
struct UnitRing {
  unsigned base;  // shared address: UQ_DEPTH full barriers (entry published: 1 arrival, the
                  // claimer), UQ_DEPTH empty barriers (entry read by every reader warp), then
                  // UQ_DEPTH int entries
  __device__ __forceinline__ unsigned full(int s) const { return base + 8 * s; }
  __device__ __forceinline__ unsigned empty(int s) const { return base + 8 * (UQ_DEPTH + s); }
  __device__ __forceinline__ unsigned entry(int s) const { return base + 16 * UQ_DEPTH + 4 * s; }
};

__device__ __forceinline__ void st_shared_s32(unsigned addr, int v) {
  asm volatile("st.shared.s32 [%0], %1;\n" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_shared_s32(unsigned addr) {
  int v;
  asm volatile("ld.shared.s32 %0, [%1];\n" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// The claiming thread: next unit index of this CTA, or -1 when the launch has none left.
template <class Src>
struct UnitClaimer {
  const Src& src;
  UnitRing q;
  int n = 0;
  __device__ __forceinline__ int next() {
    const int slot = n % UQ_DEPTH;
    mbar_wait(q.empty(slot), (unsigned)(((n / UQ_DEPTH) & 1) ^ 1), src.status());
    int u = -1;
    if ((*(volatile unsigned*)src.status() & STATUS_WAIT_TIMEOUT) == 0u) {
      u = atomicAdd(src.counter(), 1);
      if (u >= src.total()) u = -1;
    }
    st_shared_s32(q.entry(slot), u);
    mbar_arrive(q.full(slot));  // release: the entry is visible to the readers' acquire
    ++n;
    return u;
  }
};

// A reader warp (all 32 lanes call next() together), or a lone thread (lone = true) whose
// warp has no other active lanes.  release = false reads an entry without freeing it (a
// second cursor of the same warp frees it later).
struct UnitReader {
  UnitRing q;
  unsigned* status;
  bool release;
  int n = 0;
  bool lone = false;
  __device__ __forceinline__ int next() {
    const int slot = n % UQ_DEPTH;
    mbar_wait(q.full(slot), (unsigned)((n / UQ_DEPTH) & 1), status);
    int u = ld_shared_s32(q.entry(slot));
    if ((*(volatile unsigned*)status & STATUS_WAIT_TIMEOUT) != 0u) u = -1;
    if (release) {
      if (lone) {
        mbar_arrive(q.empty(slot));
      } else {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(q.empty(slot));
      }
    }
    ++n;
    return u;
  }
};

__device__ __forceinline__ void unit_ring_init(const UnitRing& q, unsigned readers) {
  for (int s = 0; s < UQ_DEPTH; ++s) {
    mbar_init(q.full(s), 1);
    mbar_init(q.empty(s), readers);
  }
}

// ------------------------------------------------------------------------------------
// Producer: flattened stream of load units (k step s, term t) over the CTA's work units.
// ------------------------------------------------------------------------------------
struct LoadIter {
  int u;            // work unit index
  Unit w;
  Prod p;
  int T;
  int s, t;
  bool valid;
  // term t of the product, fetched when the iterator moves so that the global loads are
  // off the producer's critical path
  Term ta, tb;
};

// What a launch's claims need (UnitClaimer).
struct OneJob {
  const GemmArgs& a;
  __device__ __forceinline__ int total() const { return num_units(a); }
  __device__ __forceinline__ unsigned* status() const { return a.status; }
  __device__ __forceinline__ int* counter() const { return a.counter; }
};

__device__ __forceinline__ int num_ksteps(const GemmArgs& a) { return (a.ks + BK - 1) / BK; }

__device__ __forceinline__ void load_terms(const GemmArgs& a, LoadIter& it) {
  if (it.t < it.p.na) it.ta = a.terms[it.p.a0 + it.t];
  if (it.t < it.p.nb) it.tb = a.terms[it.p.b0 + it.t];
}

__device__ __forceinline__ void iter_enter_unit(const GemmArgs& a, LoadIter& it) {
  it.w = decode_unit(a, it.u);
  it.p = a.prods[it.w.r];
  it.T = prod_T(it.p);
  it.s = 0;
  it.t = 0;
  load_terms(a, it);
}

template <class Nx>
__device__ __forceinline__ void load_iter_unit(const GemmArgs& a, LoadIter& it, Nx& nx) {
  it.u = nx.next();
  it.valid = it.u >= 0;
  if (it.valid) iter_enter_unit(a, it);
}

template <class Nx>
__device__ __forceinline__ void load_iter_next(const GemmArgs& a, LoadIter& it, Nx& nx) {
  if (++it.t < it.T) {
    load_terms(a, it);
    return;
  }
  it.t = 0;
  if (++it.s < num_ksteps(a)) {
    if (it.T > 1) load_terms(a, it);
    return;
  }
  load_iter_unit(a, it, nx);
}

// Raw slot layout (thread-private, conflict-free): pair e of A at [e][pt] (16 B each),
// then the B pairs.  A term tile: 128 (m) x 8 (k) = 512 m-pairs, 4 per thread; B term
// tile: 8 (k) x 128 (n) = 512 k-pairs, 4 per thread.
constexpr int PA = EA / 2;  // A pairs per thread per term
constexpr int PB = EB / 2;

__device__ __forceinline__ void issue_unit(const GemmArgs& a, const LoadIter& it, double* raw_slot, int pt) {
  const unsigned sbase = smem_u32(raw_slot);
  if (it.t < it.p.na) {
    const double* M0 = a.A;
    const long long ld = a.lda;
    const long long off = (long long)it.ta.row * a.ms + (long long)it.ta.col * a.ks * ld;
    const double* base = M0 + off;
    const bool al16 = ((off & 1) == 0) && ((ld & 1) == 0) && ((reinterpret_cast<uintptr_t>(M0) & 15) == 0);
#pragma unroll
    for (int e = 0; e < PA; ++e) {
      const int q = e * NPROD + pt;        // pair index
      const int mm = 2 * (q % (BM / 2)), kk = q / (BM / 2);
      const int gm = it.w.m0 + mm, gk = it.s * BK + kk;
      const unsigned dst = sbase + (unsigned)(q * 16);
      if (al16) {
        const int nb = (gk < a.ks) ? ((gm + 1 < a.ms) ? 16 : (gm < a.ms ? 8 : 0)) : 0;
        cp_async16(dst, nb ? base + gm + (long long)gk * ld : M0, nb);
      } else {
        const bool v0 = (gk < a.ks) && (gm < a.ms), v1 = (gk < a.ks) && (gm + 1 < a.ms);
        cp_async8(dst, v0 ? base + gm + (long long)gk * ld : M0, v0 ? 8 : 0);
        cp_async8(dst + 8, v1 ? base + gm + 1 + (long long)gk * ld : M0, v1 ? 8 : 0);
      }
    }
  }
  if (it.t < it.p.nb) {
    const double* M0 = a.B;
    const long long ld = a.ldb;
    const long long off = (long long)it.tb.row * a.ks + (long long)it.tb.col * a.ns * ld;
    const double* base = M0 + off;
    const bool al16 = ((off & 1) == 0) && ((ld & 1) == 0) && ((reinterpret_cast<uintptr_t>(M0) & 15) == 0);
#pragma unroll
    for (int e = 0; e < PB; ++e) {
      const int q = e * NPROD + pt;
      const int kk = 2 * (q % (BK / 2)), nn = q / (BK / 2);
      const int gk = it.s * BK + kk, gn = it.w.n0 + nn;
      const unsigned dst = sbase + (unsigned)((PA * NPROD + q) * 16);
      if (al16) {
        const int nb = (gn < a.ns) ? ((gk + 1 < a.ks) ? 16 : (gk < a.ks ? 8 : 0)) : 0;
        cp_async16(dst, nb ? base + gk + (long long)gn * ld : M0, nb);
      } else {
        const bool v0 = (gn < a.ns) && (gk < a.ks), v1 = (gn < a.ns) && (gk + 1 < a.ks);
        cp_async8(dst, v0 ? base + gk + (long long)gn * ld : M0, v0 ? 8 : 0);
        cp_async8(dst + 8, v1 ? base + gk + 1 + (long long)gn * ld : M0, v1 ? 8 : 0);
      }
    }
  }
}

// Fold one staged term into the operand stage.  A producer thread reads back only the
// elements it copied itself, so no barrier is needed between arrival and use; the
// stage itself belongs to the producer between its empty and full barrier phases.
__device__ __forceinline__ void fold_unit(const LoadIter& it, const double* raw_slot, double* opA, double* opB,
                                          int pt) {
  if (it.t < it.p.na) {
    const double c = it.ta.coef;
#pragma unroll
    for (int e = 0; e < PA; ++e) {
      const int q = e * NPROD + pt;
      const int mm = 2 * (q % (BM / 2)), kk = q / (BM / 2);
      const double2 v = reinterpret_cast<const double2*>(raw_slot)[q];
      double2* dst = reinterpret_cast<double2*>(opA + kk * LDA_S + mm);
      if (it.t == 0) {
        *dst = make_double2(c * v.x, c * v.y);
      } else {
        const double2 o = *dst;
        *dst = make_double2(fma(c, v.x, o.x), fma(c, v.y, o.y));
      }
    }
  }
  if (it.t < it.p.nb) {
    const double c = it.tb.coef;
#pragma unroll
    for (int e = 0; e < PB; ++e) {
      const int q = e * NPROD + pt;
      const int kk = 2 * (q % (BK / 2)), nn = q / (BK / 2);
      const double2 v = reinterpret_cast<const double2*>(raw_slot)[PA * NPROD + q];
      double2* dst = reinterpret_cast<double2*>(opB + nn * LDB_S + kk);
      if (it.t == 0) {
        *dst = make_double2(c * v.x, c * v.y);
      } else {
        const double2 o = *dst;
        *dst = make_double2(fma(c, v.x, o.x), fma(c, v.y, o.y));
      }
    }
  }
}

// Warp 0 of the per-thread-copy producer: lane 0 claims, the warp shares the index.
struct WarpClaimer {
  UnitClaimer<OneJob> c;
  __device__ __forceinline__ int next() {
    int u = 0;
    if ((threadIdx.x & 31) == 0) u = c.next();
    return __shfl_sync(0xffffffffu, u, 0);
  }
};

// The per-thread-copy producer's cursor that runs ahead (issuing copies): warp 0 claims the
// units, the other producer warps read the ring without freeing entries; the trailing
// cursor (folding) frees them.
struct IssueCursor {
  WarpClaimer c;
  UnitReader r;
  bool claim;  // warp-uniform
  __device__ __forceinline__ int next() { return claim ? c.next() : r.next(); }
};

__device__ __forceinline__ void producer(const GemmArgs& a, double* stages, double* raw, unsigned full0, unsigned empty0,
                                         int pt, const UnitRing& q) {
  const OneJob src{a};
  IssueCursor inx{WarpClaimer{UnitClaimer<OneJob>{src, q}}, UnitReader{q, a.status, false}, pt < 32};
  UnitReader cnx{q, a.status, true};
  LoadIter iss, con;
  load_iter_unit(a, iss, inx);
  load_iter_unit(a, con, cnx);
  // prologue: NRAW - 1 load units in flight
#pragma unroll 1
  for (int i = 0; i < NRAW - 1; ++i) {
    if (iss.valid) {
      issue_unit(a, iss, raw + (size_t)(i % NRAW) * RAW_SZ, pt);
      load_iter_next(a, iss, inx);
    }
    cp_async_commit();
  }
  long long kc = 0;  // operand stages filled so far
  int unit = 0;
#pragma unroll 1
  while (con.valid) {
    const int stage = (int)(kc % NSTAGE);
    double* opA = stages + (size_t)stage * STAGE_SZ;
    double* opB = opA + OPA_SZ;
    if (con.t == 0) mbar_wait(empty0 + 8 * stage, (unsigned)(((kc / NSTAGE) & 1) ^ 1), a.status);
    cp_async_wait<NRAW - 2>();
    fold_unit(con, raw + (size_t)(unit % NRAW) * RAW_SZ, opA, opB, pt);
    const bool last_term = (con.t == con.T - 1);
    if (iss.valid) {
      issue_unit(a, iss, raw + (size_t)((unit + NRAW - 1) % NRAW) * RAW_SZ, pt);
      load_iter_next(a, iss, inx);
    }
    cp_async_commit();
    ++unit;
    if (last_term) {
      __syncwarp();
      if ((pt & 31) == 0) mbar_arrive(full0 + 8 * stage);
      ++kc;
    }
    load_iter_next(a, con, cnx);
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------
// TMA producer.  Warp 0, lane 0 is the issuer: per k step it copies single-term
// operands (coefficient 1, full k step, aligned) straight into the operand stage and
// every term of a summed operand into a raw slot.  Warps 1..7 fold the raw slots of a
// k step into registers (sum with coefficients, k tail masked) and store the result
// into the stage once.  The stage's full barrier completes on the issuer's arrival
// with its byte count plus one arrival per folding warp.
// ------------------------------------------------------------------------------------
struct KStep {
  bool dirA, dirB;  // operand copied straight into the stage
  int T;            // raw loads for the summed operands
};

__device__ __forceinline__ KStep kstep_info(const GemmArgs& a, const LoadIter& it) {
  KStep k;
  const bool whole = (it.s + 1) * BK <= a.ks;
  k.dirA = whole && it.p.na == 1 && it.ta.coef == 1.0;
  k.dirB = whole && it.p.nb == 1 && it.tb.coef == 1.0 && ((it.tb.row * a.ks) & 1) == 0;
  const int tA = k.dirA ? 0 : it.p.na, tB = k.dirB ? 0 : it.p.nb;
  k.T = tA > tB ? tA : tB;
  return k;
}

// Per-k-step iterator over (unit, k step); ta / tb hold the first A / B term.
template <class Nx>
__device__ __forceinline__ void kiter_next(const GemmArgs& a, LoadIter& it, Nx& nx) {
  it.t = 0;
  if (++it.s >= num_ksteps(a)) load_iter_unit(a, it, nx);
}

__device__ __forceinline__ void tma_issuer(const GemmArgs& a, double* stages, double* raw, SlotMeta* meta, unsigned full0,
                                           unsigned empty0, unsigned rfull0, unsigned rempty0, const UnitRing& q) {
  const OneJob src{a};
  UnitClaimer<OneJob> nx{src, q};
  LoadIter it;
  load_iter_unit(a, it, nx);
  long long kc = 0, rc = 0;
#pragma unroll 1
  while (it.valid) {
    const int stage = (int)(kc % NSTAGE);
    double* opA = stages + (size_t)stage * STAGE_SZ;
    const KStep ks = kstep_info(a, it);
    const int k0 = it.s * BK;
    mbar_wait(empty0 + 8 * stage, (unsigned)(((kc / NSTAGE) & 1) ^ 1), a.status);
    const unsigned fb = full0 + 8 * stage;
    mbar_arrive_expect_tx(fb, (ks.dirA ? TMA_BYTES_A : 0u) + (ks.dirB ? TMA_BYTES_B8 : 0u));
    if (ks.dirA)
      tma_load_2d(smem_u32(opA), &a.tmA, it.ta.row * a.ms + it.w.m0, it.ta.col * a.ks + k0, fb);
    if (ks.dirB)
      tma_load_2d(smem_u32(opA + OPA_SZ), &a.tmB, it.tb.row * a.ks + k0, it.tb.col * a.ns + it.w.n0, fb);
#pragma unroll 1
    for (int t = 0; t < ks.T; ++t, ++rc) {
      const int slot = (int)(rc % NRAW_TMA);
      if (rc >= NRAW_TMA) mbar_wait(rempty0 + 8 * slot, (unsigned)(((rc / NRAW_TMA) - 1) & 1), a.status);
      const bool hasA = !ks.dirA && t < it.p.na, hasB = !ks.dirB && t < it.p.nb;
      const unsigned rb = rfull0 + 8 * slot;
      double* rs = raw + (size_t)slot * TRAW_SZ;
      const Term tA = hasA ? (t == 0 ? it.ta : a.terms[it.p.a0 + t]) : Term{0, 0, 0.0, 0, 0};
      const Term tB = hasB ? (t == 0 ? it.tb : a.terms[it.p.b0 + t]) : Term{0, 0, 0.0, 0, 0};
      const int xk = tB.row * a.ks + k0;  // B box k coordinate, rounded down to even: TMA needs 16-byte x
      meta[slot].ca = tA.coef;
      meta[slot].cb = tB.coef;
      meta[slot].shift = xk & 1;
      mbar_arrive_expect_tx(rb, (hasA ? TMA_BYTES_A : 0u) + (hasB ? TMA_BYTES_B : 0u));
      if (hasA)
        tma_load_2d(smem_u32(rs), &a.tmA, tA.row * a.ms + it.w.m0, tA.col * a.ks + k0, rb);
      if (hasB) tma_load_2d(smem_u32(rs + TRAW_A), &a.tmB2, xk & ~1, tB.col * a.ns + it.w.n0, rb);
    }
    ++kc;
    kiter_next(a, it, nx);
  }
  // raw-slot copies still in flight (only on an error path) land before the CTA exits
  for (long long q = rc - NRAW_TMA; q < rc; ++q)
    if (q >= 0) mbar_wait_drain(rfull0 + 8 * (int)(q % NRAW_TMA), (unsigned)((q / NRAW_TMA) & 1));
}

// One raw slot folded into the running sums.  A: element pairs along m (16-byte
// loads, conflict-free); B: single elements with consecutive k per lane, which spreads
// the 80-byte box columns over all banks.  The k tail of a sub-block (k >= ks) only
// exists on a product's last k step and is masked there.
template <bool TAIL>
__device__ __forceinline__ void fold_slot(const double* rs, const SlotMeta& m, bool hasA, bool hasB, bool first,
                                          double2 (&accA)[FPAIRS], double (&accB)[FELEMS], int ft, int kvalid) {
  if (hasA) {
    const double c = m.ca;
#pragma unroll
    for (int e = 0; e < FPAIRS; ++e) {
      const int q = ft + e * NFOLD;
      if (q < BM * BK / 2) {
        const int mm = 2 * (q % (BM / 2)), kk = q / (BM / 2);
        double2 v = reinterpret_cast<const double2*>(rs)[(kk * BM + mm) / 2];
        if (TAIL && kk >= kvalid) v = make_double2(0.0, 0.0);
        accA[e] = first ? make_double2(c * v.x, c * v.y) : make_double2(fma(c, v.x, accA[e].x), fma(c, v.y, accA[e].y));
      }
    }
  }
  if (hasB) {
    const double c = m.cb;
    const double* rb = rs + TRAW_A + m.shift;
#pragma unroll
    for (int e = 0; e < FELEMS; ++e) {
      const int q = ft + e * NFOLD;
      if (q < BN * BK) {
        const int kk = q % BK, nn = q / BK;
        double v = rb[nn * TB_K + kk];
        if (TAIL && kk >= kvalid) v = 0.0;
        accB[e] = first ? c * v : fma(c, v, accB[e]);
      }
    }
  }
}

__device__ __forceinline__ void tma_folder(const GemmArgs& a, double* stages, const double* raw, const SlotMeta* meta,
                                           unsigned full0, unsigned empty0, unsigned rfull0, unsigned rempty0, int ft,
                                           const UnitRing& q) {
  UnitReader nx{q, a.status, true};
  LoadIter it;
  load_iter_unit(a, it, nx);
  long long kc = 0, rc = 0;
  const int lane = ft & 31;
#pragma unroll 1
  while (it.valid) {
    const int stage = (int)(kc % NSTAGE);
    double* opA = stages + (size_t)stage * STAGE_SZ;
    double* opB = opA + OPA_SZ;
    const KStep ks = kstep_info(a, it);
    const int kvalid = a.ks - it.s * BK;  // valid k values in this step (>= BK except at the tail)
    // Every folding warp waits for the stage to be released before it arrives on the
    // stage's full barrier, even when it has nothing to fold: an arrival made earlier
    // could land in the barrier's previous phase (whose issuer arrival and bytes may
    // still be outstanding) and break that phase's transaction accounting.
    mbar_wait(empty0 + 8 * stage, (unsigned)(((kc / NSTAGE) & 1) ^ 1), a.status);
    if (ks.T > 0) {
      double2 accA[FPAIRS];
      double accB[FELEMS];
#pragma unroll 1
      for (int t = 0; t < ks.T; ++t, ++rc) {
        const int slot = (int)(rc % NRAW_TMA);
        mbar_wait(rfull0 + 8 * slot, (unsigned)((rc / NRAW_TMA) & 1), a.status);
        const double* rs = raw + (size_t)slot * TRAW_SZ;
        const bool hasA = !ks.dirA && t < it.p.na, hasB = !ks.dirB && t < it.p.nb;
        if (kvalid >= BK)
          fold_slot<false>(rs, meta[slot], hasA, hasB, t == 0, accA, accB, ft, kvalid);
        else
          fold_slot<true>(rs, meta[slot], hasA, hasB, t == 0, accA, accB, ft, kvalid);
        __threadfence_block();  // raw-slot loads complete before the slot can be refilled
        __syncwarp();
        if (lane == 0) mbar_arrive(rempty0 + 8 * slot);
      }
      if (!ks.dirA) {
#pragma unroll
        for (int e = 0; e < FPAIRS; ++e) {
          const int q = ft + e * NFOLD;
          if (q < BM * BK / 2) {
            const int mm = 2 * (q % (BM / 2)), kk = q / (BM / 2);
            *reinterpret_cast<double2*>(opA + kk * LDA_S + mm) = accA[e];
          }
        }
      }
      if (!ks.dirB) {
#pragma unroll
        for (int e = 0; e < FELEMS; ++e) {
          const int q = ft + e * NFOLD;
          if (q < BN * BK) opB[(q / BK) * LDB_S + q % BK] = accB[e];
        }
      }
      // The stage is written here through the generic proxy and later refilled by TMA
      // (async proxy): order these stores before any later async-proxy access to it.
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(full0 + 8 * stage);
    ++kc;
    kiter_next(a, it, nx);
  }
}

// ------------------------------------------------------------------------------------
// Consumers: DMMA over the stages, then the multi-destination epilogue.
//
// Consumer warp (wm, wn) owns tile rows wm*64 + 16i + 0..15 and tile columns
// frag_col(wn, j) + 0..7 for fragments i, j = 0..3.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ int frag_col(int wn, int j) { return wn * 8 + j * 32; }

// One operand stage into the 64 x 32 warp tile.
__device__ __forceinline__ void mma_stage(const double* opA, const double* opB, double (&acc)[4][4][4], int wm, int wn,
                                          int g, int t4) {
#pragma unroll
  for (int kq = 0; kq < BK / 4; ++kq) {
    double af[4][2], bf[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = wm * 64 + i * 16 + g;
      af[i][0] = opA[(kq * 4 + t4) * LDA_S + row];
      af[i][1] = opA[(kq * 4 + t4) * LDA_S + row + 8];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) bf[j] = opB[(frag_col(wn, j) + g) * LDB_S + kq * 4 + t4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dmma_16x8x4(acc[i][j], af[i], bf[j]);
  }
}

__device__ __forceinline__ void epilogue(const GemmArgs& a, const Prod& p, const double (&acc)[4][4][4],
                                         int m0, int n0, int wm, int wn, int g, int t4) {
  // C_l += w * M_r, 4 * C_BATCH_J elements at a time: all loads of a batch are issued before
  // any store, so a batch costs one memory round trip instead of one per element.
#pragma unroll 1
  for (int c = 0; c < p.nc; ++c) {
    const Term tm = a.terms[p.c0 + c];
    const double w = tm.coef;
    double* Cb = a.C + (long long)tm.row * a.ms + (long long)tm.col * a.ns * a.ldc;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int jb = 0; jb < 4; jb += C_BATCH_J) {
        double cv[C_BATCH_J][4];
#pragma unroll
        for (int j = 0; j < C_BATCH_J; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int rr = m0 + wm * 64 + i * 16 + g + 8 * h;
              const int cc = n0 + frag_col(wn, jb + j) + t4 * 2 + q;
              cv[j][2 * h + q] = (rr < a.ms && cc < a.ns) ? Cb[rr + (long long)cc * a.ldc] : 0.0;
            }
#pragma unroll
        for (int j = 0; j < C_BATCH_J; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int rr = m0 + wm * 64 + i * 16 + g + 8 * h;
              const int cc = n0 + frag_col(wn, jb + j) + t4 * 2 + q;
              if (rr < a.ms && cc < a.ns)
                Cb[rr + (long long)cc * a.ldc] = fma(w, acc[i][jb + j][2 * h + q], cv[j][2 * h + q]);
            }
      }
  }
}

// Pull the C tiles an epilogue will update into L2 while the product's last k steps run.
__device__ __forceinline__ void prefetch_c_tiles(const GemmArgs& a, const Prod& p, int m0, int n0, int ct) {
  for (int c = 0; c < p.nc; ++c) {
    const Term tm = a.terms[p.c0 + c];
    const double* Cb = a.C + (long long)tm.row * a.ms + (long long)tm.col * a.ns * a.ldc;
#pragma unroll
    for (int e = 0; e < (BN * BM / 16) / NCONS; ++e) {  // 128-byte lines: 16 rows of one column
      const int l = ct + e * NCONS;
      const int rr = m0 + (l % (BM / 16)) * 16, cc = n0 + l / (BM / 16);
      if (rr < a.ms && cc < a.ns)
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(Cb + rr + (long long)cc * a.ldc));
    }
  }
}

// Wait until the previous product chunk of this tile has finished its C updates.
__device__ __forceinline__ void ticket_wait(const GemmArgs& a, int tile, int chunk, int ct) {
  if (ct == 0) ticket_spin(a.tickets + tile, chunk, a.status, 256);
  named_bar_sync(1, NCONS);
}

__device__ __forceinline__ void ticket_release(const GemmArgs& a, int tile, int chunk, int ct) {
  __threadfence();
  named_bar_sync(1, NCONS);
  if (ct == 0) st_release(a.tickets + tile, chunk + 1);
}

__device__ __forceinline__ void consumer(const GemmArgs& a, const double* stages, unsigned full0, unsigned empty0,
                                         int ct, const UnitRing& q) {
  const int warp = ct >> 5, lane = ct & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = warp >> 2, wn = warp & 3;
  UnitReader nx{q, a.status, true};
  long long kc = 0;
  double acc[4][4][4];
  const int nks = num_ksteps(a);
  const bool ordered = a.nprod > 1;
#pragma unroll 1
  for (int u = nx.next(); u >= 0; u = nx.next()) {
    const Unit w = decode_unit(a, u);
    const Prod p = a.prods[w.r];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
#pragma unroll 1
    for (int s = 0; s < nks; ++s) {
      const int stage = (int)(kc % NSTAGE);
      const double* opA = stages + (size_t)stage * STAGE_SZ;
      const double* opB = opA + OPA_SZ;
      mbar_wait(full0 + 8 * stage, (unsigned)((kc / NSTAGE) & 1), a.status);
      if (s == (nks > C_PREFETCH_STEPS ? nks - C_PREFETCH_STEPS : 0)) prefetch_c_tiles(a, p, w.m0, w.n0, ct);
      mma_stage(opA, opB, acc, wm, wn, g, t4);
      // The stage is refilled by TMA as soon as every warp has arrived; the fence
      // makes this warp's shared-memory fragment loads complete before its arrival
      // (measured: without it a refill could overwrite fragments still in flight).
      __threadfence_block();
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + 8 * stage);
      ++kc;
    }
    if (ordered) ticket_wait(a, w.tile, w.r, ct);
    epilogue(a, p, acc, w.m0, w.n0, wm, wn, g, t4);
    if (ordered) ticket_release(a, w.tile, w.r, ct);
  }
}

// Persistent: one CTA per SM takes work units in claim order (UnitClaimer) until none is left.
// TMA = true stages operands with tensor copies (A, B 16-byte aligned, even leading
// dimensions); TMA = false with per-thread cp.async (any alignment).
template <bool TMA>
__global__ void __launch_bounds__(NTHREADS, 1) fmm_gemm_kernel(const __grid_constant__ GemmArgs a) {
  extern __shared__ __align__(128) double smem[];
  double* stages = smem;                                  // [NSTAGE][STAGE_SZ]
  double* raw = stages + (size_t)NSTAGE * STAGE_SZ;       // [NRAW][RAW_SZ] or [NRAW_TMA][TRAW_SZ]
  SlotMeta* meta = reinterpret_cast<SlotMeta*>(raw + (TMA ? (size_t)NRAW_TMA * TRAW_SZ : (size_t)NRAW * RAW_SZ));
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(meta + (TMA ? NRAW_TMA : 0));
  const unsigned full0 = smem_u32(bars);
  const unsigned empty0 = smem_u32(bars + NSTAGE);
  const unsigned rfull0 = smem_u32(bars + 2 * NSTAGE);
  const unsigned rempty0 = smem_u32(bars + 2 * NSTAGE + NRAW_TMA);
  const UnitRing q{smem_u32(bars + 2 * NSTAGE + 2 * NRAW_TMA)};
  const int tid = threadIdx.x;
  if (tid == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      // full: TMA path = issuer (1) + folding warps; cp.async path = the 4 producer warps
      mbar_init(full0 + 8 * s, TMA ? 1 + NFOLD / 32 : NPROD / 32);
      mbar_init(empty0 + 8 * s, NCONS / 32);
    }
    if (TMA) {
      for (int s = 0; s < NRAW_TMA; ++s) {
        mbar_init(rfull0 + 8 * s, 1);
        mbar_init(rempty0 + 8 * s, NFOLD / 32);
      }
    }
    // ring readers: folding + consumer warps (TMA); every producer and consumer warp (cp.async)
    unit_ring_init(q, TMA ? (NFOLD + NCONS) / 32 : (NPROD + NCONS) / 32);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (tid < NPROD) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(PROD_REGS));
    if (TMA) {
      if (tid == 0)
        tma_issuer(a, stages, raw, meta, full0, empty0, rfull0, rempty0, q);
      else if (tid >= 32)
        tma_folder(a, stages, raw, meta, full0, empty0, rfull0, rempty0, tid - 32, q);
    } else {
      producer(a, stages, raw, full0, empty0, tid, q);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(CONS_REGS));
    consumer(a, stages, full0, empty0, tid - NPROD, q);
  }
}

// Operand sums in HBM: slot j = sum_t coef_t * X_{blk_t} over the A (or B) terms of product
// plist[j], the slot's k extent rounded up with zeros.  HBM bound: every input element once,
// every slot element once; an input element feeds nnz(U) / blocks sums (15 for 222-1 x 333-1),
// which come from L1 and L2.  A CTA takes chunks of element positions (a row pair a thread) and
// walks all its outputs for each, so that the blocks' values at those positions stay close;
// the terms' offsets and coefficients and the outputs' places among them are in shared
// memory, made once per CTA.  For calls of less than a chunk per SM and plans whose blocks or terms do not fit
// the staged kernel below.  Measured on B200 at four CTAs per SM (the registers' limit) against
// one chunk per CTA, tables per chunk and masked groups of four terms: 222-1 2048^3 50 -> 39 us,
// 8192^3 644 -> 455 us; 222-2 8192^3 1050 -> 936 us; 222-1 x 333-1 16384^3 8.0 -> 7.7 ms.  One to
// three CTAs per SM, whose positions would fit L1, took 1.1 to 2.3 times as long, two
// positions per thread 1.1 to 1.3 times on plans of many blocks.
struct PTerm {
  int row, col;  // block
  double coef;
};

struct PresumSide {
  const double* X;
  long long ldx;
  int rows, cols;          // block size
  int orows, ocols;        // slot size (orows even)
  int blk_row_stride;      // rows per block row (ms for A, ks for B)
  int blk_col_stride;      // cols per block column (ks for A, ns for B)
  double* out;
  long long ldo;           // even
  long long out_stride;
  const int* plist;        // product of each output; nullptr = output j is product j
  const int* first;        // per product its first term (R + 1 entries)
  const PTerm* terms;
  int nout;
  int brows, bcols;        // block grid of the operand (fmm_presum_staged_kernel)
  int pad;
};

constexpr int PS_THREADS = 256;
constexpr int PS_TERMS = 2048;  // terms of one pass over the outputs (32 KB of shared memory at most)
constexpr int PS_OUTS = 512;    // outputs of one pass

struct PresumOff {
  long long off;
  double coef;
};
__host__ __device__ constexpr size_t presum_smem_bytes(int cap) {
  return sizeof(PresumOff) * (size_t)cap + sizeof(int2) * PS_OUTS;
}

__device__ __forceinline__ PresumOff presum_term(const PresumSide& a, const PTerm& t) {
  return PresumOff{(long long)t.row * a.blk_row_stride + (long long)t.col * a.blk_col_stride * a.ldx, t.coef};
}

// A thread's position: rows i, i + 1 of a column; v0, v1: inside the block.
struct PresumPos {
  const double* x;
  bool v0, v1;
};

// Ordinary loads: these kernels may start while the operand's last writer (C of the call before) still
// runs, which loads for read-only memory do not allow.
template <bool VEC>
__device__ __forceinline__ double2 presum_load(const PresumPos& p, long long off) {
  double2 x = make_double2(0.0, 0.0);
  if (VEC) {
    if (p.v1) x = __ldca(reinterpret_cast<const double2*>(p.x + off));
  } else {
    if (p.v0) x.x = __ldca(p.x + off);
    if (p.v1) x.y = __ldca(p.x + off + 1);
  }
  return x;
}

// v += N terms in order, all their loads issued first.
template <bool VEC, int N, class Tm>
__device__ __forceinline__ void presum_add(const PresumPos& p, Tm&& term, int t, double2& v) {
  PresumOff o[N];
  double2 x[N];
#pragma unroll
  for (int q = 0; q < N; ++q) o[q] = term(t + q);
#pragma unroll
  for (int q = 0; q < N; ++q) x[q] = presum_load<VEC>(p, o[q].off);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    v.x = fma(o[q].coef, x[q].x, v.x);
    v.y = fma(o[q].coef, x[q].y, v.y);
  }
}

template <bool VEC, class Tm>
__device__ __forceinline__ double2 presum_sum(const PresumPos& p, int n, Tm&& term) {
  double2 v = make_double2(0.0, 0.0);
  int t = 0;
#pragma unroll 1
  for (; t + 4 <= n; t += 4) presum_add<VEC, 4>(p, term, t, v);
  switch (n - t) {
    case 1: presum_add<VEC, 1>(p, term, t, v); break;
    case 2: presum_add<VEC, 2>(p, term, t, v); break;
    case 3: presum_add<VEC, 3>(p, term, t, v); break;
    default: break;
  }
  return v;
}

__device__ __forceinline__ long long presum_chunks(const PresumSide& a) {
  return ((long long)(a.orows / 2) * a.ocols + PS_THREADS - 1) / PS_THREADS;
}

// Outputs [j, je) (their terms in the table, or with tab == nullptr one output from global
// memory) at the positions of chunks c0, c0 + cstep, ...
template <bool VEC>
__device__ __forceinline__ void presum_chunk_loop(const PresumSide& a, const PresumOff* tab, const int2* dsc, int j, int je,
                                                  const PTerm* tg, int ntg, long long c0, long long cstep) {
  const int hr = a.orows / 2;
  const long long nc = presum_chunks(a);
  for (long long ch = c0; ch < nc; ch += cstep) {
    const long long e = ch * PS_THREADS + threadIdx.x;
    if (e >= (long long)hr * a.ocols) continue;
    const long long c = e / hr;
    const int i = 2 * (int)(e - c * hr);
    const bool in = c < a.cols;
    const PresumPos p{a.X + i + c * a.ldx, in && i < a.rows, in && i + 1 < a.rows};
    double* o = a.out + i + c * a.ldo + j * a.out_stride;
    if (!tab) {
      *reinterpret_cast<double2*>(o) = presum_sum<false>(p, ntg, [&](int t) { return presum_term(a, tg[t]); });
      continue;
    }
#pragma unroll 1
    for (int q = 0; q < je - j; ++q, o += a.out_stride) {
      const int2 d = dsc[q];
      const PresumOff* tp = tab + d.x;
      *reinterpret_cast<double2*>(o) = presum_sum<VEC>(p, d.y, [&](int t) { return tp[t]; });
    }
  }
}

// Outputs [j0, j1) of one side at the position chunks c0, c0 + cstep, ...
__device__ __forceinline__ void presum_side(const PresumSide& a, PresumOff* tab, int cap, int j0, int j1, long long c0,
                                            long long cstep) {
  int2* dsc = reinterpret_cast<int2*>(tab + cap);  // per output of a pass: first term in the table, terms
  // pairs are 16-byte aligned and whole: even strides, base aligned, even row count
  const bool vec = ((reinterpret_cast<uintptr_t>(a.X) & 15) == 0) && ((a.ldx | a.blk_row_stride | a.rows) & 1) == 0;
  auto prod = [&](int j) { return a.plist ? __ldg(a.plist + j) : j; };
  for (int j = j0; j < j1;) {
    // as many outputs as the tables hold (usually all of them)
    const int t0 = __ldg(a.first + prod(j));
    int je = min(j1, j + PS_OUTS);
    if (__ldg(a.first + prod(je - 1) + 1) - t0 > cap) {
      const int lim = je;
      je = j;
      while (je < lim && __ldg(a.first + prod(je) + 1) - t0 <= cap) ++je;
    }
    if (je == j) {  // one output with more terms than the table
      presum_chunk_loop<false>(a, nullptr, nullptr, j, j + 1, a.terms + t0, __ldg(a.first + prod(j) + 1) - t0, c0, cstep);
      ++j;
      continue;
    }
    const int nt = __ldg(a.first + prod(je - 1) + 1) - t0;
    __syncthreads();
    for (int t = threadIdx.x; t < nt; t += PS_THREADS) tab[t] = presum_term(a, a.terms[t0 + t]);
    for (int q = threadIdx.x; q < je - j; q += PS_THREADS) {
      const int r = prod(j + q), f = __ldg(a.first + r);
      dsc[q] = make_int2(f - t0, __ldg(a.first + r + 1) - f);
    }
    __syncthreads();
    if (vec)
      presum_chunk_loop<true>(a, tab, dsc, j, je, nullptr, 0, c0, cstep);
    else
      presum_chunk_loop<false>(a, tab, dsc, j, je, nullptr, 0, c0, cstep);
    j = je;
  }
}

// Both sides of one call: CTA x takes chunks x, x + grid, ... of A's and then B's positions,
// output range blockIdx.y of each.  Also zeroes the products launch's tickets and work-unit
// counter (zero[0 .. nzero)).
struct PresumArgs {
  PresumSide s[2];
  int* zero;
  int nzero;
  int cap;  // terms the dynamic shared memory holds
};

__global__ void __launch_bounds__(PS_THREADS) fmm_presum_kernel(const __grid_constant__ PresumArgs g) {
  extern __shared__ __align__(16) PresumOff ptab[];
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (blockIdx.y == 0)
    for (long long q = (long long)blockIdx.x * PS_THREADS + threadIdx.x; q < g.nzero; q += (long long)gridDim.x * PS_THREADS)
      g.zero[q] = 0;
  long long c0 = blockIdx.x;
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    const PresumSide& a = g.s[s];
    if (a.nout == 0) continue;
    const int j0 = (int)((long long)a.nout * blockIdx.y / gridDim.y), j1 = (int)((long long)a.nout * (blockIdx.y + 1) / gridDim.y);
    const long long nc = presum_chunks(a);
    if (j0 < j1 && c0 < nc) presum_side(a, ptab, g.cap, j0, j1, c0, gridDim.x);
    // go on where this side's round robin ended
    c0 = (c0 + gridDim.x - nc % gridDim.x) % gridDim.x;
  }
}

// The same sums with the operand's blocks staged in shared memory: a thread copies its pair of
// positions of every block (cp.async, slots of its own, so that no barrier is needed) and then
// walks one flat list of all terms, which marks where a sum begins and where it is stored.  A
// gather of the kernel above is an L1 or L2 access, and of many blocks' values few are still in
// L1 (222-1 x 333-1: 540 terms of 36 blocks a side).  Bound by HBM where blocks are few (222-2 8192^3
// 5.9 TB/s), at 36 blocks by the latency of the shared memory reads that 256 threads an SM can
// hide: reading ahead over the sums' ends is what a list gives over a loop per sum (16384^3 6.0
// against 7.7 ms), and two CTAs as the launch bound leave ptxas the registers for it (40 registers:
// 6.8 ms).  Same additions in the same order.  Measured on B200 against the gathers: 222-1
// 2048^3 39 -> 35 us, 8192^3 454 -> 404; 222-2 3600 x 4200 x 2900 (odd blocks: 8-byte copies) 194 -> 144,
// 8192^3 935 -> 750; 222-1 x 333-1 2016^3 127 -> 84, 14400^2 x 480 210 -> 146, 16384^3 7.7 -> 6.0 ms.
constexpr int PSS_THREADS = 128;
constexpr int PSS_UNROLL = 8;
struct PresumOp {
  unsigned off;    // of the term's block in a thread's slots
  unsigned flags;  // PSS_FIRST, PSS_STORE
  double coef;
};
constexpr unsigned PSS_FIRST = 1, PSS_STORE = 2;
__host__ __device__ constexpr size_t presum_staged_smem(int nblk, int cap) {
  return (size_t)nblk * PSS_THREADS * 16 + sizeof(PresumOp) * (size_t)(cap + PSS_UNROLL);
}

__global__ void __launch_bounds__(PSS_THREADS, 2) fmm_presum_staged_kernel(const __grid_constant__ PresumArgs g) {
  extern __shared__ __align__(16) unsigned char pss[];
  const int tid = threadIdx.x;
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (blockIdx.y == 0)
    for (long long q = (long long)blockIdx.x * PSS_THREADS + tid; q < g.nzero; q += (long long)gridDim.x * PSS_THREADS)
      g.zero[q] = 0;
  long long c0 = blockIdx.x;
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    const PresumSide& a = g.s[s];
    if (a.nout == 0) continue;
    const int hr = a.orows / 2;
    const long long total = (long long)hr * a.ocols, nc = (total + PSS_THREADS - 1) / PSS_THREADS;
    const int j0 = (int)((long long)a.nout * blockIdx.y / gridDim.y), j1 = (int)((long long)a.nout * (blockIdx.y + 1) / gridDim.y);
    if (j0 < j1 && c0 < nc) {
      // the terms of products r0 .. r1 in one list: a term of coefficient 0 pads it to whole steps, and
      // products without a slot are summed and not stored
      PresumOp* ops = reinterpret_cast<PresumOp*>(pss + (size_t)a.brows * a.bcols * PSS_THREADS * 16);
      const int r0 = a.plist ? __ldg(a.plist + j0) : j0, r1 = a.plist ? __ldg(a.plist + j1 - 1) : j1 - 1;
      const int t0 = __ldg(a.first + r0), nt = __ldg(a.first + r1 + 1) - t0;
      const int ntp = (nt + PSS_UNROLL - 1) / PSS_UNROLL * PSS_UNROLL;
      __syncthreads();  // the other side's list is no longer read
      for (int t = tid; t < ntp; t += PSS_THREADS) {
        PresumOp op{0u, PSS_FIRST, 0.0};
        if (t < nt) {
          const PTerm tm = a.terms[t0 + t];
          op = PresumOp{(unsigned)(tm.row * a.bcols + tm.col) * (PSS_THREADS * 16), 0u, tm.coef};
        }
        ops[t] = op;
      }
      __syncthreads();
      for (int r = r0 + tid; r <= r1; r += PSS_THREADS)
        if (__ldg(a.first + r) - t0 < nt) ops[__ldg(a.first + r) - t0].flags = PSS_FIRST;
      __syncthreads();
      for (int q = j0 + tid; q < j1; q += PSS_THREADS)
        ops[__ldg(a.first + (a.plist ? __ldg(a.plist + q) : q) + 1) - 1 - t0].flags |= PSS_STORE;
      __syncthreads();
      const unsigned char* mine = pss + tid * 16;
      // pairs are 16-byte aligned and whole: even strides, base aligned, even row count
      const bool vec = ((reinterpret_cast<uintptr_t>(a.X) & 15) == 0) && ((a.ldx | a.blk_row_stride | a.rows) & 1) == 0;
      for (long long ch = c0; ch < nc; ch += gridDim.x) {
        const long long e = ch * PSS_THREADS + tid;
        if (e >= total) continue;
        const long long c = e / hr;
        const int i = 2 * (int)(e - c * hr);
        const bool v0 = c < a.cols && i < a.rows, v1 = c < a.cols && i + 1 < a.rows;
        const double* x = a.X + (v0 ? i + c * a.ldx : 0);  // what is not copied still names an address
        unsigned dst = smem_u32(mine);
        for (int br = 0; br < a.brows; ++br)
          for (int bc = 0; bc < a.bcols; ++bc, dst += PSS_THREADS * 16) {
            const double* xb = v0 ? x + (long long)br * a.blk_row_stride + (long long)bc * a.blk_col_stride * a.ldx : x;
            if (vec) {
              cp_async16(dst, xb, v1 ? 16 : 0);
            } else {
              cp_async8(dst, xb, v0 ? 8 : 0);
              cp_async8(dst + 8, v1 ? xb + 1 : xb, v1 ? 8 : 0);
            }
          }
        cp_async_commit();
        cp_async_wait<0>();
        double* o = a.out + i + c * a.ldo + j0 * a.out_stride;
        double2 v = make_double2(0.0, 0.0);
#pragma unroll 1
        for (int t = 0; t < ntp; t += PSS_UNROLL) {
          PresumOp op[PSS_UNROLL];
          double2 xv[PSS_UNROLL];
#pragma unroll
          for (int q = 0; q < PSS_UNROLL; ++q) op[q] = ops[t + q];
#pragma unroll
          for (int q = 0; q < PSS_UNROLL; ++q) xv[q] = *reinterpret_cast<const double2*>(mine + op[q].off);
#pragma unroll
          for (int q = 0; q < PSS_UNROLL; ++q) {
            if (op[q].flags & PSS_FIRST) v = make_double2(0.0, 0.0);
            v.x = fma(op[q].coef, xv[q].x, v.x);
            v.y = fma(op[q].coef, xv[q].y, v.y);
            if (op[q].flags & PSS_STORE) {
              *reinterpret_cast<double2*>(o) = v;
              o += a.out_stride;
            }
          }
        }
      }
    }
    // go on where this side's round robin ended
    c0 = (c0 + gridDim.x - nc % gridDim.x) % gridDim.x;
  }
}

// The operand sums of many problems in one launch (task blockIdx.z).
__global__ void __launch_bounds__(PS_THREADS) fmm_presum_batch_kernel(const PresumSide* tasks, int cap) {
  extern __shared__ __align__(16) PresumOff ptab[];
  const PresumSide a = tasks[blockIdx.z];
  const int j0 = (int)((long long)a.nout * blockIdx.y / gridDim.y), j1 = (int)((long long)a.nout * (blockIdx.y + 1) / gridDim.y);
  if (j0 < j1 && blockIdx.x < presum_chunks(a)) presum_side(a, ptab, cap, j0, j1, blockIdx.x, gridDim.x);
}

// Column-major copies between pitches, many in one launch (task blockIdx.y): used to give
// operands with an odd leading dimension the even pitch (16-byte column starts) that
// tensor-memory-access staging needs.
struct PitchCopy {
  const double* src;
  long long lds;
  double* dst;
  long long ldd;
  int rows, cols;
};

__device__ __forceinline__ void pitch_copy_body(const PitchCopy& t) {
  for (int j = blockIdx.x; j < t.cols; j += gridDim.x) {
    const double* s = t.src + (long long)j * t.lds;
    double* d = t.dst + (long long)j * t.ldd;
    for (int i = threadIdx.x; i < t.rows; i += blockDim.x) d[i] = s[i];
  }
}

__global__ void fmm_pitch_copy_kernel(const PitchCopy* tasks) { pitch_copy_body(tasks[blockIdx.y]); }
__global__ void fmm_pitch_copy1_kernel(const PitchCopy t) { pitch_copy_body(t); }

// C_l += sum_r W[l, r] * M_r for every C block, the blocks in groups of up to COMBINE_GROUP: a
// thread owns P element positions and walks the groups; for a group it keeps the running values of
// its member blocks in registers, walks the union of their products in increasing r (one
// load of M_r per position, COMBINE_G_BATCH loads in flight) and applies M_r to every member
// whose W[l, r] is nonzero, c_l = fma(W[l, r], M_r, c_l).  Each block still gets exactly the
// epilogue's fma sequence (products in increasing r), so the result is bit-identical to the
// direct schedule.  The host groups blocks that share products (greedy by overlap), which
// cuts the M loads per position from nnz(W) toward R (222-1 x 333-1: 540 -> 299 in 5
// groups) with no shared-memory read-modify-write.  Tables (shared memory, per CTA):
//   group g: gdesc[g * GDESC + 0..4] = first entry, #entries, #members, first chunk, first
//            operation; gdesc[g * GDESC + GD_MEMBERS + q] = block id of member q (row * grid_n + col)
//   entry e: er[e] = product r, em[e] = member mask | (first coefficient of e) << 8,
//            the coefficients of its set bits, member order, from ec[first coefficient]
constexpr int COMBINE_GROUP = 8;
constexpr int GD_MEMBERS = 5;
constexpr int GDESC = GD_MEMBERS + COMBINE_GROUP;
constexpr int COMBINE_G_THREADS = 256;
constexpr int COMBINE_G_BATCH = 16;

struct CombineGroupArgs {
  double* C;
  long long ldc;
  int ms, ns;
  const double* M;
  long long ldm;
  long long m_stride;
  int grid_n;
  int ngroup, nent, ncoef;
  const int* gdesc;
  const int* er;
  const int* em;
  const double* ec;
  int nprod;  // products (slabs of M)
  // staged kernel: the entries of each group in chunks of CST_CHUNK
  int nchunk, nop;
  const int* chr;                 // [nchunk][CST_CHUNK] products (past a group's end: its last)
  const unsigned long long* chn;  // [nchunk] byte q: operations on member q
  const struct CombineOp* op;     // the operations in the order they run: per chunk, per member
};

// c_member += coef * M of the chunk's slot at byte offset `off` of the stage.
struct CombineOp {
  double coef;
  int off;
  int pad;
};

__host__ __device__ constexpr size_t combine_group_smem_bytes(int ngroup, int nent, int ncoef) {
  return sizeof(double) * (size_t)ncoef + sizeof(int) * (2 * (size_t)nent + (size_t)GDESC * ngroup) + 16;
}

template <int P>
__global__ void __launch_bounds__(COMBINE_G_THREADS) fmm_combine_kernel(const CombineGroupArgs a) {
  extern __shared__ __align__(16) double gtab[];
  double* sc = gtab;                               // [ncoef]
  int* sr = reinterpret_cast<int*>(sc + a.ncoef);  // [nent]
  int* sm = sr + a.nent;                           // [nent]
  int* sg = sm + a.nent;                           // [GDESC * ngroup]
  for (int q = threadIdx.x; q < a.ncoef; q += blockDim.x) sc[q] = a.ec[q];
  for (int q = threadIdx.x; q < a.nent; q += blockDim.x) {
    sr[q] = a.er[q];
    sm[q] = a.em[q];
  }
  for (int q = threadIdx.x; q < GDESC * a.ngroup; q += blockDim.x) sg[q] = a.gdesc[q];
  __syncthreads();
  const int nt = blockDim.x;
  const long long total = (long long)a.ms * a.ns;
  for (long long e0 = (long long)blockIdx.x * nt * P; e0 < total; e0 += (long long)gridDim.x * nt * P) {
    // position p of this thread: e0 + threadIdx.x + p * nt (clamped to the last one, whose
    // stores then repeat the same values)
    long long cofs[P], mofs[P];
    bool live[P];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const long long e = e0 + threadIdx.x + (long long)p * nt;
      live[p] = e < total;
      const long long ee = live[p] ? e : total - 1;
      const int i = (int)(ee % a.ms);
      const long long j = ee / a.ms;
      cofs[p] = i + j * a.ldc;
      mofs[p] = i + j * a.ldm;
    }
    if (!live[0]) continue;
#pragma unroll 1
    for (int g = 0; g < a.ngroup; ++g) {
      const int* gd = sg + g * GDESC;
      const int ef = gd[0], ne = gd[1], nm = gd[2];
      double c[COMBINE_GROUP][P];
      long long cb[COMBINE_GROUP];
#pragma unroll
      for (int q = 0; q < COMBINE_GROUP; ++q) {
        const int b = gd[GD_MEMBERS + (q < nm ? q : 0)];
        cb[q] = (long long)(b / a.grid_n) * a.ms + (long long)(b % a.grid_n) * a.ns * a.ldc;
#pragma unroll
        for (int p = 0; p < P; ++p) c[q][p] = q < nm ? a.C[cb[q] + cofs[p]] : 0.0;
      }
#pragma unroll 1
      for (int q0 = 0; q0 < ne; q0 += COMBINE_G_BATCH) {
        double mv[COMBINE_G_BATCH][P];
#pragma unroll
        for (int t = 0; t < COMBINE_G_BATCH; ++t) {
          const long long mo = (long long)sr[ef + min(q0 + t, ne - 1)] * a.m_stride;
#pragma unroll
          for (int p = 0; p < P; ++p) mv[t][p] = __ldcg(a.M + mo + mofs[p]);
        }
#pragma unroll
        for (int t = 0; t < COMBINE_G_BATCH; ++t) {
          if (q0 + t >= ne) break;
          const int mk = sm[ef + q0 + t];
          int k = mk >> 8;
#pragma unroll
          for (int q = 0; q < COMBINE_GROUP; ++q)
            if (mk & (1 << q)) {
              const double w = sc[k++];
#pragma unroll
              for (int p = 0; p < P; ++p) c[q][p] = fma(w, mv[t][p], c[q][p]);
            }
        }
      }
#pragma unroll
      for (int q = 0; q < COMBINE_GROUP; ++q)
        if (q < nm) {
#pragma unroll
          for (int p = 0; p < P; ++p)
            if (live[p]) a.C[cb[q] + cofs[p]] = c[q][p];
        }
    }
  }
}

// The same combine with the M values staged in shared memory by bulk copies: a tile of
// CST_TILE consecutive element positions (M_r[e0 .. e0 + CST_TILE) is contiguous when
// ldm == ms) and a group at a time, CST_CHUNK products per step; a
// producer warp copies each chunk's M_r tiles (cp.async.bulk, 2 KB each) into a ring of
// CST_STAGES stages while the compute warps apply earlier chunks.  HBM bound: every M_r and C
// element once, and the M_r tiles a later group reads again that have left L2 by then (222-1 x
// 333-1: 1.3 x the algorithmic bytes; C goes past L2 with streaming hints so that fewer do).  A
// compute thread owns two positions (16-byte loads) and keeps its group's running C values in
// registers; what to do with a chunk is a list of operations per member in shared memory, so
// an update of two values costs two loads, two FMAs and the loop.  The arithmetic per block is
// the register kernel's (bit-identical).  Measured on B200 against one position per thread
// with bit masks walked per chunk: 222-1 x 333-1 14400^2 x 480 2.65 -> 2.23 ms, 222-2 8192^3
// split 0.58 -> 0.49 ms; fewer or single-position warps, a software pipeline over the
// operations and loading the next group's C ahead were slower or the same.  Where tiles are
// fewer than the CTAs of the chip each group is a unit of its own (528^3 42 -> 21 us); at
// 14400^2 x 480 that takes 2.47 ms.
// Waits are bounded (status word on timeout).
constexpr int CST_THREADS = 128;  // compute threads, two positions each
constexpr int CST_TILE = 2 * CST_THREADS;
constexpr int CST_CHUNK = 8;      // products per stage
constexpr int CST_STAGES = 3;     // 48 KB of stages: three CTAs per SM
constexpr size_t CST_STAGE_DOUBLES = (size_t)CST_CHUNK * CST_TILE;

__host__ __device__ constexpr size_t combine_staged_smem_bytes(int ngroup, int nchunk, int nop) {
  return sizeof(double) * CST_STAGE_DOUBLES * CST_STAGES + 16 * CST_STAGES + sizeof(CombineOp) * (size_t)nop +
         (sizeof(unsigned long long) + sizeof(int) * CST_CHUNK) * (size_t)nchunk +
         (sizeof(long long) * COMBINE_GROUP + sizeof(int) * GDESC) * (size_t)ngroup + 16;
}

__device__ __forceinline__ void bulk_load_1d(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Two consecutive C values of every member of a group at element offset cofs.
__device__ __forceinline__ void combine_load(const CombineGroupArgs& a, const long long* off, int nm, long long cofs,
                                             bool live, bool vec, double2 (&c)[COMBINE_GROUP]) {
#pragma unroll
  for (int q = 0; q < COMBINE_GROUP; ++q) {
    c[q] = make_double2(0.0, 0.0);
    if (q < nm && live) {
      const double* p = a.C + off[q] + cofs;
      if (vec) {
        c[q] = __ldcs(reinterpret_cast<const double2*>(p));
      } else {
        c[q].x = __ldcs(p);
        c[q].y = __ldcs(p + 1);
      }
    }
  }
}

// CombineGroupArgs plus the status word; requires ldm == ms, M and m_stride 16-byte
// multiples (in doubles: m_stride even) and ms even (pairs of positions lie in one column, and
// every tile's byte count is a multiple of 16).
template <bool SPLIT>
__global__ void __launch_bounds__(CST_THREADS + 32, 3) fmm_combine_staged_kernel(const CombineGroupArgs a,
                                                                                 unsigned* status) {
  extern __shared__ __align__(128) double cst[];
  double* stages = cst;                                                    // [STAGES][CHUNK][TILE]
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(stages + CST_STAGE_DOUBLES * CST_STAGES);
  CombineOp* sop = reinterpret_cast<CombineOp*>(bars + 2 * CST_STAGES);    // [nop]
  unsigned long long* scn = reinterpret_cast<unsigned long long*>(sop + a.nop);  // [nchunk]
  long long* sgo = reinterpret_cast<long long*>(scn + a.nchunk);           // [ngroup][GROUP] block offsets in C
  int* sr = reinterpret_cast<int*>(sgo + (size_t)a.ngroup * COMBINE_GROUP);  // [nchunk][CHUNK]
  int* sg = sr + (size_t)a.nchunk * CST_CHUNK;                             // [GDESC * ngroup]
  const unsigned full0 = smem_u32(bars), empty0 = smem_u32(bars + CST_STAGES);
  const int tid = threadIdx.x;
  for (int q = tid; q < a.nop; q += blockDim.x) sop[q] = a.op[q];
  for (int q = tid; q < a.nchunk; q += blockDim.x) scn[q] = a.chn[q];
  for (int q = tid; q < a.nchunk * CST_CHUNK; q += blockDim.x) sr[q] = a.chr[q];
  for (int q = tid; q < GDESC * a.ngroup; q += blockDim.x) sg[q] = a.gdesc[q];
  for (int q = tid; q < COMBINE_GROUP * a.ngroup; q += blockDim.x) {
    const int b = a.gdesc[(q / COMBINE_GROUP) * GDESC + GD_MEMBERS + q % COMBINE_GROUP];
    sgo[q] = (long long)(b / a.grid_n) * a.ms + (long long)(b % a.grid_n) * a.ns * a.ldc;
  }
  if (tid == 0) {
    for (int s = 0; s < CST_STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, CST_THREADS / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;\n" ::: "memory");  // the products (the tables above never change)
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  const long long total = (long long)a.ms * a.ns;
  const long long nunit = (total + CST_TILE - 1) / CST_TILE * (SPLIT ? a.ngroup : 1);
  long long k = 0;  // stage step of this CTA
  if (tid >= CST_THREADS) {  // producer warp: lane 0 issues the copies
    if (tid != CST_THREADS) return;
    for (long long u = blockIdx.x; u < nunit; u += gridDim.x) {
      const long long t = SPLIT ? u / a.ngroup : u, e0 = t * CST_TILE;
      const unsigned bytes = (unsigned)(8 * min((long long)CST_TILE, total - e0));
      const int g0 = SPLIT ? (int)(u - t * a.ngroup) : 0, g1 = SPLIT ? g0 + 1 : a.ngroup;
      for (int g = g0; g < g1; ++g) {
        const int ne = sg[g * GDESC + 1], c0 = sg[g * GDESC + 3];
        for (int q0 = 0; q0 < ne; q0 += CST_CHUNK, ++k) {
          const int s = (int)(k % CST_STAGES);
          mbar_wait(empty0 + 8 * s, (unsigned)(((k / CST_STAGES) & 1) ^ 1), status);
          const int nq = min(CST_CHUNK, ne - q0);
          const int* rr = sr + (size_t)(c0 + q0 / CST_CHUNK) * CST_CHUNK;
          mbar_arrive_expect_tx(full0 + 8 * s, bytes * nq);
          for (int q = 0; q < nq; ++q) {
            int r = rr[q];
            if ((unsigned)r >= (unsigned)a.nprod) {  // never with host-checked tables
              atomicOr(status, STATUS_TABLE);
              r = 0;
            }
            bulk_load_1d(smem_u32(stages + (size_t)s * CST_STAGE_DOUBLES + (size_t)q * CST_TILE),
                         a.M + (long long)r * a.m_stride + e0, bytes, full0 + 8 * s);
          }
        }
      }
    }
    // copies still in flight (only on an error path) land before the CTA exits
    for (long long q = k - CST_STAGES; q < k; ++q)
      if (q >= 0) mbar_wait_drain(full0 + 8 * (int)(q % CST_STAGES), (unsigned)((q / CST_STAGES) & 1));
    return;
  }
  const int lane = tid & 31;
  const bool vec = ((reinterpret_cast<uintptr_t>(a.C) & 15) == 0) && (a.ldc & 1) == 0;
  double2 c[COMBINE_GROUP];
  for (long long u = blockIdx.x; u < nunit; u += gridDim.x) {
    const long long t = SPLIT ? u / a.ngroup : u, e = t * CST_TILE + 2 * tid;  // this thread's pair of positions
    const bool live = e < total;
    const long long ee = live ? e : 0;
    const long long cofs = (ee % a.ms) + (ee / a.ms) * a.ldc;  // element offset in a C block
    const int g0 = SPLIT ? (int)(u - t * a.ngroup) : 0, g1 = SPLIT ? g0 + 1 : a.ngroup;
    const CombineOp* op = sop + sg[g0 * GDESC + 4];  // runs on from group to group
    for (int g = g0; g < g1; ++g) {
      const int* gd = sg + g * GDESC;
      const int ne = gd[1], nm = gd[2], c0 = gd[3];
      combine_load(a, sgo + g * COMBINE_GROUP, nm, cofs, live, vec, c);
      for (int q0 = 0; q0 < ne; q0 += CST_CHUNK, ++k) {
        const int s = (int)(k % CST_STAGES);
        const unsigned long long cnt = scn[c0 + q0 / CST_CHUNK];
        mbar_wait(full0 + 8 * s, (unsigned)((k / CST_STAGES) & 1), status);
        const unsigned char* st = reinterpret_cast<const unsigned char*>(stages + (size_t)s * CST_STAGE_DOUBLES) + 16 * tid;
#pragma unroll
        for (int b = 0; b < COMBINE_GROUP; ++b) {
          const int n = (int)(cnt >> (8 * b)) & 0xff;
#pragma unroll 2
          for (int i = 0; i < n; ++i) {
            const CombineOp o = op[i];
            const double2 m = *reinterpret_cast<const double2*>(st + o.off);
            c[b].x = fma(o.coef, m.x, c[b].x);
            c[b].y = fma(o.coef, m.y, c[b].y);
          }
          op += n;
        }
        __threadfence_block();  // the stage's loads complete before it can be refilled
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * s);
      }
      if (live) {
#pragma unroll
        for (int q = 0; q < COMBINE_GROUP; ++q)
          if (q < nm) {
            double* p = a.C + sgo[g * COMBINE_GROUP + q] + cofs;
            if (vec) {
              __stcs(reinterpret_cast<double2*>(p), c[q]);
            } else {
              __stcs(p, c[q].x);
              __stcs(p + 1, c[q].y);
            }
          }
      }
    }
  }
}

// M_Add: C_l += sum_r W[l, r] * M_r for every C block l, products applied in order r.
struct ScatterArgs {
  double* C;
  long long ldc;
  int ms, ns;
  const double* M;
  long long ldm;
  long long m_stride;
  const int* cblk;          // per C block: row, col, first entry, #entries (4 ints)
  const int* ent_r;         // entries: product index
  const double* ent_w;      // entries: coefficient
};

__global__ void fmm_scatter_kernel(const ScatterArgs a) {
  const int l = blockIdx.y;
  const int row = a.cblk[4 * l + 0], col = a.cblk[4 * l + 1];
  const int e0 = a.cblk[4 * l + 2], ne = a.cblk[4 * l + 3];
  double* Cb = a.C + (long long)row * a.ms + (long long)col * a.ns * a.ldc;
  const long long total = (long long)a.ms * a.ns;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % a.ms);
    const long long j = e / a.ms;
    double c = Cb[i + j * a.ldc];
    for (int q = 0; q < ne; ++q) {
      const double mv = a.M[(long long)a.ent_r[e0 + q] * a.m_stride + i + j * a.ldm];
      c = fma(a.ent_w[e0 + q], mv, c);
    }
    Cb[i + j * a.ldc] = c;
  }
}

}  // namespace fmm
