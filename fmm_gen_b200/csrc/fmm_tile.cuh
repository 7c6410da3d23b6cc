// The FP64 GEMM kernels (DMMA): the plain GEMM and the fringe strips (fmm_tile_gemm_kernel), the
// products of an FMM (fmm_products_kernel) and of a batch of problems
// (fmm_products_batch_kernel).  sm_100a only.
//
// Bound by the FP64 tensor pipe: mma.m16n8k4 issues every 32 cycles per SM sub-partition,
// 37.2 TFLOP/s over 148 SMs, a single warp with one accumulator chain keeps a pipe full, and
// nothing overlaps with it but other warps' loads.  So the warp that multiplies does little
// else: one producer warp per CTA brings the operands in by tensor copies, four consumer
// warps only load fragments (16 bytes a lane, no bank conflicts: see the stage layout) and
// multiply, and three 64 x 64 CTAs (five 32 x 32) share an SM, so that one's C update, start
// and end run under the others' DMMAs.  Measured on B200 against the kernel this replaced (one
// 128 x 128 CTA per SM, 64-bit fragment loads with 4-way conflicts, a separate epilogue
// group): plain 4096^3 33.9 -> 35.6 TFLOP/s (cuBLAS 35.5), 2048^3 32.7 -> 34.7, 1024^3 25 ->
// 30; plain 701 x 503 x 615 108 -> 26 us; whole calls (with the operand sums and combine as they are
// now) 222-1 240^3 126 -> 17.6 us, 1501 x 1203 x 999 421 -> 174 us, 2048^3 568 -> 519 us; 222-1 x 333-1
// 16384^3 205.6 -> 196.1 ms; the 512-problem batch 96.8 -> 89.1 ms (sums in k parts, which cost 2 to 3 % where there
// are any, included: consume_k).  A 64 x 64 tile reads twice the operand bytes of a 128 x 128 one (16 bytes
// per cycle and SM from L2), which costs nothing measurable, and wastes a quarter as much on
// partial tiles and a launch's last round.  Three 64 x 64 CTAs leave a thread 128 registers: the plain kernel fits,
// the products kernels spill 88 to 148 bytes of their units' state (16384^3 runs at 0.95 of the pipe all the same).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "fmm_kernels.cuh"

namespace fmmt {

constexpr int NC = 128;       // consumer threads: 2 x 2 warps
constexpr int NT = NC + 32;   // + the producer warp
constexpr int BK = 16;        // k depth of a stage: two groups of eight
constexpr int MAX_JOBS = 3;   // a launch covers up to three independent GEMMs (the fringe strips)
constexpr int MAX_SPLIT = 8;  // k parts = CTAs of a cluster
// The last units of a products launch are cut into strips of TAIL_ROWS rows (64-row tiles only), so that
// the SMs, which each hold three units at a time, finish closer together.
constexpr int TAIL_ROWS = 16;

// A classical update C += A * B.  The k range is cut into S parts of depth d (a multiple of 8;
// S > 1: one CTA of a cluster each); every C element receives its parts' sums in increasing
// order, c = c + part.
struct TileJob {
  CUtensorMap tmA;  // A (m, k), box 16 x BK, 128-byte swizzle (when a_tma)
  CUtensorMap tmB;  // B (k, n), box 8 x TN (when b_tma)
  const double* A;
  const double* B;
  double* C;
  long long lda, ldb, ldc;
  int m, n, k;
  int tiles_m, tiles_n;
  int S, d;
  int depth;         // of the parts of a CTA's sum (consume_k)
  int first;         // first CTA of the job, a multiple of the launch's cluster size
  int units;         // CTAs
  int a_tma, b_tma;  // 0: per-lane copies (odd leading dimension or unaligned base)
};

struct TileArgs {
  TileJob job[MAX_JOBS];
  int njob;
  int ahead;  // distance of prefetch_update, in CTAs
  unsigned* status;
};

template <int TM, int TN>
struct TileShape {
  static constexpr int WM = TM / 2, WN = TN / 2;  // warp tile
  static constexpr int NI = WM / 16, NJ = WN / 8;
  static constexpr unsigned ABYTES = sizeof(double) * BK * TM, BBYTES = sizeof(double) * BK * TN;
  static constexpr unsigned STAGE = ABYTES + BBYTES;  // bytes
  static constexpr int STAGES = TM == 64 ? 4 : 5;
  static constexpr int CTAS = TM == 64 ? 3 : 5;  // per SM
  static constexpr size_t SMEM = (size_t)STAGE * STAGES + 16 * STAGES + 1024;
  static constexpr unsigned STRIP_ABYTES = sizeof(double) * BK * TAIL_ROWS;
  static_assert(sizeof(double) * TM * TN <= (size_t)STAGE * STAGES, "the part exchange reuses the stages");
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %cluster_ctarank;\n" : "=r"(r));
  return r;
}

__device__ __forceinline__ double2 ld_cluster_f64x2(unsigned addr, unsigned rank) {
  double2 v;
  asm volatile(
      "{\n .reg .b32 r;\n mapa.shared::cluster.u32 r, %2, %3;\n ld.shared::cluster.v2.f64 {%0, %1}, [r];\n}\n"
      : "=d"(v.x), "=d"(v.y)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}

// The barrier receives this lane's arrival once its copies issued so far have landed.
__device__ __forceinline__ void cp_async_arrive(unsigned bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}

// Stage layout.  A: groups of 16 rows, each [k][16 rows] in rows of 128 bytes whose 16-byte
// chunks are XORed with k % 8 (what the 128-byte swizzle of a tensor copy writes); B: the two
// k halves, each [n][8 k] in rows of 64 bytes.  Both are free of bank conflicts for the
// consumers' 16-byte loads (two rows of A at one k, two k of B in one column).
//
// Per-lane copies of one stage, for operands whose columns do not start on 16 bytes.
template <int TM, int TN>
struct LaneCopy {
  const double* pa[TM / 32];
  const double* pb;
  long long lda, ldb2;
  unsigned da[TM / 32], db;
  unsigned va, vb;  // valid rows / columns
  int kb;

  // A and B at the tile's first row / column and first k; vr rows, vc columns inside the block
  __device__ __forceinline__ void init(const double* A, long long ldA, const double* B, long long ldB, int vr, int vc,
                                       int lane) {
    lda = ldA;
    ldb2 = 2 * ldB;
    va = vb = 0;
#pragma unroll
    for (int h = 0; h < TM / 32; ++h) {
      const int m = lane + 32 * h;
      if (m < vr) va |= 1u << h;
      pa[h] = m < vr ? A + m : A;  // a masked-off lane's copy still names an address
      da[h] = (unsigned)((m / 16) * 16 * BK * 8 + (m % 16) * 8);
    }
    kb = lane % 16;
    const int n = lane / 16;
#pragma unroll
    for (int e = 0; e < TN / 2; ++e)
      if (n + 2 * e < vc) vb |= 1u << e;
    pb = vb ? B + kb + (long long)n * ldB : B;
    db = (unsigned)((kb / 8) * TN * 64 + n * 64 + (kb % 8) * 8);
  }
  __device__ __forceinline__ void load_a(unsigned st, int kleft) {
#pragma unroll
    for (int h = 0; h < TM / 32; ++h) {
      const double* p = pa[h];
      const bool v = (va >> h) & 1;
#pragma unroll
      for (int k = 0; k < BK; ++k, p += lda) {
        const bool ok = v && k < kleft;
        fmm::cp_async8(st + (da[h] ^ (unsigned)((k & 7) * 16)) + k * 128, ok ? p : pa[0], ok ? 8 : 0);
      }
      pa[h] = p;
    }
  }
  __device__ __forceinline__ void load_b(unsigned st, int kleft) {
    const double* p = pb;
    const bool kv = kb < kleft;
#pragma unroll
    for (int e = 0; e < TN / 2; ++e, p += ldb2) {
      const bool ok = kv && ((vb >> e) & 1);
      fmm::cp_async8(st + db + e * 128, ok ? p : pb, ok ? 8 : 0);
    }
    pb += BK;
  }
};

// Producer warp: wait for a stage to be free; false when the wait (or an earlier one of the
// launch) gave up, and then nothing more is issued: a copy into a stage still in use, or a
// second arrival in its barrier's phase, must not happen.
__device__ __forceinline__ bool stage_free(unsigned bar, unsigned parity, unsigned* status) {
  fmm::mbar_wait(bar, parity, status);
  return __all_sync(0xffffffffu, fmm::mbar_try_wait(bar, parity));
}

// Tensor copies of one stage: A rows xa.., columns ya..; B rows xb.., columns yb.. .
template <int TM>
__device__ __forceinline__ void tma_stage_a(unsigned st, const CUtensorMap* map, int x, int y, unsigned fb) {
#pragma unroll
  for (int i = 0; i < TM / 16; ++i) fmm::tma_load_2d(st + i * 16 * BK * 8, map, x + 16 * i, y, fb);
}
template <int TN>
__device__ __forceinline__ void tma_stage_b(unsigned st, const CUtensorMap* map, int x, int y, unsigned fb) {
#pragma unroll
  for (int h = 0; h < 2; ++h) fmm::tma_load_2d(st + h * TN * 64, map, x + 8 * h, y, fb);
}

// A C tile of which m x n elements exist to L2, 128-byte lines spread over the warp.
template <int TM, int TN>
__device__ __forceinline__ void prefetch_tile(const double* C, long long ldc, int m, int n, int lane) {
  for (int l = lane; l < (TM / 16) * TN; l += 32) {
    const int r = (l % (TM / 16)) * 16, c = l / (TM / 16);
    if (r < m && c < n) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(C + r + (long long)c * ldc));
  }
}

// Tiles in groups of 16 tile rows: concurrent CTAs share operand panels in L2.
template <int TM, int TN>
__device__ __forceinline__ void tile_origin(int bid, int tiles_m, int tiles_n, int& m0, int& n0) {
  constexpr int G = 16;
  const int per = G * tiles_n, first_m = (bid / per) * G;
  const int rows = min(tiles_m - first_m, G), in = bid % per;
  m0 = (first_m + in % rows) * TM;
  n0 = (in / rows) * TN;
}

// Updates of few stages wait for C and for little else: the CTA of tile t brings the C tile of tile t + ahead to
// L2, those of the first round their own too.  With streaming stores 12000 x 12000 x 8 takes 456 us (5.05 TB/s),
// without both 634; x 2 took 467, in groups of 64 or 256 tile rows instead of 16 about 500.
template <int TM, int TN>
__device__ __forceinline__ void prefetch_update(const TileJob& J, int m0, int n0, int t, int ahead, int lane) {
  if (J.first + t < ahead) prefetch_tile<TM, TN>(J.C + m0 + (long long)n0 * J.ldc, J.ldc, J.m - m0, J.n - n0, lane);
  if (t + ahead >= J.units) return;
  tile_origin<TM, TN>(t + ahead, J.tiles_m, J.tiles_n, m0, n0);
  prefetch_tile<TM, TN>(J.C + m0 + (long long)n0 * J.ldc, J.ldc, J.m - m0, J.n - n0, lane);
}

template <int TM, int TN>
__device__ __forceinline__ void produce(const TileJob& J, unsigned s0, unsigned full0, unsigned empty0, unsigned* status,
                                        int m0, int n0, int kbeg, int kend, int pre, int ahead, int lane) {
  using S = TileShape<TM, TN>;
  const int nst = (kend - kbeg + BK - 1) / BK;
  const bool at = J.a_tma != 0, bt = J.b_tma != 0;
  LaneCopy<TM, TN> lc;
  if (!at || !bt)
    lc.init(J.A + m0 + (long long)kbeg * J.lda, J.lda, J.B + kbeg + (long long)n0 * J.ldb, J.ldb, J.m - m0, J.n - n0,
            lane);
  const unsigned tx = (at ? S::ABYTES : 0u) + (bt ? S::BBYTES : 0u);
  int s = 0;
#pragma unroll 1
  for (; s < nst; ++s) {
    const int slot = s % S::STAGES;
    const unsigned st = s0 + slot * S::STAGE, fb = full0 + 8 * slot;
    if (!stage_free(empty0 + 8 * slot, (unsigned)(((s / S::STAGES) & 1) ^ 1), status)) break;
    if (lane == 0 && tx) {
      fmm::mbar_arrive_expect_tx(fb, tx);
      const int k = kbeg + s * BK;
      if (at) tma_stage_a<TM>(st, &J.tmA, m0, k, fb);
      if (bt) tma_stage_b<TN>(st + S::ABYTES, &J.tmB, k, n0, fb);
    }
    if (!at || !bt) {
      const int kleft = kend - kbeg - s * BK;
      if (!at) lc.load_a(st, kleft);
      if (!bt) lc.load_b(st + S::ABYTES, kleft);
      cp_async_arrive(fb);
    }
  }
  if (pre >= 0) prefetch_update<TM, TN>(J, m0, n0, pre, ahead, lane);
  // copies still in flight (only on an error path) land before the CTA exits
  for (int q = max(0, s - S::STAGES); q < s; ++q)
    fmm::mbar_wait_drain(full0 + 8 * (q % S::STAGES), (unsigned)((q / S::STAGES) & 1));
}

// A k group of eight (kh = 0, 1 of the stage) into the accumulators: DMMA slot t of the first
// half takes k = 2 t, of the second 2 t + 1; MMA row g is tile row 2 g, row g + 8 is 2 g + 1.
template <int TM, int TN, int IM, int JN>
__device__ __forceinline__ void mma_group(const unsigned char* sa, const unsigned char* sb, unsigned oa0, unsigned oa1, int kh,
                                          double (&acc)[TileShape<TM, TN>::NI][TileShape<TM, TN>::NJ][4]) {
  double2 bf[JN];
#pragma unroll
  for (int j = 0; j < JN; ++j) bf[j] = *reinterpret_cast<const double2*>(sb + kh * (TN * 64) + j * 512);
#pragma unroll
  for (int kq = 0; kq < 2; ++kq) {
    double2 af[IM];
#pragma unroll
    for (int i = 0; i < IM; ++i)
      af[i] = *reinterpret_cast<const double2*>(sa + (kq ? oa1 : oa0) + kh * 1024 + i * (16 * BK * 8));
#pragma unroll
    for (int i = 0; i < IM; ++i)
#pragma unroll
      for (int j = 0; j < JN; ++j) {
        const double a[2] = {af[i].x, af[i].y};
        fmm::dmma_16x8x4(acc[i][j], a, kq ? bf[j].y : bf[j].x);
      }
  }
}

// The k loop over a product's stages for the fragments i < IM, j < JN (0, 0: only the stage
// hand-off).  Counts known at compile time keep the loop straight-line code.
template <int TM, int TN, int IM, int JN>
__device__ __forceinline__ void consume_loop(const unsigned char* smem, unsigned full0, unsigned empty0, unsigned* status,
                                             int kleft, double (&acc)[TileShape<TM, TN>::NI][TileShape<TM, TN>::NJ][4],
                                             int row, int col, int lane, int& slot, unsigned& ph) {
  using S = TileShape<TM, TN>;
  const int g = lane >> 2, t4 = lane & 3;
  const unsigned oa0 = (unsigned)(2 * t4 * 128 + ((g ^ (2 * t4)) * 16));
  const unsigned oa1 = (unsigned)((2 * t4 + 1) * 128 + ((g ^ (2 * t4 + 1)) * 16));
  const unsigned char* a0 = smem + row * BK * 8;
  const unsigned char* b0 = smem + S::ABYTES + (col + g) * 64 + t4 * 16;
#pragma unroll 1
  for (; kleft > 0; kleft -= BK) {
    fmm::mbar_wait(full0 + 8 * slot, ph, status);
    if constexpr (IM > 0) {
      const unsigned char *sa = a0 + slot * S::STAGE, *sb = b0 + slot * S::STAGE;
      mma_group<TM, TN, IM, JN>(sa, sb, oa0, oa1, 0, acc);
      if (kleft > 8) mma_group<TM, TN, IM, JN>(sa, sb, oa0, oa1, 1, acc);
      __threadfence_block();  // fragment loads complete before the stage can be refilled
    }
    __syncwarp();
    if (lane == 0) fmm::mbar_arrive(empty0 + 8 * slot);
    if (++slot == S::STAGES) {
      slot = 0;
      ph ^= 1;
    }
  }
}

// The fragments that hold elements of the block, i < im, j < jn, run in the next larger of a
// few compiled shapes (extra fragments are harmless: their sums are never stored).  Measured:
// one loop with a test per fragment cost 3000^3 plain 6 % over 3008^3, for 4 % partial tiles
// most of whose fragments are all needed.
template <int TM, int TN>
__device__ __forceinline__ void consume(const unsigned char* smem, unsigned full0, unsigned empty0, unsigned* status, int kleft,
                                        double (&acc)[TileShape<TM, TN>::NI][TileShape<TM, TN>::NJ][4], int row, int col,
                                        int lane, int im, int jn, int& slot, unsigned& ph) {
  constexpr int NI = TileShape<TM, TN>::NI, NJ = TileShape<TM, TN>::NJ;
  if (im == 0 || jn == 0)
    consume_loop<TM, TN, 0, 0>(smem, full0, empty0, status, kleft, acc, row, col, lane, slot, ph);
  else if (jn <= NJ / 2 && im <= NI / 2)
    consume_loop<TM, TN, (NI + 1) / 2, NJ / 2>(smem, full0, empty0, status, kleft, acc, row, col, lane, slot, ph);
  else if (jn <= NJ / 2)
    consume_loop<TM, TN, NI, NJ / 2>(smem, full0, empty0, status, kleft, acc, row, col, lane, slot, ph);
  else if (im <= NI / 2)
    consume_loop<TM, TN, (NI + 1) / 2, NJ>(smem, full0, empty0, status, kleft, acc, row, col, lane, slot, ph);
  else
    consume_loop<TM, TN, NI, NJ>(smem, full0, empty0, status, kleft, acc, row, col, lane, slot, ph);
}

template <int TM, int TN>
__device__ __forceinline__ void zero_acc(double (&acc)[TileShape<TM, TN>::NI][TileShape<TM, TN>::NJ][4]) {
#pragma unroll
  for (int i = 0; i < TileShape<TM, TN>::NI; ++i)
#pragma unroll
    for (int j = 0; j < TileShape<TM, TN>::NJ; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
}

// The sum over k into acc.  PARTS: in parts of `depth` (a multiple of BK, or k): a part is summed
// from zero and the parts before it are added, so rounding grows with the parts' depth and their number and
// not with k.  The part loop and the earlier parts' sums cost 64-row tiles 1 to 3 % (three parts of
// 168 against one: 222-1 1501 x 1203 x 999 167.4 -> 172 us; kernels without it keep their time), about half of it
// for the first boundary and half for the additions; folding fragment by fragment under the next one's DMMAs took
// 1 % longer in batches.
template <int TM, int TN, bool PARTS>
__device__ __forceinline__ void consume_k(const unsigned char* smem, unsigned full0, unsigned empty0, unsigned* status, int k,
                                          int depth, double (&acc)[TileShape<TM, TN>::NI][TileShape<TM, TN>::NJ][4],
                                          int row, int col, int lane, int im, int jn, int& slot, unsigned& ph) {
  using S = TileShape<TM, TN>;
  if constexpr (!PARTS) {
    zero_acc<TM, TN>(acc);
    consume<TM, TN>(smem, full0, empty0, status, k, acc, row, col, lane, im, jn, slot, ph);
  } else {
    double2 sum[S::NI][S::NJ][2];
    // in local memory: left to ptxas, these values and the k loop's competed for registers (2 to 3 %)
    if constexpr (TM == 64) asm volatile("" ::"l"(&sum[0][0][0]) : "memory");
#pragma unroll 1
    for (int left = k; left > 0; left -= depth) {
      zero_acc<TM, TN>(acc);
      consume<TM, TN>(smem, full0, empty0, status, min(left, depth), acc, row, col, lane, im, jn, slot, ph);
      if (left < k) {
#pragma unroll
        for (int i = 0; i < S::NI; ++i)
#pragma unroll
          for (int j = 0; j < S::NJ; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const double2 v = sum[i][j][e];
              acc[i][j][2 * e] += v.x;
              acc[i][j][2 * e + 1] += v.y;
            }
      }
      if (left > depth) {
#pragma unroll
        for (int i = 0; i < S::NI; ++i)
#pragma unroll
          for (int j = 0; j < S::NJ; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) sum[i][j][e] = make_double2(acc[i][j][2 * e], acc[i][j][2 * e + 1]);
      }
    }
  }
}

// Fragments of this warp inside a block of which vr x vc elements lie right and below the warp
// tile's corner: i < im, j < jn.
template <int TM, int TN>
__device__ __forceinline__ void frag_counts(int vr, int vc, int& im, int& jn) {
  im = vr <= 0 ? 0 : min(TileShape<TM, TN>::NI, (vr + 15) >> 4);
  jn = vc <= 0 ? 0 : min(TileShape<TM, TN>::NJ, (vc + 7) >> 3);
}

// C += w acc (or C = acc) for a warp's fragments; C at the warp tile's first element of an
// m x n remainder.  Rows 2 g, 2 g + 1 of a column are one 16-byte access where the columns
// allow it (vec), and a warp access covers 128 bytes of four columns; a fragment row's loads
// are all issued before its stores.  STREAM: the stores leave L2 first (an update that C's traffic bounds).
template <int TM, int TN, bool STORE, bool STREAM = false>
__device__ __forceinline__ void update_c(double* C, long long ldc, int m, int n, bool vec, double w,
                                         const double (&acc)[TileShape<TM, TN>::NI][TileShape<TM, TN>::NJ][4], int g,
                                         int t4) {
  using S = TileShape<TM, TN>;
#pragma unroll
  for (int i = 0; i < S::NI; ++i) {
    const int rr = i * 16 + 2 * g;
    const bool two = vec && rr + 1 < m;
    double2 cv[S::NJ][2];
    if (!STORE) {
#pragma unroll
      for (int j = 0; j < S::NJ; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int cc = j * 8 + 2 * t4 + q;
          cv[j][q] = make_double2(0.0, 0.0);
          if (cc >= n) continue;
          const double* cp = C + rr + (long long)cc * ldc;
          if (two) {
            cv[j][q] = *reinterpret_cast<const double2*>(cp);
          } else {
            if (rr < m) cv[j][q].x = cp[0];
            if (rr + 1 < m) cv[j][q].y = cp[1];
          }
        }
    }
#pragma unroll
    for (int j = 0; j < S::NJ; ++j)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int cc = j * 8 + 2 * t4 + q;
        if (cc >= n) continue;
        double* cp = C + rr + (long long)cc * ldc;
        const double x = STORE ? acc[i][j][q] : fma(w, acc[i][j][q], cv[j][q].x);
        const double y = STORE ? acc[i][j][2 + q] : fma(w, acc[i][j][2 + q], cv[j][q].y);
        if (two) {
          if (STREAM)
            __stcs(reinterpret_cast<double2*>(cp), make_double2(x, y));
          else
            *reinterpret_cast<double2*>(cp) = make_double2(x, y);
        } else {
          if (rr < m) STREAM ? __stcs(cp, x) : (void)(cp[0] = x);
          if (rr + 1 < m) STREAM ? __stcs(cp + 1, y) : (void)(cp[1] = y);
        }
      }
  }
}

__device__ __forceinline__ bool vec_ok(const double* C, long long ldc) {
  return ((reinterpret_cast<uintptr_t>(C) & 15) == 0) && ((ldc & 1) == 0);
}

// Wait for the launch's predecessors (programmatic dependent launch): nothing before this
// touches global memory that they write.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void grid_launch() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// One CTA per (tile, part) of up to three independent classical updates C += A * B: the plain
// GEMM and the fringe strips.  The parts of a tile are the CTAs of a cluster, which leave their
// sums in shared memory and then add every part, in order, to their share of the tile.
// PARTS: some CTA's sum is made of parts of its own (consume_k).  SHALLOW: C's traffic bounds the launch, whose
// jobs have one part each.
template <int TM, int TN, bool PARTS, bool SHALLOW = false>
__global__ void __launch_bounds__(NT, (TileShape<TM, TN>::CTAS)) fmm_tile_gemm_kernel(const __grid_constant__ TileArgs g) {
  using S = TileShape<TM, TN>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (fmm::smem_u32(smem_raw) & 1023)) & 1023);  // swizzle atoms
  const unsigned s0 = fmm::smem_u32(smem), full0 = s0 + S::STAGE * S::STAGES, empty0 = full0 + 8 * S::STAGES;
  int ji = 0;
#pragma unroll
  for (int q = 1; q < MAX_JOBS; ++q)
    if (q < g.njob && (int)blockIdx.x >= g.job[q].first) ji = q;
  const TileJob& J = g.job[ji];
  const int u = (int)blockIdx.x - J.first;
  // Padding to whole clusters, where the launch's cluster is larger than this job's part count.  The cluster's
  // barriers do not count threads that have exited, and a tile's parts never address another tile's CTAs.
  if (u >= J.units) return;
  const int part = u % J.S, t = u / J.S;
  int m0, n0;
  tile_origin<TM, TN>(t, J.tiles_m, J.tiles_n, m0, n0);
  const int kbeg = part * J.d, kend = min(J.k, kbeg + J.d);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    const unsigned nfull = (J.a_tma || J.b_tma ? 1u : 0u) + (J.a_tma && J.b_tma ? 0u : 32u);
    for (int s = 0; s < S::STAGES; ++s) {
      fmm::mbar_init(full0 + 8 * s, nfull);
      fmm::mbar_init(empty0 + 8 * s, NC / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  grid_wait();
  grid_launch();
  const int g4 = lane >> 2, t4 = lane & 3, wm = (warp >> 1) & 1, wn = warp & 1;
  const bool vec = vec_ok(J.C, J.ldc);
  if (warp == NC / 32) {
    produce<TM, TN>(J, s0, full0, empty0, g.status, m0, n0, kbeg, kend, SHALLOW ? t : -1, g.ahead, lane);
    if (J.S == 1) return;
    __syncwarp();
  } else {
    double acc[S::NI][S::NJ][4];
    const int vr = J.m - m0 - wm * S::WM, vc = J.n - n0 - wn * S::WN;
    int im, jn, slot = 0;
    unsigned ph = 0;
    frag_counts<TM, TN>(vr, vc, im, jn);
    consume_k<TM, TN, PARTS>(smem, full0, empty0, g.status, kend - kbeg, J.depth, acc, wm * S::WM, wn * S::WN, lane, im, jn,
                             slot, ph);
    if (J.S == 1) {
      double* C = J.C + (m0 + wm * S::WM) + (long long)(n0 + wn * S::WN) * J.ldc;
      if (SHALLOW && !vec)  // code without the wide accesses
        update_c<TM, TN, false, SHALLOW>(C, J.ldc, vr, vc, false, 1.0, acc, g4, t4);
      else
        update_c<TM, TN, false, SHALLOW>(C, J.ldc, vr, vc, vec, 1.0, acc, g4, t4);
      return;
    }
    fmm::named_bar_sync(1, NC);  // every consumer warp is done with the stages
    double2* red = reinterpret_cast<double2*>(smem);  // [TN][TM / 2] row pairs
#pragma unroll
    for (int i = 0; i < S::NI; ++i)
#pragma unroll
      for (int j = 0; j < S::NJ; ++j)
#pragma unroll
        for (int q = 0; q < 2; ++q)
          red[(wn * S::WN + j * 8 + 2 * t4 + q) * (TM / 2) + (wm * S::WM + i * 16) / 2 + g4] =
              make_double2(acc[i][j][q], acc[i][j][2 + q]);
  }
  cluster_sync();
  // the tile's parts are neighbours in the cluster, which may hold several tiles
  const unsigned rank0 = cluster_rank() - (unsigned)part;
  constexpr int P = TM / 2 * TN;
  for (int q = P * part / J.S + tid; q < P * (part + 1) / J.S; q += NT) {
    const int rr = m0 + 2 * (q % (TM / 2)), cc = n0 + q / (TM / 2);
    if (rr >= J.m || cc >= J.n) continue;
    double* cp = J.C + rr + (long long)cc * J.ldc;
    const bool two = vec && rr + 1 < J.m;
    double2 c = make_double2(0.0, 0.0);
    if (two) {
      c = *reinterpret_cast<const double2*>(cp);
    } else {
      c.x = cp[0];
      if (rr + 1 < J.m) c.y = cp[1];
    }
    const unsigned addr = s0 + (unsigned)q * 16;
    for (int s = 0; s < J.S; ++s) {
      const double2 v = ld_cluster_f64x2(addr, rank0 + (unsigned)s);
      c.x += v.x;
      c.y += v.y;
    }
    if (two) {
      *reinterpret_cast<double2*>(cp) = c;
    } else {
      cp[0] = c.x;
      if (rr + 1 < J.m) cp[1] = c.y;
    }
  }
  cluster_sync();  // no CTA leaves while another still reads its part
}

// ------------------------------------------------------------------------------------
// FMM products: persistent CTAs over (tile, product range) units, each product's operands one
// block each (a block of A / B or a slot of the pre-summed workspaces), the product added to
// every C block of its W column or stored to its workspace slab.
// ------------------------------------------------------------------------------------
struct ProdArgs {
  CUtensorMap tmA, tmAw;  // A and the pre-summed S, box 16 x BK, 128-byte swizzle
  CUtensorMap tmB, tmBw;  // B and T, box 8 x 64
  const double* A;        // lane copies (a_tma / b_tma == 0)
  const double* B;
  long long lda, ldb;
  double* C;              // MODE_ACCUM_C
  long long ldc;
  double* M;              // MODE_STORE_M: product r at M + r * m_stride, ld = ms
  long long m_stride;
  const fmm::Prod* prods;
  const fmm::Term* terms;
  int* tickets;           // per warp tile (4 per tile) and, nbt > 0, per C block: updates done, in
                          // product order; zeroed before the launch
  unsigned* status;
  int* counter;           // work units claimed so far, zeroed before the launch
  int ms, ns, ks;         // product sizes
  int kcap;               // k extent of A and B (a k split's last part may end early)
  int nprod, tiles_m, tiles_n;
  int chunks;             // units per tile: consecutive product ranges
  int mode;
  int nbt, nbc;           // > 0: tickets per C block too, nbt blocks in rows of nbc
  int a_tma, b_tma;
  int tail, claims;       // fmm_products_kernel: units from `tail` on are cut into row strips (only in launches
                          // without tickets), and the claims that makes
  int depth;              // of the parts of a product's sum (consume_k)
  int pad[1];
};
static_assert(sizeof(ProdArgs) % 64 == 0, "tensor maps in a job table start on 64 bytes");

struct OneProd {
  const ProdArgs& a;
  __device__ __forceinline__ const ProdArgs& get(int) const { return a; }
  __device__ __forceinline__ int find(int) const { return 0; }
  __device__ __forceinline__ int first_unit(int) const { return 0; }
  __device__ __forceinline__ int tail() const { return a.tail; }
  __device__ __forceinline__ int claims() const { return a.claims; }
  __device__ __forceinline__ unsigned* status() const { return a.status; }
  __device__ __forceinline__ int* counter() const { return a.counter; }
  __device__ __forceinline__ void acquire_maps(int) const {}
};

struct ProdBatchArgs {
  const ProdArgs* jobs;   // global memory
  const int* unit_start;  // njobs + 1 entries
  int njobs, units;
  unsigned* status;
  int* counter;
};

struct ProdBatch {
  const ProdBatchArgs& b;
  __device__ __forceinline__ const ProdArgs& get(int j) const { return b.jobs[j]; }
  __device__ __forceinline__ int find(int u) const {  // last j with unit_start[j] <= u
    int lo = 0, hi = b.njobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(b.unit_start + mid) <= u)
        lo = mid;
      else
        hi = mid - 1;
    }
    return lo;
  }
  __device__ __forceinline__ int first_unit(int j) const { return __ldg(b.unit_start + j); }
  __device__ __forceinline__ int tail() const { return b.units; }
  __device__ __forceinline__ int claims() const { return b.units; }
  __device__ __forceinline__ unsigned* status() const { return b.status; }
  __device__ __forceinline__ int* counter() const { return b.counter; }
  // the maps were written by a copy before the launch; order it before the tensor-map proxy
  __device__ __forceinline__ void acquire_maps(int j) const {
    const CUtensorMap* m = &b.jobs[j].tmA;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(m + q) : "memory");
  }
};

// A claim: a unit of a job, or a row strip of one (strip >= 0).
struct PClaim {
  int unit, strip;
};
template <int T, bool STRIPS>
__device__ __forceinline__ PClaim decode_claim(int v, int tail) {
  constexpr int N = T / TAIL_ROWS;
  return STRIPS && v >= tail ? PClaim{tail + (v - tail) / N, (v - tail) % N} : PClaim{v, -1};
}

struct PUnit {
  int m0, n0, tile, chunk, r0, r1;
  bool strip;
};

template <int T>
__device__ __forceinline__ PUnit decode(const ProdArgs& a, int u, int strip) {
  const int ntiles = a.tiles_m * a.tiles_n;
  PUnit w;
  w.chunk = u / ntiles;  // chunk-major: the units of one tile are a whole tile grid apart
  w.tile = u % ntiles;
  w.r0 = (int)((long long)a.nprod * w.chunk / a.chunks);
  w.r1 = (int)((long long)a.nprod * (w.chunk + 1) / a.chunks);
  tile_origin<T, T>(w.tile, a.tiles_m, a.tiles_n, w.m0, w.n0);
  w.strip = strip >= 0;
  if (w.strip) {
    w.m0 += strip * TAIL_ROWS;
    if (w.m0 >= a.ms) w.r1 = w.r0;  // a strip below the last row
  }
  return w;
}

template <int T>
struct ProdShape {
  static constexpr size_t SMEM = TileShape<T, T>::SMEM + fmm::RING_BYTES;
};

constexpr int C_PREFETCH_STAGES = 12;  // stages before a product's end at which its C tiles go to L2

// C tiles a product will update, 128-byte lines spread over the warp.
template <int T>
__device__ __forceinline__ void prefetch_c(const ProdArgs& a, const fmm::Prod& p, int m0, int n0, int lane) {
  for (int c = 0; c < p.nc; ++c) {
    const fmm::Term tm = a.terms[p.c0 + c];
    const double* Cb = a.C + (long long)tm.row * a.ms + (long long)tm.col * a.ns * a.ldc;
    for (int l = lane; l < (T / 16) * T; l += 32) {
      const int rr = m0 + (l % (T / 16)) * 16, cc = n0 + l / (T / 16);
      if (rr < a.ms && cc < a.ns) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(Cb + rr + (long long)cc * a.ldc));
    }
  }
}

template <int T, bool LANES, bool STRIPS, class Src>
__device__ __forceinline__ void prod_producer(const Src& src, const fmm::UnitRing& q, unsigned s0, unsigned full0,
                                              unsigned empty0, int lane) {
  using S = TileShape<T, T>;
  long long kc = 0;
  int mapped = -1;
  bool ok = true;
#pragma unroll 1
  for (int n = 0; ok; ++n) {
    int u = -1;
    if (lane == 0) {  // claim the next unit and publish it to the consumers
      const int e = n % fmm::UQ_DEPTH;
      fmm::mbar_wait(q.empty(e), (unsigned)(((n / fmm::UQ_DEPTH) & 1) ^ 1), src.status());
      if ((*(volatile unsigned*)src.status() & fmm::STATUS_WAIT_TIMEOUT) == 0u) {
        u = atomicAdd(src.counter(), 1);
        if (u >= src.claims()) u = -1;
      }
      fmm::st_shared_s32(q.entry(e), u);
      fmm::mbar_arrive(q.full(e));
    }
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u < 0) break;
    const PClaim cl = decode_claim<T, STRIPS>(u, src.tail());
    const int job = src.find(cl.unit);
    const ProdArgs& a = src.get(job);
    if (job != mapped) {
      if (lane == 0) src.acquire_maps(job);
      mapped = job;
    }
    const PUnit w = decode<T>(a, cl.unit - src.first_unit(job), STRIPS ? cl.strip : -1);
    const int nst = (a.ks + BK - 1) / BK;
    const int spre = a.mode == fmm::MODE_ACCUM_C ? max(0, nst - C_PREFETCH_STAGES) : -1;
#pragma unroll 1
    for (int r = w.r0; r < w.r1 && ok; ++r) {
      const fmm::Prod p = a.prods[r];
      const fmm::Term ta = a.terms[p.a0], tb = a.terms[p.b0];
      const CUtensorMap* ma = ta.src ? &a.tmAw : &a.tmA;
      const CUtensorMap* mb = tb.src ? &a.tmBw : &a.tmB;
      const int xa = ta.row * a.ms + w.m0, ya = ta.col * a.ks;
      const int xb = tb.row * a.ks, yb = tb.col * a.ns + w.n0;
      const bool at = !LANES || ta.src || a.a_tma, bt = !LANES || tb.src || a.b_tma;
      const unsigned tx = (at ? (STRIPS && w.strip ? S::STRIP_ABYTES : S::ABYTES) : 0u) + (bt ? S::BBYTES : 0u);
      LaneCopy<T, T> lc;
      if (LANES && (!at || !bt))
        lc.init(a.A + xa + (long long)ya * a.lda, a.lda, a.B + xb + (long long)yb * a.ldb, a.ldb,
                a.ms - w.m0, a.ns - w.n0, lane);
#pragma unroll 1
      for (int s = 0; s < nst; ++s, ++kc) {
        const int slot = (int)(kc % S::STAGES);
        const unsigned st = s0 + slot * S::STAGE, fb = full0 + 8 * slot;
        if (s == spre) prefetch_c<T>(a, p, w.m0, w.n0, lane);
        ok = stage_free(empty0 + 8 * slot, (unsigned)(((kc / S::STAGES) & 1) ^ 1), src.status());
        if (!ok) break;
        if (lane == 0) {
          fmm::mbar_arrive_expect_tx(fb, tx);
          if (STRIPS && w.strip)
            tma_stage_a<TAIL_ROWS>(st, ma, xa, ya + s * BK, fb);
          else if (at)
            tma_stage_a<T>(st, ma, xa, ya + s * BK, fb);
          if (bt) tma_stage_b<T>(st + S::ABYTES, mb, xb + s * BK, yb, fb);
        }
        if (LANES) {
          if (at && bt) {
            fmm::mbar_arrive(fb);  // every lane: the barrier counts 32 lanes and the issuer
          } else {
            // the product's own k range, ending at the operands' (a last part may be short)
            if (!at) lc.load_a(st, min(a.ks, a.kcap - ya) - s * BK);
            if (!bt) lc.load_b(st + S::ABYTES, min(a.ks, a.kcap - xb) - s * BK);
            cp_async_arrive(fb);
          }
        }
        __syncwarp();
      }
    }
  }
  // copies still in flight (only on an error path) land before the CTA exits
  for (long long k = kc > S::STAGES ? kc - S::STAGES : 0; k < kc; ++k)
    fmm::mbar_wait_drain(full0 + 8 * (int)(k % S::STAGES), (unsigned)((k / S::STAGES) & 1));
}

template <int T, bool STRIPS, bool PARTS, class Src>
__device__ __forceinline__ void prod_consumer(const Src& src, const fmm::UnitRing& q, const unsigned char* smem,
                                              unsigned full0, unsigned empty0, int warp, int lane) {
  using S = TileShape<T, T>;
  const int g4 = lane >> 2, t4 = lane & 3, wm = warp >> 1, wn = warp & 1;
  fmm::UnitReader nx{q, src.status(), true};
  int slot = 0;
  unsigned ph = 0;
  double acc[S::NI][S::NJ][4];
#pragma unroll 1
  for (int u = nx.next(); u >= 0; u = nx.next()) {
    const PClaim cl = decode_claim<T, STRIPS>(u, src.tail());
    const int job = src.find(cl.unit);
    const ProdArgs& a = src.get(job);
    const PUnit w = decode<T>(a, cl.unit - src.first_unit(job), STRIPS ? cl.strip : -1);
    // two by two warps over a tile, four side by side over a row strip
    const bool strip = STRIPS && w.strip;
    const int wrow = strip ? 0 : wm * S::WM, wcol = strip ? warp * (T / 4) : wn * S::WN;
    const int vr = strip ? min(a.ms - w.m0, TAIL_ROWS) : a.ms - w.m0 - wrow;
    const int vc = strip ? min(a.ns - w.n0 - wcol, T / 4) : a.ns - w.n0 - wcol;
    int im, jn;
    frag_counts<T, T>(vr, vc, im, jn);
    const bool ordered = a.mode == fmm::MODE_ACCUM_C && a.chunks > 1;
#pragma unroll 1
    for (int r = w.r0; r < w.r1; ++r) {
      consume_k<T, T, PARTS>(smem, full0, empty0, src.status(), a.ks, a.depth, acc, wrow, wcol, lane, im, jn, slot, ph);
      const long long row = w.m0 + wrow, col = w.n0 + wcol;
      if (a.mode == fmm::MODE_STORE_M) {
        update_c<T, T, true>(a.M + (long long)r * a.m_stride + row + col * a.ms, a.ms, vr, vc,
                             vec_ok(a.M + (long long)r * a.m_stride, a.ms), 1.0, acc, g4, t4);
        continue;
      }
      const fmm::Prod p = a.prods[r];
      const bool vec = vec_ok(a.C, a.ldc);
      const bool per_block = ordered && a.nbt > 0;
      // a ticket belongs to one warp tile: the warps of a CTA do not wait for one another
      if (ordered && !per_block && r == w.r0) {
        if (lane == 0) fmm::ticket_spin(a.tickets + w.tile * 4 + warp, w.chunk, a.status, 128);
        __syncwarp();
      }
#pragma unroll 1
      for (int c = 0; c < p.nc; ++c) {
        const fmm::Term tm = a.terms[p.c0 + c];
        int* tk = nullptr;
        if (per_block) {  // wait for the previous product that updates this C block
          tk = a.tickets + (long long)(w.tile * 4 + warp) * a.nbt + tm.row * a.nbc + tm.col;
          if (lane == 0) fmm::ticket_spin(tk, tm.pad, a.status, 64);
          __syncwarp();
        }
        update_c<T, T, false>(a.C + (tm.row * (long long)a.ms + row) + (tm.col * (long long)a.ns + col) * a.ldc, a.ldc,
                              vr, vc, vec && ((tm.row * a.ms) & 1) == 0, tm.coef, acc, g4, t4);
        if (tk) {  // this block's update is visible before the next product may start its own
          __threadfence();
          __syncwarp();
          if (lane == 0) fmm::st_release(tk, tm.pad + 1);
        }
      }
    }
    if (ordered && a.nbt == 0) {
      __threadfence();
      __syncwarp();
      if (lane == 0) fmm::st_release(a.tickets + w.tile * 4 + warp, w.chunk + 1);
    }
  }
}

// LANES: some operands are read by per-lane copies; STRIPS: the last units run as row strips (not with LANES);
// PARTS: some products' sums are made of parts (consume_k).
template <int T, bool LANES, bool STRIPS, bool PARTS, class Src>
__device__ __forceinline__ void prod_cta(const Src& src) {
  using S = TileShape<T, T>;
  static_assert(!(LANES && STRIPS), "per-lane copies fill whole tiles");
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024 - (fmm::smem_u32(smem_raw) & 1023)) & 1023);  // swizzle atoms
  const unsigned s0 = fmm::smem_u32(smem), full0 = s0 + S::STAGE * S::STAGES, empty0 = full0 + 8 * S::STAGES;
  const fmm::UnitRing q{empty0 + 8 * S::STAGES};
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < S::STAGES; ++s) {
      fmm::mbar_init(full0 + 8 * s, LANES ? 33 : 1);
      fmm::mbar_init(empty0 + 8 * s, NC / 32);
    }
    fmm::unit_ring_init(q, NC / 32);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  grid_wait();
  grid_launch();
  if (warp == NC / 32)
    prod_producer<T, LANES, STRIPS>(src, q, s0, full0, empty0, lane);
  else
    prod_consumer<T, STRIPS, PARTS>(src, q, smem, full0, empty0, warp, lane);
}

template <int T, bool STRIPS, bool PARTS>
__global__ void __launch_bounds__(NT, (TileShape<T, T>::CTAS)) fmm_products_kernel(const __grid_constant__ ProdArgs a) {
  prod_cta<T, false, STRIPS, PARTS>(OneProd{a});
}

template <bool LANES, bool PARTS>
__global__ void __launch_bounds__(NT, (TileShape<64, 64>::CTAS))
    fmm_products_batch_kernel(const __grid_constant__ ProdBatchArgs b) {
  prod_cta<64, LANES, false, PARTS>(ProdBatch{b});
}

}  // namespace fmmt
