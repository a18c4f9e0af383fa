// gemm_f64.cu -- grouped FP64 block GEMM on the DMMA tensor pipe.
//
// All dense contractions of one commutator stage (the ladders of
// matrix_mult222, the intermediates of commutator_221, the one-body products
// of commutator_111 and the Pandya products of construct_cc_ints) run as ONE
// launch over a task list that covers every (M_L,M_S) block of uneven size.
//
// Problem = one output sub-block C (M x N, column-major, ldc) and a list of
// K-segments  acc += alpha_s * op(A_s) op(B_s); the segments are concatenated
// along K so every output tile is accumulated in registers and written once.
// Epilogue modes:
//   ACC       C += V
//   SET       C  = V
//   ACC_PAIR  C += V + sigma V^T      (M == N; the CTA computes the tile pair
//   SET_PAIR  C  = V + sigma V^T       (I,J),(J,I) so V^T is at hand)
// (sigma = +-1).  The pair modes carry the "hA*W^T - hB*W" transpose-adds of the reference
// (src/commutators.f90:1002-1127, :154-169) without a second GEMM.
//
// Tiles of 64 or 32 rows by 64, 32 or 16 columns and 16 k (64 x 64: 4 warps,
// each 32 x 32 = 4 x 4 DMMA m8n8k4 fragments); the rows and columns of a
// problem are cut into full tiles and one narrower rest (see cuts), 32 x 32
// throughout where a program has too few tiles to fill the chip;
// 3-stage cp.async (8-byte, zero-fill) pipeline; FP64 accumulate.
// tcgen05 has no f64 kind, so mma.sync DMMA is the FP64 tensor path here (the
// shapes m8n8k4 to m16n8k16 all reach 36 to 37 TFLOP/s from registers).
// Bound: keeping the tensor pipe fed.  A tile pair (I,J), (J,I) is one product
// of twice the K -- V(J,I)^T is the product of the transposed operands in the
// other order, so C(I,J) = V(I,J) + sigma V(J,I)^T accumulates in one set of
// registers and C(J,I) = sigma C(I,J)^T -- and the panels are swizzled instead
// of padded: 48 KB of shared memory and 128 registers, four CTAs on an SM.
// (With V(I,J) kept in shared memory while V(J,I) was formed: 85.5 KB, two
// CTAs, the tensor pipe 59% active: the ladders of two dense operators at
// N=20, R=20 took 6.18 ms, 5.38 in this form.)
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "dev_common.cuh"

namespace qd {

constexpr int BM = 64, BN = 64, BK = 16, NSTAGE = 3, TLD = 65;  // the largest tile
constexpr int GEMM_THREADS = 128;
// tile shapes of k_grouped_gemm as a task names them
__host__ __device__ constexpr int tile_shape(int tm, int tn) { return tm * 128 + tn; }
constexpr int PANEL = BK * BM;  // doubles of one panel [k][m]
constexpr size_t GEMM_SMEM = sizeof(double) * 2 * NSTAGE * PANEL;
static_assert(BN * TLD <= 2 * NSTAGE * PANEL, "the epilogue's tile uses the pipeline's buffers");

// Position of (k, m) in a panel: m is permuted within 16 by k, so that every
// access touches each bank once -- stores along m, stores along k (16 k of
// one m), and a DMMA fragment (4 k x 8 m).
__device__ __forceinline__ int panel_pos(int k, int m) { return k * BM + (m ^ (((k & 3) << 2) | ((k >> 2) & 3))); }

__device__ __forceinline__ void cp_async8(double* s, const double* g, bool pred) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(s);
  int sz = pred ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(g), "r"(sz));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ bool seg_active(const GSeg& s, unsigned mA, unsigned mB) {
  auto dead = [&](int src, int dep) {
    if (dep < 0) return false;
    unsigned m = src == 0 ? mA : (src == 1 ? mB : 0u);
    return ((m >> dep) & 1u) != 0;
  };
  return !dead(s.srcA, s.depA) && !dead(s.srcB, s.depB);
}

// k-slab [k0, k0 + BK) of W rows (columns) from x0 on of one operand, into a
// panel [k][x].  contig: x is the contiguous index in memory (threads along
// x), else k is (threads along k).  Out-of-range elements are zero-filled.
template <int W>
__device__ __forceinline__ void load_panel(const double* G, bool contig, int ld, int X, int K, int x0, int k0,
                                           double* s) {
  const int tid = threadIdx.x;
  constexpr int IT = (W * BK) / GEMM_THREADS;
  if (contig) {  // element (x, k) at G[x + k ld]
    constexpr int KP = GEMM_THREADS / W;  // k per pass
    const int x = tid & (W - 1), kk0 = tid / W;
    const bool xok = x0 + x < X;
    const double* g = G + (x0 + x) + (i64)(k0 + kk0) * ld;
    const i64 step = (i64)KP * ld;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int kk = kk0 + KP * it;
      const bool ok = xok && (k0 + kk < K);
      cp_async8(s + panel_pos(kk, x), ok ? g : G, ok);
      g += step;
    }
  } else {  // at G[k + x ld]
    const int kk = tid & (BK - 1), xx0 = tid >> 4;
    const bool kok = k0 + kk < K;
    const double* g = G + (k0 + kk) + (i64)(x0 + xx0) * ld;
    const i64 step = (i64)8 * ld;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
      const int x = xx0 + 8 * it;
      const bool ok = kok && (x0 + x < X);
      cp_async8(s + panel_pos(kk, x), ok ? g : G, ok);
      g += step;
    }
  }
}

// Active segments of the CTA's problem, kept in shared memory.
constexpr int SEG_MAX = 8;  // problems have up to four segments, pair problems up to two (a tile pair doubles them)
struct SegList {
  GSeg seg[SEG_MAX];
  const double* A[SEG_MAX];  // operand bases (buffer + offset)
  const double* B[SEG_MAX];
  double alpha[SEG_MAX];
  int nact;
  int total;  // k-tiles over all active segments
};

// Advance a (segment, k0) cursor by one k-tile.
__device__ __forceinline__ void cursor_next(const SegList& sl, int& si, int& k0) {
  k0 += BK;
  if (k0 >= sl.seg[si].K) {
    ++si;
    k0 = 0;
  }
}

// One TM x TN tile, WM x (4 / WM) warps.
template <int TM, int TN, int WM>
struct Tile {
  static constexpr int WN = 4 / WM, MI = TM / WM / 8, NJ = TN / WN / 8;  // DMMA fragments of a warp
  double acc[MI][NJ][2];

  // Accumulate the tile (row0, col0) of problem P over the listed segments.
  __device__ __forceinline__ void mainloop(const GProb& P, const SegList& sl, int row0, int col0, double* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp % WM, wn = warp / WM;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int total = sl.total;
    if (total == 0) return;
    double* sA = smem;
    double* sB = smem + NSTAGE * PANEL;
    int ls = 0, lk = 0;  // load cursor
    int cs = 0, ck = 0;  // compute cursor
    auto load = [&](int st) {
      const GSeg& g = sl.seg[ls];
      load_panel<TM>(sl.A[ls], !g.tA, g.lda, P.M, g.K, row0, lk, sA + st * PANEL);
      load_panel<TN>(sl.B[ls], g.tB, g.ldb, P.N, g.K, col0, lk, sB + st * PANEL);
      cursor_next(sl, ls, lk);
    };
#pragma unroll
    for (int st = 0; st < NSTAGE - 1; ++st) {
      if (st < total) load(st);
      cp_commit();
    }
    for (int g = 0; g < total; ++g) {
      const int gl = g + NSTAGE - 1;
      if (gl < total) load(gl % NSTAGE);
      cp_commit();
      cp_wait<NSTAGE - 1>();
      __syncthreads();
      const double alpha = sl.alpha[cs];
      const double* a_s = sA + (g % NSTAGE) * PANEL;
      const double* b_s = sB + (g % NSTAGE) * PANEL;
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
        double af[MI], bf[NJ];
        const int kr = kk + (lane & 3);
#pragma unroll
        for (int i = 0; i < MI; ++i) af[i] = a_s[panel_pos(kr, (wm * MI + i) * 8 + (lane >> 2))];
#pragma unroll
        for (int j = 0; j < NJ; ++j) bf[j] = b_s[panel_pos(kr, (wn * NJ + j) * 8 + (lane >> 2))];
        if (alpha == -1.0) {
#pragma unroll
          for (int i = 0; i < MI; ++i) af[i] = -af[i];
        } else if (alpha != 1.0) {
#pragma unroll
          for (int i = 0; i < MI; ++i) af[i] *= alpha;
        }
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
          for (int j = 0; j < NJ; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
      }
      cursor_next(sl, cs, ck);
      __syncthreads();
    }
    cp_wait<0>();
    __syncthreads();
  }

  // accumulator fragments -> smem tile T[col * TLD + row]
  __device__ __forceinline__ void stash(double* T) const {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = warp % WM, wn = warp / WM;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int r = (wm * MI + i) * 8 + (lane >> 2), c = (wn * NJ + j) * 8 + 2 * (lane & 3);
        T[c * TLD + r] = acc[i][j][0];
        T[(c + 1) * TLD + r] = acc[i][j][1];
      }
  }
};

// Rows r < mr and columns c < nc of an R x C tile at out (leading dimension
// ld) from val(r, c): set or added; the reads of up to eight entries go out
// together.
template <int R, int CO, class F>
__device__ __forceinline__ void write_tile(double* __restrict__ out, int ld, int mr, int nc, bool acc, F val) {
  constexpr int PER = R * CO / GEMM_THREADS, CH = PER < 8 ? PER : 8;
#pragma unroll 1
  for (int k0 = 0; k0 < PER; k0 += CH) {
    double cv[CH];
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const int idx = threadIdx.x + (k0 + k) * GEMM_THREADS, r = idx % R, c = idx / R;
      cv[k] = acc && r < mr && c < nc ? out[r + (i64)c * ld] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < CH; ++k) {
      const int idx = threadIdx.x + (k0 + k) * GEMM_THREADS, r = idx % R, c = idx / R;
      if (r < mr && c < nc) out[r + (i64)c * ld] = acc ? cv[k] + val(r, c) : val(r, c);
    }
  }
}

// One task of problem P; twin: with the transposed tile.
template <int TM, int TN, int WM>
__device__ __forceinline__ void run_tile(const GProb& P, const SegList& sl, int r0, int c0, bool pair, bool twin,
                                         bool acc_mode, double sigma, double* out, double* smem) {
  Tile<TM, TN, WM> t;
  double* T = smem;  // the pipeline's buffers, free after the main loop
  t.mainloop(P, sl, r0, c0, smem);
  t.stash(T);
  __syncthreads();
  const int mr = min(TM, P.M - r0), nc = min(TN, P.N - c0);
  double* o = out + r0 + (i64)c0 * P.ldc;
  if (pair && !twin)
    write_tile<TM, TN>(o, P.ldc, mr, nc, acc_mode,
                       [&](int r, int c) { return T[c * TLD + r] + sigma * T[r * TLD + c]; });
  else
    write_tile<TM, TN>(o, P.ldc, mr, nc, acc_mode, [&](int r, int c) { return T[c * TLD + r]; });
  if (twin)
    write_tile<TN, TM>(out + c0 + (i64)r0 * P.ldc, P.ldc, nc, mr, acc_mode,
                       [&](int r, int c) { return sigma * T[r * TLD + c]; });
}

__global__ void __launch_bounds__(GEMM_THREADS, 4) k_grouped_gemm(const GTask* __restrict__ tasks,
                                                                  const GProb* __restrict__ probs,
                                                                  const GSeg* __restrict__ segs, Bufs bufs, double hv0,
                                                                  double hv1, unsigned maskA, unsigned maskB) {
  extern __shared__ double smem[];
  const GTask t = tasks[blockIdx.x];
  const GProb P = probs[t.prob];
  double* out = const_cast<double*>(bufs.p[P.outbuf]) + P.offC;
  const bool pair = P.mode == GM_ACC_PAIR || P.mode == GM_SET_PAIR;
  const bool acc_mode = P.mode == GM_ACC || P.mode == GM_ACC_PAIR;
  const int r0 = t.r0, c0 = t.c0;
  const bool twin = pair && r0 != c0;  // with the tile (J,I)
  const double sigma = pair ? P.sc * (P.spa ? hv0 : 1.0) * (P.spb ? hv1 : 1.0) : 0.0;

  __shared__ SegList sl;
  if (threadIdx.x == 0) {
    int na = 0, tot = 0;
    for (int k = 0; k < P.nseg && na < SEG_MAX; ++k) {
      const GSeg sg = segs[P.seg0 + k];
      if (!seg_active(sg, maskA, maskB) || sg.K <= 0) continue;
      const double alpha = sg.c * (sg.pa ? hv0 : 1.0) * (sg.pb ? hv1 : 1.0);
      sl.seg[na] = sg;
      sl.A[na] = bufs.p[sg.srcA] + sg.offA;
      sl.B[na] = bufs.p[sg.srcB] + sg.offB;
      sl.alpha[na] = alpha;
      tot += (sg.K + BK - 1) / BK;
      ++na;
      if (twin) {  // sigma (op(A) op(B))^T = sigma op(B)^T op(A)^T
        GSeg sw = sg;
        sw.lda = sg.ldb;
        sw.ldb = sg.lda;
        sw.tA = !sg.tB;
        sw.tB = !sg.tA;
        sl.seg[na] = sw;
        sl.A[na] = sl.B[na - 1];
        sl.B[na] = sl.A[na - 1];
        sl.alpha[na] = sigma * alpha;
        tot += (sg.K + BK - 1) / BK;
        ++na;
      }
    }
    sl.nact = na;
    sl.total = tot;
  }
  __syncthreads();
#define QD_TILE(TM, TN, WM) run_tile<TM, TN, WM>(P, sl, r0, c0, pair, twin, acc_mode, sigma, out, smem)
  switch (t.shape) {
    case tile_shape(64, 64): QD_TILE(64, 64, 2); break;
    case tile_shape(64, 32): QD_TILE(64, 32, 2); break;
    case tile_shape(64, 16): QD_TILE(64, 16, 4); break;
    case tile_shape(32, 64): QD_TILE(32, 64, 2); break;
    case tile_shape(32, 32): QD_TILE(32, 32, 2); break;
    default: QD_TILE(32, 16, 4); break;
  }
#undef QD_TILE
}

// ---------------------------------------------------------------------------
// K-short problems: every active segment together spans K <= KS_K (blocks
// with few hh pairs or few cross-coupled pairs).  Such a tile is one read-
// modify-write of C: no pipeline, the panels of all segments are staged once
// (alpha folded in), the two products of a pair tile are formed from four
// panels, and the shared memory is reused for the two transpose stashes
// (66.5 KB per CTA: three CTAs of eight warps on an SM).
// ---------------------------------------------------------------------------
constexpr int KS_K = 16, KS_THREADS = 256, KS_LDS = 68;
constexpr int KS_PANEL = KS_K * KS_LDS;                            // doubles per panel
// shared memory: stash 1 [BN*TLD] | panels A1 B1 A2 B2 (stash 2 overlaps the panels once the products are done)
constexpr int KS_PANEL0 = BN * TLD;
constexpr size_t KS_SMEM = sizeof(double) * (KS_PANEL0 + 4 * KS_PANEL > 2 * BN * TLD ? KS_PANEL0 + 4 * KS_PANEL
                                                                                      : 2 * BN * TLD);

// panel of op(A) rows [row0, row0+64) (sA[k][m]) and op(B) columns
// [col0, col0+64) (sB[k][n]) over the concatenated active segments; zeros
// outside M, N and beyond the total K
__device__ __forceinline__ void ks_panels(const SegList& sl, int M, int N, int row0, int col0, double* sA,
                                          double* sB) {
  for (int i = threadIdx.x; i < KS_PANEL; i += KS_THREADS) {
    sA[i] = 0.0;
    sB[i] = 0.0;
  }
  __syncthreads();
  int kb = 0;
  for (int si = 0; si < sl.nact; ++si) {
    const GSeg& s = sl.seg[si];
    const double* A = sl.A[si];
    const double* B = sl.B[si];
    const double al = sl.alpha[si];
    for (int e = threadIdx.x; e < s.K * BM; e += KS_THREADS) {
      // element (m or n fastest when that index is contiguous in memory)
      int m, k;
      if (!s.tA) { m = e % BM; k = e / BM; } else { k = e % s.K; m = e / s.K; }
      if (row0 + m < M) sA[(kb + k) * KS_LDS + m] = al * (s.tA ? A[k + (i64)(row0 + m) * s.lda] : A[(row0 + m) + (i64)k * s.lda]);
      int n, k2;
      if (s.tB) { n = e % BN; k2 = e / BN; } else { k2 = e % s.K; n = e / s.K; }
      if (col0 + n < N) sB[(kb + k2) * KS_LDS + n] = s.tB ? B[(col0 + n) + (i64)k2 * s.ldb] : B[k2 + (i64)(col0 + n) * s.ldb];
    }
    kb += s.K;
  }
  __syncthreads();
}

// acc[4][2][2] (warp tile 32 x 16) = sA^T sB over KS_K
__device__ __forceinline__ void ks_mma(const double* sA, const double* sB, double acc[4][2][2]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp & 1, wn = warp >> 1;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int kk = 0; kk < KS_K; kk += 4) {
    const int kr = kk + (lane & 3);
    double af[4], bf[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) af[i] = sA[kr * KS_LDS + wm * 32 + i * 8 + (lane >> 2)];
#pragma unroll
    for (int j = 0; j < 2; ++j) bf[j] = sB[kr * KS_LDS + wn * 16 + j * 8 + (lane >> 2)];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
  }
}

__device__ __forceinline__ void ks_stash(double* T, const double acc[4][2][2]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp & 1, wn = warp >> 1;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = wm * 32 + i * 8 + (lane >> 2);
      const int c = wn * 16 + j * 8 + 2 * (lane & 3);
      T[c * TLD + r] = acc[i][j][0];
      T[(c + 1) * TLD + r] = acc[i][j][1];
    }
}

__global__ void __launch_bounds__(KS_THREADS, 3) k_gemm_kshort(const GTask* __restrict__ tasks,
                                                            const GProb* __restrict__ probs,
                                                            const GSeg* __restrict__ segs, Bufs bufs, double hv0,
                                                            double hv1, unsigned maskA, unsigned maskB) {
  extern __shared__ double smem[];
  __shared__ SegList sl;
  const GTask t = tasks[blockIdx.x];
  const GProb P = probs[t.prob];
  double* out = const_cast<double*>(bufs.p[P.outbuf]) + P.offC;
  if (threadIdx.x == 0) {
    int na = 0, tot = 0;
    for (int k = 0; k < P.nseg && na < SEG_MAX; ++k) {
      const GSeg sg = segs[P.seg0 + k];
      if (!seg_active(sg, maskA, maskB) || sg.K <= 0) continue;
      sl.seg[na] = sg;
      sl.A[na] = bufs.p[sg.srcA] + sg.offA;
      sl.B[na] = bufs.p[sg.srcB] + sg.offB;
      sl.alpha[na] = sg.c * (sg.pa ? hv0 : 1.0) * (sg.pb ? hv1 : 1.0);
      tot += sg.K;
      ++na;
    }
    sl.nact = na;
    sl.total = tot;  // <= KS_K (the host routes only such problems here)
  }
  __syncthreads();
  const bool pair = P.mode == GM_ACC_PAIR || P.mode == GM_SET_PAIR;
  const bool acc_mode = P.mode == GM_ACC || P.mode == GM_ACC_PAIR;
  const int r0 = t.r0, c0 = t.c0;
  double* pA1 = smem + KS_PANEL0;
  double* pB1 = pA1 + KS_PANEL;
  double* T = smem;  // stash 1: below the panels
  double v1[4][2][2];
  if (!pair || r0 == c0) {
    ks_panels(sl, P.M, P.N, r0, c0, pA1, pB1);
    ks_mma(pA1, pB1, v1);
    __syncthreads();
    ks_stash(T, v1);
    __syncthreads();
    const double sigma = pair ? P.sc * (P.spa ? hv0 : 1.0) * (P.spb ? hv1 : 1.0) : 0.0;
    const int mr = min(BM, P.M - r0), nc = min(BN, P.N - c0);
    // read-modify-write of C: a thread's loads of a chunk first, then the stores
    constexpr int PER = BM * BN / KS_THREADS, CH = 8;
#pragma unroll
    for (int k0 = 0; k0 < PER; k0 += CH) {
      double cv[CH];
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int idx = threadIdx.x + (k0 + k) * KS_THREADS, r = idx & (BM - 1), c = idx >> 6;
        cv[k] = (acc_mode && r < mr && c < nc) ? out[(r0 + r) + (i64)(c0 + c) * P.ldc] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int idx = threadIdx.x + (k0 + k) * KS_THREADS, r = idx & (BM - 1), c = idx >> 6;
        if (r < mr && c < nc) {
          const double v = pair ? T[c * TLD + r] + sigma * T[r * TLD + c] : T[c * TLD + r];
          out[(r0 + r) + (i64)(c0 + c) * P.ldc] = acc_mode ? cv[k] + v : v;
        }
      }
    }
    return;
  }
  // off-diagonal tile pair: V(I,J) = A_I B_J^T and V(J,I) = A_J B_I^T, each
  // stashed right after its product (one accumulator live at a time), then
  // C(I,J) = V(I,J) + sigma V(J,I)^T and C(J,I) = V(J,I) + sigma V(I,J)^T
  // written column by column
  double* pA2 = pB1 + KS_PANEL;
  double* pB2 = pA2 + KS_PANEL;
  double* T1 = smem;
  double* T2 = smem + BN * TLD;  // overlaps the panels: written after every product is done
  ks_panels(sl, P.M, P.N, r0, c0, pA1, pB1);
  ks_panels(sl, P.M, P.N, c0, r0, pA2, pB2);
  ks_mma(pA1, pB1, v1);
  ks_stash(T1, v1);
  ks_mma(pA2, pB2, v1);
  __syncthreads();
  ks_stash(T2, v1);
  __syncthreads();
  const double sigma = P.sc * (P.spa ? hv0 : 1.0) * (P.spb ? hv1 : 1.0);
  const int mI = min(BM, P.M - r0), mJ = min(BM, P.M - c0);
  constexpr int PER = BM * BN / KS_THREADS;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const double* Ta = side == 0 ? T1 : T2;
    const double* Tb = side == 0 ? T2 : T1;
    const int rb = side == 0 ? r0 : c0, cb = side == 0 ? c0 : r0;
    const int mr = side == 0 ? mI : mJ, nc = side == 0 ? mJ : mI;
    constexpr int CH = 8;
#pragma unroll
    for (int k0 = 0; k0 < PER; k0 += CH) {
      double cv[CH];  // read-modify-write of C: a chunk's loads first, then its stores
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int idx = threadIdx.x + (k0 + k) * KS_THREADS, r = idx & (BM - 1), c = idx >> 6;
        cv[k] = (acc_mode && r < mr && c < nc) ? out[(rb + r) + (i64)(cb + c) * P.ldc] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < CH; ++k) {
        const int idx = threadIdx.x + (k0 + k) * KS_THREADS, r = idx & (BM - 1), c = idx >> 6;
        if (r < mr && c < nc) {
          const double x = Ta[c * TLD + r] + sigma * Tb[r * TLD + c];
          out[(rb + r) + (i64)(cb + c) * P.ldc] = acc_mode ? cv[k] + x : x;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Host side: program construction and launch
// ---------------------------------------------------------------------------
namespace {

struct Builder {
  GemmProgram& P;
  int cur = -1;
  explicit Builder(GemmProgram& p) : P(p) {}
  void prob(int M, int N, i64 offC, int ldc, int mode, int outbuf, double sc = 0.0, int spa = 0, int spb = 0) {
    GProb g;
    std::memset(&g, 0, sizeof(g));
    g.M = M;
    g.N = N;
    g.ldc = ldc;
    g.offC = offC;
    g.mode = mode;
    g.outbuf = outbuf;
    g.seg0 = (int)P.segs.size();
    g.nseg = 0;
    g.sc = sc;
    g.spa = (signed char)spa;
    g.spb = (signed char)spb;
    P.probs.push_back(g);
    cur = (int)P.probs.size() - 1;
  }
  // acc += c * hv0^pa * hv1^pb * op(A) op(B)
  void seg(int srcA, i64 offA, int lda, bool tA, int depA, int srcB, i64 offB, int ldb, bool tB, int depB, int K,
           double c, int pa = 0, int pb = 0) {
    if (K <= 0) return;
    GSeg s;
    std::memset(&s, 0, sizeof(s));
    s.offA = offA;
    s.offB = offB;
    s.lda = std::max(1, lda);
    s.ldb = std::max(1, ldb);
    s.K = K;
    s.srcA = (signed char)srcA;
    s.srcB = (signed char)srcB;
    s.tA = tA;
    s.tB = tB;
    s.depA = (signed char)depA;
    s.depB = (signed char)depB;
    s.pa = (signed char)pa;
    s.pb = (signed char)pb;
    s.c = c;
    P.segs.push_back(s);
    P.probs[cur].nseg++;
  }
  void drop_if_empty() {
    if (cur >= 0 && P.probs[cur].nseg == 0) {
      P.probs.pop_back();
      cur = -1;
    }
  }
};

// operand buffer ids
enum { BA = 0, BB = 1, BXA = 2, BXB = 3, BO0 = 4, BO1 = 5, BZ = 6 };
const bool N_ = false, T_ = true;

}  // namespace

static int upload_program(GemmProgram& P) {
  size_t pb = std::max<size_t>(1, P.probs.size()) * sizeof(GProb);
  size_t sb = std::max<size_t>(1, P.segs.size()) * sizeof(GSeg);
  QD_CUDA(cudaMalloc(&P.d_probs, pb));
  QD_CUDA(cudaMalloc(&P.d_segs, sb));
  if (!P.probs.empty())
    QD_CUDA(copy_table(P.d_probs, P.probs.data(), P.probs.size() * sizeof(GProb)));
  if (!P.segs.empty())
    QD_CUDA(copy_table(P.d_segs, P.segs.data(), P.segs.size() * sizeof(GSeg)));
  return QD_OK;
}

static int make_programs(qd_layout* L) {
  const int n = L->n, mp = L->mp;
  // ---- matrix_mult222 ladders (ACC into C) ----
  for (int gen = 0; gen < 2; ++gen) {
    GemmProgram& P = gen ? L->prog_ladder_gen : L->prog_ladder;
    Builder b(P);
    for (int q = 0; q < L->nblock; ++q) {
      const int nh = L->blk[q].x, nb = L->blk[q].y, np = L->blk[q].z;
      const i64* o = &L->boff[6 * q];
      if (gen && (nh == 0 || gen_ladder_fused(L, q))) continue;  // no hh pairs: no ladder has a live factor
      const i64 hhhh = o[0], pppp = o[1], pphh = o[2], phph = o[3], ppph = o[4], phhh = o[5];
      if (nh > 0) {  // V = -hB Bpphh^T Apphh - Ahhhh Bhhhh ; C += V + s V^T
        b.prob(nh, nh, hhhh, nh, GM_ACC_PAIR, BO0, -1.0, 1, 1);
        if (np > 0) b.seg(BB, pphh, np, T_, P_PPHH, BA, pphh, np, N_, P_PPHH, np, -1.0, 0, 1);
        b.seg(BA, hhhh, nh, N_, P_HHHH, BB, hhhh, nh, N_, P_HHHH, nh, -1.0);
        b.drop_if_empty();
      }
      if (np > 0) {  // V = -hB Apphh Bpphh^T - Bpppp Apppp
        b.prob(np, np, pppp, np, GM_ACC_PAIR, BO0, -1.0, 1, 1);
        if (nh > 0) b.seg(BA, pphh, np, N_, P_PPHH, BB, pphh, np, T_, P_PPHH, nh, -1.0, 0, 1);
        b.seg(BB, pppp, np, N_, P_PPPP, BA, pppp, np, N_, P_PPPP, np, -1.0);
        b.drop_if_empty();
      }
      if (nb > 0) {  // V = -hB (Aphhh Bphhh^T + Bppph^T Appph)
        b.prob(nb, nb, phph, nb, GM_ACC_PAIR, BO0, -1.0, 1, 1);
        if (nh > 0) b.seg(BA, phhh, nb, N_, P_PHHH, BB, phhh, nb, T_, P_PHHH, nh, -1.0, 0, 1);
        if (np > 0) b.seg(BB, ppph, np, T_, P_PPPH, BA, ppph, np, N_, P_PPPH, np, -1.0, 0, 1);
        b.drop_if_empty();
      }
      if (np > 0 && nh > 0) {  // Apppp Bpphh - Bpppp Apphh - Apphh Bhhhh + Bpphh Ahhhh
        b.prob(np, nh, pphh, np, GM_ACC, BO0);
        b.seg(BA, pppp, np, N_, P_PPPP, BB, pphh, np, N_, P_PPHH, np, 1.0);
        b.seg(BB, pppp, np, N_, P_PPPP, BA, pphh, np, N_, P_PPHH, np, -1.0);
        b.seg(BA, pphh, np, N_, P_PPHH, BB, hhhh, nh, N_, P_HHHH, nh, -1.0);
        b.seg(BB, pphh, np, N_, P_PPHH, BA, hhhh, nh, N_, P_HHHH, nh, 1.0);
        b.drop_if_empty();
      }
      if (nb > 0 && nh > 0) {  // hA Appph^T Bpphh - hB Bppph^T Apphh - Aphhh Bhhhh + Bphhh Ahhhh
        b.prob(nb, nh, phhh, nb, GM_ACC, BO0);
        if (np > 0) {
          b.seg(BA, ppph, np, T_, P_PPPH, BB, pphh, np, N_, P_PPHH, np, 1.0, 1, 0);
          b.seg(BB, ppph, np, T_, P_PPPH, BA, pphh, np, N_, P_PPHH, np, -1.0, 0, 1);
        }
        b.seg(BA, phhh, nb, N_, P_PHHH, BB, hhhh, nh, N_, P_HHHH, nh, -1.0);
        b.seg(BB, phhh, nb, N_, P_PHHH, BA, hhhh, nh, N_, P_HHHH, nh, 1.0);
        b.drop_if_empty();
      }
      if (np > 0 && nb > 0) {  // -hB Apphh Bphhh^T + hA Bpphh Aphhh^T + Apppp Bppph - Bpppp Appph
        b.prob(np, nb, ppph, np, GM_ACC, BO0);
        if (nh > 0) {
          b.seg(BA, pphh, np, N_, P_PPHH, BB, phhh, nb, T_, P_PHHH, nh, -1.0, 0, 1);
          b.seg(BB, pphh, np, N_, P_PPHH, BA, phhh, nb, T_, P_PHHH, nh, 1.0, 1, 0);
        }
        b.seg(BA, pppp, np, N_, P_PPPP, BB, ppph, np, N_, P_PPPH, np, 1.0);
        b.seg(BB, pppp, np, N_, P_PPPP, BA, ppph, np, N_, P_PPPH, np, -1.0);
        b.drop_if_empty();
      }
    }
  }
  // ---- commutator_221 intermediates (SET into w1 = BO0, w2 = BO1) ----
  {
    GemmProgram& P = L->prog_221;
    Builder b(P);
    for (int q = 0; q < L->nblock; ++q) {
      const int nh = L->blk[q].x, nb = L->blk[q].y, np = L->blk[q].z;
      const i64* o = &L->boff[6 * q];
      const i64 hhhh = o[0], pppp = o[1], pphh = o[2], phph = o[3], ppph = o[4], phhh = o[5];
      if (np * nh != 0) {
        b.prob(np, np, pppp, np, GM_SET, BO0);  // w1%Vpppp = Apphh Bpphh^T
        b.seg(BA, pphh, np, N_, P_PPHH, BB, pphh, np, T_, P_PPHH, nh, 1.0);
      }
      if (np * nb != 0) {
        b.prob(nb, nb, phph, nb, GM_SET, BO0);  // w1%Vphph = Bppph^T Appph
        b.seg(BB, ppph, np, T_, P_PPPH, BA, ppph, np, N_, P_PPPH, np, 1.0);
      }
      if (nh * np != 0) {
        b.prob(nh, nh, hhhh, nh, GM_SET, BO0);  // w1%Vhhhh = Bpphh^T Apphh
        b.seg(BB, pphh, np, T_, P_PPHH, BA, pphh, np, N_, P_PPHH, np, 1.0);
      }
      if (nh * nb != 0) {
        b.prob(nb, nb, phph, nb, GM_SET, BO1);  // w2%Vphph = Aphhh Bphhh^T
        b.seg(BA, phhh, nb, N_, P_PHHH, BB, phhh, nb, T_, P_PHHH, nh, 1.0);
      }
      if (nh * nb * np != 0) {
        b.prob(nb, nh, phhh, nb, GM_SET, BO0);  // w1%Vphhh = Bppph^T Apphh
        b.seg(BB, ppph, np, T_, P_PPPH, BA, pphh, np, N_, P_PPHH, np, 1.0);
        b.prob(nb, nh, phhh, nb, GM_SET, BO1);  // w2%Vphhh = Appph^T Bpphh
        b.seg(BA, ppph, np, T_, P_PPPH, BB, pphh, np, N_, P_PPHH, np, 1.0);
        b.prob(np, nb, ppph, np, GM_SET, BO0);  // w1%Vppph = Apphh Bphhh^T
        b.seg(BA, pphh, np, N_, P_PPHH, BB, phhh, nb, T_, P_PHHH, nh, 1.0);
        b.prob(np, nb, ppph, np, GM_SET, BO1);  // w2%Vppph = Bpphh Aphhh^T
        b.seg(BB, pphh, np, N_, P_PPHH, BA, phhh, nb, T_, P_PHHH, nh, 1.0);
      }
    }
  }
  // ---- commutator_111 (SET into C's one-body part) ----
  {
    GemmProgram& P = L->prog_111;
    Builder b(P);
    if (n > 0) {  // V = Afhh Bfhh - hB Bfph^T Afph ; fhh = V + s V^T
      b.prob(n, n, L->o_fhh, n, GM_SET_PAIR, BO0, -1.0, 1, 1);
      b.seg(BA, L->o_fhh, n, N_, P_FHH, BB, L->o_fhh, n, N_, P_FHH, n, 1.0);
      if (mp > 0) b.seg(BB, L->o_fph, mp, T_, P_FPH, BA, L->o_fph, mp, N_, P_FPH, mp, -1.0, 0, 1);
    }
    if (mp > 0) {  // V = hB Afph Bfph^T - Bfpp Afpp ; fpp = V + s V^T
      b.prob(mp, mp, L->o_fpp, mp, GM_SET_PAIR, BO0, -1.0, 1, 1);
      if (n > 0) b.seg(BA, L->o_fph, mp, N_, P_FPH, BB, L->o_fph, mp, T_, P_FPH, n, 1.0, 0, 1);
      b.seg(BB, L->o_fpp, mp, N_, P_FPP, BA, L->o_fpp, mp, N_, P_FPP, mp, -1.0);
    }
    if (mp > 0 && n > 0) {  // fph = Afph Bfhh - Bfph Afhh + Afpp Bfph - Bfpp Afph
      b.prob(mp, n, L->o_fph, mp, GM_SET, BO0);
      b.seg(BA, L->o_fph, mp, N_, P_FPH, BB, L->o_fhh, n, N_, P_FHH, n, 1.0);
      b.seg(BB, L->o_fph, mp, N_, P_FPH, BA, L->o_fhh, n, N_, P_FHH, n, -1.0);
      b.seg(BA, L->o_fpp, mp, N_, P_FPP, BB, L->o_fph, mp, N_, P_FPH, mp, 1.0);
      b.seg(BB, L->o_fpp, mp, N_, P_FPP, BA, L->o_fph, mp, N_, P_FPH, mp, -1.0);
    }
  }
  // ---- construct_cc_ints: Z = XCC - YCC = hB P - hA P^T, P = X_A X_B^T ----
  // The re-coupling adds Z of block q at [(u,x),(y,v)] to Z of the opposite
  // block qr at [(v,y),(x,u)], the reversed pairs.  With qr's rows in q's order
  // that sum is W + s W^T, W = hB X_A X_B^T of q - hA X_A X_B^T of qr: one
  // problem of q's size with both blocks' columns as its K, half the outputs
  // and half the reads of the re-coupling.  In the block of no transfer both
  // sit in the same block in different order: Z itself is stored.
  {
    GemmProgram& P = L->prog_pandya;
    Builder b(P);
    for (int q = 0; q < L->ncc; ++q) {
      const int r = L->ccdim[q].x, nb = L->ccdim[q].y, qr = L->ncc - 1 - q;
      if (r == 0 || q < qr) continue;
      b.prob(r, r, L->cczoff[q], r, GM_SET_PAIR, BZ, -1.0, 1, 1);  // nb == 0 writes zeros
      if (nb > 0) b.seg(BXA, L->ccxoff[q], r, N_, -1, BXB, L->ccxoff[q], r, T_, -1, nb, 1.0, 0, 1);
      if (q > qr) b.seg(BXA, L->ccxoff[qr], r, N_, -1, BXB, L->ccxoff[qr], r, T_, -1, L->ccdim[qr].y, -1.0, 1, 0);
    }
  }
  for (GemmProgram* P : {&L->prog_ladder, &L->prog_ladder_gen, &L->prog_221, &L->prog_111, &L->prog_pandya}) {
    const int rc = upload_program(*P);
    if (rc) return rc;
  }
  QD_CUDA(cudaFuncSetAttribute(k_grouped_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM));
  QD_CUDA(cudaFuncSetAttribute(k_gemm_kshort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KS_SMEM));
  return QD_OK;
}

// All programs of the layout or, on failure, none: the next call starts anew.
int build_programs(qd_layout* L) {
  if (L->programs_built) return QD_OK;
  const int rc = make_programs(L);
  if (!rc) {
    L->programs_built = true;
    return QD_OK;
  }
  for (GemmProgram* P : {&L->prog_ladder, &L->prog_ladder_gen, &L->prog_221, &L->prog_111, &L->prog_pandya}) {
    P->clear_device();
    P->probs.clear();
    P->segs.clear();
  }
  return rc;
}

// The products of the particle-hole channel of a generator-like A (ph_gen.cu)
int build_ph_products(qd_layout* L, const std::vector<PhProduct>& v, GemmProgram& P) {
  (void)L;
  Builder b(P);
  for (const PhProduct& x : v) {
    b.prob(x.r, x.rows, x.offY, x.r, GM_SET, BZ);  // nb == 0 writes zeros
    b.seg(BXB, x.offB, x.r, N_, -1, BXA, x.offA, x.rows, T_, -1, x.nb, 1.0);
  }
  return upload_program(P);
}

// Ladder sums of the EOM product for a non-scalar target (eom.cu): per bra
// block q with ket block partner[q] (pairs of M_q minus the target), the
// npp(q) x nhh(partner[q]) output Wb[q] = Vpppp[q] Qb[q] + Qb[q] Vhhhh[partner[q]]
// (the c<d and k<l sums of HQ_comm_2b, src/commutators.f90:1246-1258).
// Buffers: H = BA, the amplitude matrices Qb = BB, the output Wb = BO0.
int build_eom_ladders(qd_layout* L, const std::vector<int>& partner, const std::vector<i64>& qoff, GemmProgram& P) {
  Builder b(P);
  for (int q = 0; q < L->nblock; ++q) {
    const int q2 = partner[q];
    if (q2 < 0) continue;
    const int np = L->blk[q].z, nh2 = L->blk[q2].x;
    if (np == 0 || nh2 == 0) continue;
    b.prob(np, nh2, qoff[q], np, GM_SET, BO0);
    b.seg(BA, L->boff[6 * q + 1], np, N_, P_PPPP, BB, qoff[q], np, N_, -1, np, 1.0);
    b.seg(BB, qoff[q], np, N_, -1, BA, L->boff[6 * q2 + 0], nh2, N_, P_HHHH, nh2, 1.0);
  }
  return upload_program(P);
}

static bool seg_active_host(const GSeg& s, unsigned mA, unsigned mB) {
  auto dead = [&](int src, int dep) {
    if (dep < 0) return false;
    unsigned m = src == 0 ? mA : (src == 1 ? mB : 0u);
    return ((m >> dep) & 1u) != 0;
  };
  return !dead(s.srcA, s.depA) && !dead(s.srcB, s.depB);
}

// Starts and widths of the tiles along n entries: full tiles of `w` and one
// rest of the narrowest width that holds it (of 64, 32 and, where `least` is
// 16, 16): n_h-column outputs are mostly padding in 64-wide tiles.  At N=20,
// R=20 the ladders' padded work falls from 1.22 to 1.11 times the real one.
static std::vector<std::pair<int, int>> cuts(int n, int w, int least) {
  std::vector<std::pair<int, int>> v;
  for (int x = 0; x < n; x += w) {
    int c = w;
    while (c > least && n - x <= c / 2) c /= 2;
    v.push_back({x, c});
  }
  return v;
}

// Host task lists of P for (mA, mB): [0] long-K problems, [1] K-short ones,
// each as (cost, task), longest first.  Every tile (tile pair in the pair
// modes) of every problem that has an active segment (SET problems always:
// they must write); problems whose active segments span K <= KS_K (at most
// 8 of them) go to the K-short kernel.  Tiles are 64 wide; where these are
// fewer than FEW_TILES (the chip holds 592 CTAs), 32: a tile's products take
// the same time on one SM however many SMs are idle.
constexpr size_t FEW_TILES = 1184;
static void task_vectors(const GemmProgram& P, unsigned mA, unsigned mB, std::vector<std::pair<double, GTask>> v[2]) {
  for (int w : {64, 32}) {
    v[0].clear();
    v[1].clear();
    for (size_t pi = 0; pi < P.probs.size(); ++pi) {
      const GProb& g = P.probs[pi];
      double kt = 0.0;
      int ksum = 0, nact = 0;
      for (int k = 0; k < g.nseg; ++k) {
        const GSeg& s = P.segs[g.seg0 + k];
        if (seg_active_host(s, mA, mB) && s.K > 0) {
          kt += (s.K + BK - 1) / BK;
          ksum += s.K;
          ++nact;
        }
      }
      const bool set = g.mode == GM_SET || g.mode == GM_SET_PAIR;
      if (kt == 0.0 && !set) continue;
      const int which = (ksum <= KS_K && nact <= 8) ? 1 : 0;
      const bool pair = g.mode == GM_ACC_PAIR || g.mode == GM_SET_PAIR;
      // the K-short kernel has 64 x 64 tiles only; a pair's rows and columns are cut alike
      const auto rows = which ? cuts(g.M, 64, 64) : cuts(g.M, w, 32);
      const auto cols = which ? cuts(g.N, 64, 64) : cuts(g.N, w, pair ? 32 : 16);
      for (size_t i = 0; i < rows.size(); ++i)
        for (size_t j = pair ? i : 0; j < cols.size(); ++j) {
          GTask t;
          t.prob = (int)pi;
          t.r0 = rows[i].first;
          t.c0 = cols[j].first;
          t.shape = tile_shape(rows[i].second, cols[j].second);
          const double area = rows[i].second * cols[j].second / 4096.0;
          v[which].push_back({(kt + 1.0) * ((pair && i != j) ? 2.0 : 1.0) * (which ? 1.0 : area + 0.1), t});
        }
    }
    if (v[0].size() >= FEW_TILES) break;
  }
  for (int w = 0; w < 2; ++w)
    std::stable_sort(v[w].begin(), v[w].end(), [](const auto& a, const auto& b) { return a.first > b.first; });
}

static int get_tasks(qd_layout* L, GemmProgram& P, unsigned mA, unsigned mB, GTask** d_tasks, int* ntasks,
                     GTask** d_short, int* nshort) {
  (void)L;
  auto key = std::make_pair(mA, mB);
  auto it = P.tasks.find(key);
  if (it != P.tasks.end()) {
    *d_tasks = it->second.first;
    *ntasks = it->second.second;
    *d_short = P.tasks_short[key].first;
    *nshort = P.tasks_short[key].second;
    return QD_OK;
  }
  std::vector<std::pair<double, GTask>> v[2];
  task_vectors(P, mA, mB, v);
  GTask* d[2] = {nullptr, nullptr};
  for (int w = 0; w < 2; ++w) {
    std::vector<GTask> h(v[w].size());
    for (size_t i = 0; i < v[w].size(); ++i) h[i] = v[w][i].second;
    if (h.empty()) continue;
    cudaError_t e = cudaMalloc(&d[w], h.size() * sizeof(GTask));
    if (e == cudaSuccess) e = copy_table(d[w], h.data(), h.size() * sizeof(GTask));
    if (e != cudaSuccess) {
      for (GTask* p : d)
        if (p) cudaFree(p);
      return cuda_fail(e, "task lists");
    }
  }
  P.tasks[key] = std::make_pair(d[0], (int)v[0].size());
  P.tasks_short[key] = std::make_pair(d[1], (int)v[1].size());
  *d_tasks = d[0];
  *ntasks = (int)v[0].size();
  *d_short = d[1];
  *nshort = (int)v[1].size();
  return QD_OK;
}

// Build (allocate and upload) the task lists of P for a pair of zero-part
// masks ahead of a stream capture, which must not allocate.
int prepare_program(qd_layout* L, GemmProgram& P, unsigned maskA, unsigned maskB) {
  int rc = build_programs(L);
  if (rc) return rc;
  GTask *d1, *d2;
  int n1, n2;
  return get_tasks(L, P, maskA, maskB, &d1, &n1, &d2, &n2);
}

int run_program(qd_layout* L, GemmProgram& P, const double* const* bufs, double hv0, double hv1, unsigned maskA,
                unsigned maskB) {
  int rc = build_programs(L);
  if (rc) return rc;
  if (L->split_slices > 0) return run_program_split(L, P, bufs, hv0, hv1, maskA, maskB);
  return run_program_f64(L, P, bufs, hv0, hv1, maskA, maskB);
}

// P in FP64 on the DMMA pipe whatever the layout's form (P's tables must be
// on the device: build_programs or build_eom_ladders).
int run_program_f64(qd_layout* L, GemmProgram& P, const double* const* bufs, double hv0, double hv1, unsigned maskA,
                    unsigned maskB) {
  int rc = build_programs(L);  // sets the kernels' shared-memory limits
  if (rc) return rc;
  GTask *d_tasks = nullptr, *d_short = nullptr;
  int nt = 0, ns = 0;
  if ((rc = get_tasks(L, P, maskA, maskB, &d_tasks, &nt, &d_short, &ns))) return rc;
  Bufs b;
  for (int i = 0; i < NBUF; ++i) b.p[i] = bufs[i];
  if (nt > 0) {
    k_grouped_gemm<<<nt, GEMM_THREADS, GEMM_SMEM, L->stream>>>(d_tasks, P.d_probs, P.d_segs, b, hv0, hv1, maskA,
                                                                maskB);
    ++L->nlaunch;
  }
  if (ns > 0) {
    k_gemm_kshort<<<ns, KS_THREADS, KS_SMEM, L->stream>>>(d_short, P.d_probs, P.d_segs, b, hv0, hv1, maskA, maskB);
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

}  // namespace qd
