// kernels_122.cu -- commutator_122 (src/commutators.f90:355-676) as one pass
// over independent group-pair tiles.
//
// In block q the pairs are ordered [hh | ph | pp]; the full block matrix
// V(P1,P2) holds the stored classes (class(P1) >= class(P2)) and herm * their
// transposes above.  For the stored output element <b1 b2|k1 k2> = C(P1,P2):
//   bra legs: C += sum_{t in G(b1)} [FA(b1,t) VB(t b2|P2) - FB(b1,t) VA(t b2|P2)]
//                + sum_{t in G(b2)} [FA(b2,t) VB(b1 t|P2) - FB(b2,t) VA(b1 t|P2)]
//   ket legs: C -= sum_{t in G(k1)} [FA'(k1,t) VB(P1|t k2) - FB'(k1,t) VA(P1|t k2)]
//                + sum_{t in G(k2)} [FA'(k2,t) VB(P1|k1 t) - FB'(k2,t) VA(P1|k1 t)]
// G(x) = states with the (m_l, m_s) of x: the only t whose pair (t,b2) lies in
// block q.  F/F' are the reference's one-body reads (see dev_common.cuh).
//
// Group pairs.  The pairs of block q split into the sets S(g,h) of pairs with
// one state in (m_l,m_s) group g and one in group h (g <= h).  A bra leg of
// a pair in S(g,h) replaces a state by another of the same group, so it stays
// in S(g,h); a ket leg likewise stays in the column pair's set.  Hence the
// block matrix splits into tiles S_a x S_b, and C on tile (a,b) depends only
// on A and B on the same tile and on four small one-body matrices:
//   C[S_a, S_b] = (F_g (x) 1 + 1 (x) F_h) T  -  T (F'_g' (x) 1 + 1 (x) F'_h')^T
// with T the tile in "cell" coordinates: S(g,h) indexed by cells (k1,k2) <->
// (G_g[k1], G_h[k2]), T = +-V of the stored pair (the sign orients the pair;
// when g = h both orientations (k1,k2), (k2,k1) are cells and (k,k) is 0).
//
// Kernel: one CTA per tile.  The tile of each operand needed is gathered with
// cp.async into shared memory (rows of one class of S_a are runs of
// consecutive stored rows, so the gathers coalesce in runs), the orientation
// and herm signs are applied in place, then every stored output cell sums its
// four legs from shared memory and is written once.  C is written exactly
// once (122 overwrites the two-body part), A and B are read once, apart from
// the off-diagonal class blocks, which tiles (a,b) and (b,a) both read.
// When an operand's one-body part has no hh and no pp entries (the Magnus
// generator Omega), F couples holes to particles only: a leg of a hole sums
// over the particles of its group and a leg of a particle over its holes
// (holes are the lowest members of every group).  Tiles whose parts of A are
// known to be zero skip the A term (and then stage B alone).
#include <algorithm>
#include <map>
#include <cstdio>
#include <mutex>
#include <string>
#include <type_traits>

#include "dev_common.cuh"

namespace qd {

#ifndef TRY
#define TRY(x)           \
  do {                   \
    int rc_ = (x);       \
    if (rc_) return rc_; \
  } while (0)
#endif

constexpr size_t SMEM_MAX_122 = 227 * 1024;       // opt-in shared memory per CTA on sm_100

// vectorize slot of the stored part (row class c1 >= column class c2):
// (0,0) hhhh 0, (2,2) pppp 1, (2,0) pphh 2, (1,1) phph 3, (2,1) ppph 4, (1,0) phhh 5
__host__ __device__ __forceinline__ int slot_of(int c1, int c2) {
  if (c1 == 0) return 0;
  if (c1 == 1) return c2 == 0 ? 5 : 3;
  return c2 == 0 ? 2 : (c2 == 1 ? 4 : 1);
}
__device__ __forceinline__ int cnt_of(int c, int4 bd) { return c == 0 ? bd.x : (c == 1 ? bd.y : bd.z); }

// Group-pair descriptor (two int4 per group pair u):
//   d0 = {q, n1 | n2 << 8 | (g == h) << 16, holes(g) | holes(h) << 8, F offset of g}
//   d1 = {F offset of h, first pair entry, 0, cnt_hh | cnt_ph << 10 | cnt_pp << 20}
// Pair entries (int2, sorted by class then index within the class):
//   {index w within its class, primary cell | (mirror cell + 1) << 8 | (sign < 0) << 16 |
//    k1 << 17 | k2 << 21}, the primary cell being (k1, k2) = k1 * n2 + k2
struct GpDesc {
  int q, n1, n2, hg, hh, fg, fh, pstart, cntw;
  bool same;  // g == h
  // pairs of class c (0 hh, 1 ph, 2 pp), decoded from the packed word (no local array)
  __device__ __forceinline__ int cnt(int c) const { return (cntw >> (10 * c)) & 0x3FF; }
  // pairs of the classes before c
  __device__ __forceinline__ int off(int c) const { return c == 0 ? 0 : (c == 1 ? cnt(0) : cnt(0) + cnt(1)); }
};
__device__ __forceinline__ GpDesc load_gp(const int4* __restrict__ gpd, int u) {
  const int4 a = __ldg(&gpd[2 * u]), b = __ldg(&gpd[2 * u + 1]);
  GpDesc d;
  d.q = a.x;
  d.n1 = a.y & 0xFF;
  d.n2 = (a.y >> 8) & 0xFF;
  d.same = (a.y >> 16) & 1;
  d.hg = a.z & 0xFF;
  d.hh = (a.z >> 8) & 0xFF;
  d.fg = a.w;
  d.fh = b.x;
  d.pstart = b.y;
  d.cntw = b.w;
  return d;
}

// Static tables of a layout (built once, see plan_122):
//   sbase[s] = offset of state s's row in the group-major F table
// Per call: F table [2][nfent] double2 (FA, FB) bra, then (FA', FB') ket,
// group-major: F[goff_g + k1' * |G_g| + k].
__global__ void k_ftab(DevLayout L, const int* __restrict__ sbase, const double* __restrict__ A, double hA,
                       const double* __restrict__ B, double hB, double2* __restrict__ F, int gmax, int nfent) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= L.m * gmax) return;
  int s = e / gmax, k = e % gmax;
  int g = __ldg(&L.gid[s]);
  int b = __ldg(&L.gstart[g]), sz = __ldg(&L.gstart[g + 1]) - b;
  if (k >= sz) return;
  const int t = __ldg(&L.gmem[b + k]);
  double fab, fbb, fak, fbk;
  if (t < L.n) {
    const double xa = f_hole(L, A, s, t), xb = f_hole(L, B, s, t);
    fab = xa; fbb = xb; fak = hA * xa; fbk = hB * xb;
  } else {
    const double xa = f_part(L, A, t, s), xb = f_part(L, B, t, s);
    fab = hA * xa; fbb = hB * xb; fak = xa; fbk = xb;
  }
  const int pos = __ldg(&sbase[s]) + k;
  F[pos] = make_double2(fab, fbb);
  F[nfent + pos] = make_double2(fak, fbk);
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// q = a / b and r = a % b for 0 <= a < 2^22 - 1 and b >= 1, through one
// single-precision reciprocal instead of an integer division: the exact value
// of (a + 1/2) / b is q + (r + 1/2) / b, at least 1/(2b) away from an integer,
// and the two correctly rounded float operations err by at most
// (a + 1/2) / b * 2^-23 < 1/(2b); so truncation gives q.
__device__ __forceinline__ int2 divmod_small(int a, int b) {
  const int q = __float2int_rz(((float)a + 0.5f) * __frcp_rn((float)b));
  return make_int2(q, a - q * b);
}

template <int TW>
__device__ __forceinline__ constexpr int xb_of() { return TW == 2 ? 1 : 0; }

// class of a pair from the kinds of its two states: 0 hh, 1 ph, 2 pp
__host__ __device__ __forceinline__ int pair_class(bool hole1, bool hole2) { return (hole1 ? 0 : 1) + (hole2 ? 0 : 1); }

// Whether a leg's sum over the holes (t_hole) or the particles of its group
// can add anything: the one-body factor F(k, t) of a sparse operand (no hh
// and pp entries) couples a hole k only to particles t and a particle only to
// holes; the staged operand must be able to be non-zero on the cells reached,
// whose class pair is (class of (t, other), fixed class) -- nz holds one bit
// per class pair (c1 * 3 + c2, symmetric) of the operand's non-zero parts.
__host__ __device__ __forceinline__ bool leg_ok(int sparse, bool k_hole, bool t_hole, bool other_hole, int cfix,
                                                unsigned nz) {
  if (sparse && k_hole == t_hole) return false;
  return (nz >> (pair_class(t_hole, other_hole) * 3 + cfix)) & 1u;
}

// Bit 31 of a term's leg mask: its one-body factor couples holes to
// particles only, so every leg changes the class of the pair it acts on.
constexpr unsigned LEG_SPARSE = 1u << 31;

// Regions (c1 * 3 + c2) of the staged operand that the legs of a tile read
// when every leg changes the class of its pair by one: the four neighbours of
// each stored output region (c1 >= c2) of the tile.
// All regions otherwise.
__device__ __forceinline__ unsigned regions_read(unsigned leg, const int ca[3], const int cb[3]) {
  if (!(leg & LEG_SPARSE)) return 0x1FFu;
  unsigned need = 0;
  for (int c1 = 0; c1 < 3; ++c1)
    for (int c2 = 0; c2 <= c1; ++c2) {
      if (ca[c1] == 0 || cb[c2] == 0) continue;
      if (c1 > 0) need |= 1u << ((c1 - 1) * 3 + c2);
      if (c1 < 2) need |= 1u << ((c1 + 1) * 3 + c2);
      if (c2 > 0) need |= 1u << (c1 * 3 + c2 - 1);
      if (c2 < 2) need |= 1u << (c1 * 3 + c2 + 1);
    }
  return need;
}

// Sum over t of F(k, t) T[base + t * stride] for one leg: F(k, .) is the
// leg's one-body row (component fy: 0 FA, 1 FB), t runs over the holes
// [0, h) of the leg's group when bit 1 of ok is set and over its particles
// [h, n) when bit 0 is set.
__device__ __forceinline__ double leg_sum(const double2* __restrict__ Frow, int fy, const double* __restrict__ T,
                                          int base, int stride, int n, int h, unsigned ok) {
  const int lo = (ok & 2u) ? 0 : h, hi = (ok & 1u) ? n : h;
  const double* Fd = reinterpret_cast<const double*>(Frow) + fy;
  double y = 0.0;
  for (int t = lo; t < hi; ++t) y += Fd[2 * t] * T[base + t * stride];
  return y;
}

// Task: {tile, op}; op bit 0: the B term (FA x TB), bit 1: the A term
// (-FB x TA), bit 2: accumulate into C instead of setting it.  op & 3 == 0
// writes zeros.  TW = doubles per staged cell: 1 (one operand), 2 (A and B);
// T122 = threads per CTA (picked per launch bucket by the autotuner below).
template <int TW, int T122>
__global__ void __launch_bounds__(T122, 1024 / T122) k_122_tile(DevLayout L, const int2* __restrict__ tasks,
                                                   const int2* __restrict__ tiles, const int4* __restrict__ gpd,
                                                   const int2* __restrict__ gpp,
                                                   const double2* __restrict__ F, int nfent,
                                                   const double* __restrict__ A, double hA, unsigned zA, unsigned legA,
                                                   const double* __restrict__ B, double hB, unsigned zB, unsigned legB,
                                                   double* __restrict__ C) {
  extern __shared__ __align__(16) double sm122[];
  const int2 task = tasks[blockIdx.x];
  const int2 tl = __ldg(&tiles[task.x]);
  const int op = task.y;
  const bool useB = op & 1, useA = (op >> 1) & 1, acc = (op >> 2) & 1;
  const GpDesc da = load_gp(gpd, tl.x), db = load_gp(gpd, tl.y);
  const int q = da.q;
  const int n1 = da.n1, n2 = da.n2, n3 = db.n1, n4 = db.n2;
  const int nr = n1 * n2, nc = n3 * n4, ld = nc | 1;
  const int pa = da.cnt(0) + da.cnt(1) + da.cnt(2), pb = db.cnt(0) + db.cnt(1) + db.cnt(2);
  const int4 bd = __ldg(&L.blk[q]);
  const i64* boff = L.boff + 6 * q;
  // shared memory: T [nr][ld][TW] | F1 F2 F3 F4 (double2) | row, column pairs (int2)
  double* T = sm122;
  const int tsz = (nr * ld * TW + 1) & ~1;
  double2* F1 = reinterpret_cast<double2*>(sm122 + tsz);
  double2* F2 = F1 + n1 * n1;
  double2* F3 = F2 + n2 * n2;
  double2* F4 = F3 + n3 * n3;
  const int tid = threadIdx.x;
  const bool work = useA || useB;
  // a task that writes zeros stages nothing: its shared memory holds the pair lists alone
  int2* pr = work ? reinterpret_cast<int2*>(F4 + n4 * n4) : reinterpret_cast<int2*>(sm122);
  int2* pc = pr + pa;

  if (work) {
    for (int i = tid; i < n1 * n1; i += T122) F1[i] = __ldg(&F[da.fg + i]);
    for (int i = tid; i < n2 * n2; i += T122) F2[i] = __ldg(&F[da.fh + i]);
    for (int i = tid; i < n3 * n3; i += T122) F3[i] = __ldg(&F[nfent + db.fg + i]);
    for (int i = tid; i < n4 * n4; i += T122) F4[i] = __ldg(&F[nfent + db.fh + i]);
  }
  for (int i = tid; i < pa; i += T122) pr[i] = __ldg(&gpp[da.pstart + i]);
  for (int i = tid; i < pb; i += T122) pc[i] = __ldg(&gpp[db.pstart + i]);
  __syncthreads();

  if (work) {
    // Cells that no stored element reaches -- the (t,t) cells of g = h and
    // the parts known to be zero -- stay 0: zero the tile first.
    for (int i = 2 * tid; i < tsz; i += 2 * T122) *reinterpret_cast<double2*>(T + i) = make_double2(0.0, 0.0);
    __syncthreads();
    // gather: region (c1 rows of S_a, c2 columns of S_b); the stored element
    // is (P1,P2) of part (c1,c2) when c1 >= c2, else (P2,P1) of part (c2,c1),
    // taken with herm.  It lands on its cell with the orientation sign of the
    // two pairs, and on the mirror cells (g = h) with the opposite ones.
    // The loops stay rolled: the kernel's code must fit the instruction cache.
    int ca[3], cb[3];
    for (int c = 0; c < 3; ++c) {
      ca[c] = da.cnt(c);
      cb[c] = db.cnt(c);
    }
#pragma unroll 1
    for (int x = 0; x < 2; ++x) {
      if (x == 0 ? !useA : !useB) continue;
      const double* src = x == 0 ? A : B;
      const unsigned zm = x == 0 ? zA : zB;
      // the A term's legs carry FB (legA), the B term's FA (legB)
      const unsigned need = regions_read(x == 0 ? legA : legB, ca, cb);
      const double hx = x == 0 ? hA : hB;
      const int xo = TW == 2 ? x : 0;
#pragma unroll 1
      for (int rg = 0; rg < 9; ++rg) {
        const int c1 = rg / 3, c2 = rg - 3 * c1;
        const int r1 = da.cnt(c1), r2 = db.cnt(c2);
        const bool lower = c1 >= c2;
        const int part = lower ? slot_of(c1, c2) : slot_of(c2, c1);
        if (r1 == 0 || r2 == 0 || ((zm >> (P_HHHH + part)) & 1u) || !((need >> rg) & 1u)) continue;
        const int o1 = da.off(c1), o2 = db.off(c2);
        const double* srcp = src + __ldg(boff + part);
        const i64 ldv = lower ? cnt_of(c1, bd) : cnt_of(c2, bd);
        const double hf = lower ? 1.0 : hx;
        const int total = r1 * r2;
        // e = fast + nf * slow, walked without dividing: the memory-contiguous
        // index (rows for stored parts, columns for transposed ones) is fast
        const int nf = lower ? r1 : r2;
        const int2 i0 = divmod_small(tid, nf), di = divmod_small(T122, nf);
        int fa = i0.y, sl = i0.x;
        const int dfa = di.y, dsl = di.x;
#pragma unroll 4
        for (int e = tid; e < total; e += T122) {
          const int p = lower ? fa : sl, u = lower ? sl : fa;
          fa += dfa;
          sl += dsl;
          if (fa >= nf) {
            fa -= nf;
            ++sl;
          }
          const int2 P = pr[o1 + p], Q = pc[o2 + u];
          const i64 addr = lower ? P.x + (i64)Q.x * ldv : Q.x + (i64)P.x * ldv;
          const double v = hf * __ldg(srcp + addr);
          const double sv = ((P.y ^ Q.y) & (1 << 16)) ? -v : v;
          const int r = P.y & 0xFF, rm = ((P.y >> 8) & 0xFF) - 1;
          const int s = Q.y & 0xFF, sm = ((Q.y >> 8) & 0xFF) - 1;
          T[(r * ld + s) * TW + xo] = sv;
          if (rm >= 0) T[(rm * ld + s) * TW + xo] = -sv;
          if (sm >= 0) {
            T[(r * ld + sm) * TW + xo] = -sv;
            if (rm >= 0) T[(rm * ld + sm) * TW + xo] = sv;
          }
        }
      }
    }
    __syncthreads();
  }

  // stored output cells: regions with c1 >= c2, rows of S_a fastest
#pragma unroll 1
  for (int rg = 0; rg < 6; ++rg) {
    const int c1 = rg < 1 ? 0 : (rg < 3 ? 1 : 2), c2 = rg - (c1 * (c1 + 1)) / 2;  // (0,0) (1,0) (1,1) (2,0) (2,1) (2,2)
    const int r1 = da.cnt(c1), r2 = db.cnt(c2);
    if (r1 == 0 || r2 == 0) continue;
    const int o1 = da.off(c1), o2 = db.off(c2);
    const i64 base = __ldg(boff + slot_of(c1, c2));
    const i64 ldc = cnt_of(c1, bd);
    // leg masks of this region (see leg_masks): bra legs fix class c2, ket legs c1
    const unsigned okB = ((legB >> (8 * c2)) & 0xFFu) | (((legB >> (8 * c1)) & 0xFFu) << 8);
    const unsigned okA = ((legA >> (8 * c2)) & 0xFFu) | (((legA >> (8 * c1)) & 0xFFu) << 8);
    const int2 i0 = divmod_small(tid, r1), di = divmod_small(T122, r1);
    int p = i0.y, u = i0.x;
    const int dp = di.y, du = di.x;
    for (int e = tid; e < r1 * r2; e += T122) {
      const int2 P = pr[o1 + p], Q = pc[o2 + u];
      p += dp;
      u += du;
      if (p >= r1) {
        p -= r1;
        ++u;
      }
      double y = 0.0;
      if (work) {
        const int r = P.y & 0xFF, s = Q.y & 0xFF;
        const int k1 = (P.y >> 17) & 15, k2 = (P.y >> 21) & 15;
        const int l1 = (Q.y >> 17) & 15, l2 = (Q.y >> 21) & 15;
        const int h1 = k1 < da.hg, h2 = k2 < da.hh, h3 = l1 < db.hg, h4 = l2 < db.hh;
        const int b1 = h1 * 4 + h2 * 2, b2 = h2 * 4 + h1 * 2, b3 = 8 + h3 * 4 + h4 * 2, b4 = 8 + h4 * 4 + h3 * 2;
        const int bL1 = (k2 * ld + s) * TW, sL1 = n2 * ld * TW;  // T((t,k2), s)
        const int bL2 = (k1 * n2 * ld + s) * TW, sL2 = ld * TW;  // T((k1,t), s)
        const int bL3 = (r * ld + l2) * TW, sL3 = n4 * TW;       // T(r, (t,l2))
        const int bL4 = (r * ld + l1 * n4) * TW, sL4 = TW;       // T(r, (l1,t))
        if (useB) {  // FA x TB
          const double* Tb = T + xb_of<TW>();
          y += leg_sum(F1 + k1 * n1, 0, Tb, bL1, sL1, n1, da.hg, okB >> b1);
          y += leg_sum(F2 + k2 * n2, 0, Tb, bL2, sL2, n2, da.hh, okB >> b2);
          y -= leg_sum(F3 + l1 * n3, 0, Tb, bL3, sL3, n3, db.hg, okB >> b3);
          y -= leg_sum(F4 + l2 * n4, 0, Tb, bL4, sL4, n4, db.hh, okB >> b4);
        }
        if (useA) {  // -FB x TA
          y -= leg_sum(F1 + k1 * n1, 1, T, bL1, sL1, n1, da.hg, okA >> b1);
          y -= leg_sum(F2 + k2 * n2, 1, T, bL2, sL2, n2, da.hh, okA >> b2);
          y += leg_sum(F3 + l1 * n3, 1, T, bL3, sL3, n3, db.hg, okA >> b3);
          y += leg_sum(F4 + l2 * n4, 1, T, bL4, sL4, n4, db.hh, okA >> b4);
        }
        if ((P.y ^ Q.y) & (1 << 16)) y = -y;
      }
      double* out = C + base + P.x + (i64)Q.x * ldc;
      if (acc)
        *out += y;
      else
        *out = y;
    }
  }
}

// ---- the same tiles with the legs from registers --------------------------
// k_122_tile above sums each output cell's legs by itself: two shared-memory
// reads per product.  k_122_full turns a leg into small matrix products: for
// a fixed other index a thread loads the leg's n values of T once and forms
// all n outputs from them, F read as a broadcast shared by the warp, and adds
// them into a tile Y in shared memory.  Per leg and cell: one read of T, n / 2
// broadcast reads and n products per operand, one read and write of Y.  Both
// operands are staged together (24 bytes a cell, five barriers a tile) where
// at least two such tiles fit an SM, else one after the other in the same
// space (16 bytes a cell).  Bound: shared-memory bandwidth, the FP64 pipe, and
// for small tiles the chain of barriers.  Legs known to vanish are not skipped
// one by one: for an operand whose one-body part couples holes to particles
// only, large bases keep k_122_tile (see use_full).  Measured on two dense
// operators (us): N=20 R=20 4380 with k_122_tile, 3060 with this kernel (3290
// and 3150 with both operands staged up to 30 and 48 KB, 3450 up to 112 KB);
// N=6 R=10 81 and 71; N=2 R=3 37 and 14.
// CTA sizes before tuning and launch buckets, by shared memory.
constexpr size_t FULL_SMALL = 24 * 1024, FULL_BOTH = 72 * 1024;  // beyond FULL_BOTH one operand at a time
constexpr size_t FULL_BOUNDS[6] = {6 * 1024, 12 * 1024, FULL_SMALL, FULL_BOTH, FULL_BOTH + 64 * 1024, FULL_BOTH + 112 * 1024};

// Y[base + k st] (+)= sum over operands and t of F[k np + t] T[base + t st],
// k, t < n = N, np = N rounded up to even: one leg for the item (its other
// indices) at base.  BOTH: the second operand's T lies ts after the first's,
// its F fs after.
template <int N, bool BOTH>
__device__ __forceinline__ void full_leg_n(const double* __restrict__ T, int ts, double* __restrict__ Y,
                                           const double* __restrict__ F, int fs, int base, int st, bool first) {
  constexpr int NP = (N + 1) & ~1;
  double v[NP], u[BOTH ? NP : 1];
#pragma unroll
  for (int t = 0; t < N; ++t) {
    v[t] = T[base + t * st];
    if (BOTH) u[t] = T[ts + base + t * st];
  }
  if (NP > N) {
    v[NP - 1] = 0.0;
    if (BOTH) u[NP - 1] = 0.0;
  }
  const double2* f = reinterpret_cast<const double2*>(F);
  const double2* h = reinterpret_cast<const double2*>(F + fs);
#pragma unroll 2
  for (int k = 0; k < N; ++k) {
    double* y = Y + base + k * st;
    double a = first ? 0.0 : *y, b = 0.0;
#pragma unroll
    for (int t = 0; t < NP / 2; ++t) {
      const double2 w = f[k * (NP / 2) + t];
      a += w.x * v[2 * t];
      b += w.y * v[2 * t + 1];
      if (BOTH) {
        const double2 z = h[k * (NP / 2) + t];
        a += z.x * u[2 * t];
        b += z.y * u[2 * t + 1];
      }
    }
    *y = a + b;
  }
}

// All items of a leg: e = fast + nf * slow -> base = fast * sf + slow * ss.
template <int N, int NT, bool BOTH>
__device__ __forceinline__ void full_leg(const double* T, int ts, double* Y, const double* F, int fs, int nf, int ns,
                                         int sf, int ss, int st, bool first) {
  const int2 i0 = divmod_small(threadIdx.x, nf), di = divmod_small(NT, nf);
  int fa = i0.y, sl = i0.x;
  while (sl < ns) {
    full_leg_n<N, BOTH>(T, ts, Y, F, fs, fa * sf + sl * ss, st, first);
    fa += di.y;
    sl += di.x;
    if (fa >= nf) {
      fa -= nf;
      ++sl;
    }
  }
}

template <int NT, bool BOTH>
__device__ __noinline__ void full_leg_any(int n, const double* T, int ts, double* Y, const double* F, int fs, int nf,
                                          int ns, int sf, int ss, int st, bool first) {
#define QD_LEG(N) \
  case N: full_leg<N, NT, BOTH>(T, ts, Y, F, fs, nf, ns, sf, ss, st, first); break
  switch (n) {
    QD_LEG(1); QD_LEG(2); QD_LEG(3); QD_LEG(4); QD_LEG(5); QD_LEG(6); QD_LEG(7); QD_LEG(8);
    QD_LEG(9); QD_LEG(10); QD_LEG(11); QD_LEG(12); QD_LEG(13); QD_LEG(14); QD_LEG(15); QD_LEG(16);
  }
#undef QD_LEG
}

__host__ __device__ __forceinline__ int full_fsz(int n) { return n * ((n + 1) & ~1); }

template <int NT, bool BOTH>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1) k_122_full(DevLayout L, const int* __restrict__ tasks,
                                                 const int2* __restrict__ tiles, const int4* __restrict__ gpd,
                                                 const int2* __restrict__ gpp, const double2* __restrict__ F, int nfent,
                                                 const double* __restrict__ A, double hA, unsigned zA,
                                                 const double* __restrict__ B, double hB, unsigned zB,
                                                 double* __restrict__ C) {
  extern __shared__ __align__(16) double smf[];  // T (one or two) | Y | F1 F2 F3 F4 (one or two sets) | pairs
  __shared__ i64 sboff[6];
  const int2 tl = __ldg(&tiles[tasks[blockIdx.x]]);
  const GpDesc da = load_gp(gpd, tl.x), db = load_gp(gpd, tl.y);
  const int tid = threadIdx.x, q = da.q;
  const int n1 = da.n1, n2 = da.n2, n3 = db.n1, n4 = db.n2;
  const int nr = n1 * n2, nc = n3 * n4, ld = nc | 1, tsz = (nr * ld + 1) & ~1;
  const int pa0 = da.cnt(0), pa1 = pa0 + da.cnt(1), pa = pa1 + da.cnt(2);
  const int pb0 = db.cnt(0), pb1 = pb0 + db.cnt(1), pb = pb1 + db.cnt(2);
  const int4 bd = __ldg(&L.blk[q]);
  double* T = smf;
  double* Y = T + (BOTH ? 2 : 1) * tsz;
  double* F1 = Y + tsz;
  double* F2 = F1 + full_fsz(n1);
  double* F3 = F2 + full_fsz(n2);
  double* F4 = F3 + full_fsz(n3);
  const int fs = full_fsz(n1) + full_fsz(n2) + full_fsz(n3) + full_fsz(n4);  // one set
  int2* pr = reinterpret_cast<int2*>(F1 + (BOTH ? 2 : 1) * fs);
  int2* pc = pr + pa;
  for (int i = tid; i < pa; i += NT) pr[i] = __ldg(&gpp[da.pstart + i]);
  for (int i = tid; i < pb; i += NT) pc[i] = __ldg(&gpp[db.pstart + i]);
  if (tid < 6) sboff[tid] = __ldg(L.boff + 6 * q + tid);
  const unsigned one = (1u << P_FHH) | (1u << P_FPP) | (1u << P_FPH);
  // an operand whose factor is zero counts as zero itself
  const bool on[2] = {(zA & one) != one, (zB & one) != one};  // of the B term (factor FA) and the A term
  const int2 e0 = divmod_small(tid, pa), de = divmod_small(NT, pa);
  bool first = true;
#pragma unroll 1
  for (int pass = 0; pass < (BOTH ? 1 : 2); ++pass) {  // FA x TB, then -FB x TA
    if (!BOTH && !on[pass]) continue;
    if (!first) __syncthreads();  // T and the F matrices are free again
    for (int g = 0; g < 4; ++g) {
      const int n = g == 0 ? n1 : (g == 1 ? n2 : (g == 2 ? n3 : n4)), np = (n + 1) & ~1;
      const double2* f = F + (g < 2 ? 0 : nfent) + (g == 0 ? da.fg : (g == 1 ? da.fh : (g == 2 ? db.fg : db.fh)));
      double* d = g == 0 ? F1 : (g == 1 ? F2 : (g == 2 ? F3 : F4));
      const double sg = g < 2 ? 1.0 : -1.0;
      for (int i = tid; i < n * n; i += NT) {
        const double2 v = __ldg(&f[i]);
        const int k = i / n, t = i - k * n;
        if (BOTH) {
          d[k * np + t] = sg * v.x;
          d[fs + k * np + t] = -sg * v.y;
        } else {
          d[k * np + t] = pass ? -sg * v.y : sg * v.x;
        }
      }
      if (np > n)
        for (int k = tid; k < n; k += NT) {
          d[k * np + n] = 0.0;
          if (BOTH) d[fs + k * np + n] = 0.0;
        }
    }
    if (da.same || db.same) {  // the cells (t,t) hold no pair
      for (int i = 2 * tid; i < (BOTH ? 2 : 1) * tsz; i += 2 * NT)
        *reinterpret_cast<double2*>(T + i) = make_double2(0.0, 0.0);
      __syncthreads();
    } else if (first) {
      __syncthreads();  // the pair lists
    }
    // gather: the stored element (P1,P2) of part (c1,c2) when c1 >= c2, else
    // herm times (P2,P1) of part (c2,c1), on its cell with the orientation
    // signs and on the mirror cells (g = h) with the opposite ones
    {
      int p = e0.y, u = e0.x;
#pragma unroll 4
      for (int e = tid; e < pa * pb; e += NT) {
        const int c1 = (p >= pa0) + (p >= pa1), c2 = (u >= pb0) + (u >= pb1);
        const bool lower = c1 >= c2;
        const int part = lower ? slot_of(c1, c2) : slot_of(c2, c1);
        const int2 P = pr[p], Q = pc[u];
        p += de.y;
        u += de.x;
        if (p >= pa) {
          p -= pa;
          ++u;
        }
        const int ldv = cnt_of(lower ? c1 : c2, bd);
        const i64 addr = sboff[part] + (lower ? P.x + (i64)Q.x * ldv : Q.x + (i64)P.x * ldv);
        const int r = P.y & 0xFF, rm = ((P.y >> 8) & 0xFF) - 1;
        const int c = Q.y & 0xFF, cm = ((Q.y >> 8) & 0xFF) - 1;
        const bool neg = (P.y ^ Q.y) & (1 << 16);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          if (!BOTH && x != pass) continue;
          const unsigned zm = x ? zA : zB;
          double v = !on[x] || ((zm >> (P_HHHH + part)) & 1u) ? 0.0 : __ldg((x ? A : B) + addr);
          if (!lower) v *= x ? hA : hB;
          if (neg) v = -v;
          double* t = T + (BOTH ? x * tsz : 0);
          t[r * ld + c] = v;
          if (rm >= 0) t[rm * ld + c] = -v;
          if (cm >= 0) {
            t[r * ld + cm] = -v;
            if (rm >= 0) t[rm * ld + cm] = v;
          }
        }
      }
    }
    __syncthreads();
    full_leg_any<NT, BOTH>(n1, T, tsz, Y, F1, fs, nc, n2, 1, ld, n2 * ld, first);  // items (s; k2), t = k1
    __syncthreads();
    full_leg_any<NT, BOTH>(n2, T, tsz, Y, F2, fs, nc, n1, 1, n2 * ld, ld, false);  // items (s; k1), t = k2
    __syncthreads();
    full_leg_any<NT, BOTH>(n3, T, tsz, Y, F3, fs, nr, n4, ld, 1, n4, false);       // items (r; l2), t = l1
    __syncthreads();
    full_leg_any<NT, BOTH>(n4, T, tsz, Y, F4, fs, nr, n3, ld, n4, 1, false);       // items (r; l1), t = l2
    first = false;
  }
  __syncthreads();
  // stored output cells: c1 >= c2, rows of S_a fastest
  int p = e0.y, u = e0.x;
#pragma unroll 4
  for (int e = tid; e < pa * pb; e += NT) {
    const int c1 = (p >= pa0) + (p >= pa1), c2 = (u >= pb0) + (u >= pb1);
    const int2 P = pr[p], Q = pc[u];
    p += de.y;
    u += de.x;
    if (p >= pa) {
      p -= pa;
      ++u;
    }
    if (c1 < c2) continue;
    double y = first ? 0.0 : Y[(P.y & 0xFF) * ld + (Q.y & 0xFF)];
    if ((P.y ^ Q.y) & (1 << 16)) y = -y;
    C[sboff[slot_of(c1, c2)] + P.x + (i64)Q.x * cnt_of(c1, bd)] = y;
  }
}

// ---- commutator_122 for a generator-like A --------------------------------
// When A's one-body part holds only fph (no hh or pp entries) and its
// two-body part only Vpphh -- the Magnus generator Omega, the White
// generator eta -- the leg sums above collapse, on the two largest output
// parts of a block, to a few columns (or rows) of B each: every term dropped
// is an exact zero (FA couples holes to particles only; A's other parts are
// zero).  With fA(p, h) = A's fph, fB(p, h) = B's fph, pairs indexed within
// the block, s the ordering sign of a pair (v_elem's), hA, hB the herm
// factors and only holes t in G(x) or particles as stated:
//   C_pppp = hB W^T - hA W,
//     W(:, (a,b)) = sum_{t in G(a)} fA(a,t) B_ppph(:, (t,b)) - sum_{t in G(b)} fA(b,t) B_ppph(:, (t,a));
//   C_ppph(:, (h,p)) = - sum_{particles t in G(h)} s fA(t,h) B_pppp(:, (t,p))
//                      - sum_{t in G(p)} s [hA fA(p,t) B_pphh(:, (h,t)) - hB fB(p,t) A_pphh(:, (h,t))]
//   C_ppph((a,b), :) += sum_{t in G(a)} fA(a,t) B_phph((t,b), :) - sum_{t in G(b)} fA(b,t) B_phph((t,a), :).
// (Both checked against the oracle's commutator_122 in numpy before this
// kernel was written.)  B_ppph and B_phph are small (L2 resident); the
// kernels stream C_pppp and C_ppph out once.  Term tables (per layout):
//   pp pair: {ph index of (t, b) or (t, a), t | (a or b - n) << 8 | neg << 20}
//   ph pair: {column, hole | (particle - n) << 8 | neg << 20, kind}: kind 0 a
//            B_pppp column with coefficient -s fA(t, h); kind 1 an hh column
//            (h, t) of B_pphh and A_pphh.
constexpr int SP_T = 256, SP_B = 64;

__device__ __forceinline__ double sp_coef(const DevLayout& L, const double* __restrict__ f, int code) {
  const double v = __ldg(&f[L.o_fph + ((code >> 8) & 0xFFF) + (i64)(code & 0xFF) * L.mp]);
  return (code >> 20) & 1 ? -v : v;
}

// A term staged in shared memory: its coefficient, and the source element
// off + fixed * (m & MULT_MASK) of operand B (bit 30 of m set) or A.
struct StagedTerm {
  double c;
  int off, m;
};
constexpr int MULT_MASK = 0x3FFFFFFF;

// C_pppp of a block for a generator-like A, and with it the pppp ladder of
// commutator_222 (matrix_mult222, src/commutators.f90:1010-1032), which for
// such an A is the rank-n_h update D = -hB A_pphh B_pphh^T, C += D + s D^T,
// s = -hA hB.  One task = the 64 x 64 tile pair (I, J), (J, I):
//   C(I,J)[r,c] = hB W(J,I)[c,r] - hA W(I,J)[r,c]
//                 - hB sum_k (A_I[r,k] B_J[c,k] + s A_J[c,k] B_I[r,k]),
// and C(J,I) = s C(I,J)^T (both terms change by that sign).
//   phase 0  the W terms of the columns of J and I (coefficients resolved)
//            and the n_h-column panels of A_pphh, B_pphh go to shared memory
//   phase 1  the ladder's two products on the FP64 tensor pipe; the tile then
//            takes the panels' place in shared memory
//   phase 2  hB W(J,I)^T is added, lanes along W's rows
//   phase 3  W(I,J) in registers, lanes along its rows; C(I,J) is written and
//            s C(I,J) stored in the tile
//   phase 4  C(J,I) is written from there
// Bound: writing C once (437 MB at N=20, R=20).  The tile is 64 x 64 because
// a CTA's chain of dependent table reads (~4 us) is the same for any size:
// the 32 x 32 tiles used before paid it four times as often, and the ladder
// as a separate read-modify-write of C_pppp moved its half that has hh pairs
// twice more (a commutator [Omega, X] at N=20, R=20: 875 us with these, 750
// with this kernel).
constexpr int GP_B = 64, GP_LD = GP_B + 1, GP_T = 256, GP_KMAX = 16;

// A warp takes one column at a time, its lanes the rows l and l + 32: a staged
// term is read from shared memory once for 64 rows.  Four of the warp's
// columns (c = wid + 8 (j + jj)): sums over their terms of coef * X[row + off].
// Neighbouring columns are pairs (a, b), (a, b') with b, b' of one group, so
// they mostly have the same number of terms (0 to 4).
__device__ __forceinline__ void gp_cols(const StagedTerm* T, const int* st, const double* __restrict__ X, bool ok0,
                                        bool ok1, int wid, int j, double w[4][2]) {
  int s[4], n[4], most = 0;
#pragma unroll
  for (int jj = 0; jj < 4; ++jj) {
    const int c = wid + 8 * (j + jj);
    s[jj] = st[c];
    n[jj] = st[c + 1] - s[jj];
    most = max(most, n[jj]);
    w[jj][0] = w[jj][1] = 0.0;
  }
  for (int i = 0; i < most; ++i) {
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
      if (i < n[jj]) {
        const StagedTerm t = T[s[jj] + i];
        const double* p = X + t.off;
        if (ok0) w[jj][0] += t.c * __ldg(p);
        if (ok1) w[jj][1] += t.c * __ldg(p + 32);
      }
  }
}

__constant__ double c_gp_cof[11] = QD_BCH_COF;

// Panels are [k][64] with the column swizzled by k, so that a DMMA fragment
// (4 k x 8 columns) touches every bank once.
__device__ __forceinline__ int gp_pos(int k, int m) { return k * GP_B + (m ^ ((k & 3) << 2)); }

__device__ __forceinline__ void gp_dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

template <bool UPD>
__global__ void __launch_bounds__(GP_T, UPD ? 3 : 4) k_gen_pppp(DevLayout L, const int4* __restrict__ tasks,
                                                     const int* __restrict__ ppbase, const int* __restrict__ ppstart,
                                                     const int2* __restrict__ ppterm, const double* __restrict__ A,
                                                     double hA, const double* __restrict__ B, double hB, unsigned zB,
                                                     int ladder, double* __restrict__ C, HsUpdate U) {
  extern __shared__ __align__(16) double gsm[];  // tile [64][65], before it the panels A_I, s B_I, A_J, B_J | terms
  __shared__ int sst[2][GP_B + 1];               // each column's first staged term, of J and of I
  const int4 t = tasks[blockIdx.x];
  const int q = t.x, I0 = t.y * GP_B, J0 = t.z * GP_B;
  const int4 bd = __ldg(&L.blk[q]);
  const int np = bd.z, nI = min(GP_B, np - I0), nJ = min(GP_B, np - J0);
  const i64* boff = L.boff + 6 * q;
  const bool diag = t.y == t.z;
  const int K = ladder && bd.x <= GP_KMAX ? bd.x : 0;  // as gen_ladder_fused
  double* Tt = gsm;
  StagedTerm* T = reinterpret_cast<StagedTerm*>(gsm + GP_B * GP_LD);
  const int tid = threadIdx.x, r = tid & (GP_B - 1), cq = tid >> 6;
  const bool live = !((zB >> P_PPPH) & 1u);
  const int pb = __ldg(&ppbase[q]);
  const int j0 = __ldg(&ppstart[pb + J0]), jn = live ? __ldg(&ppstart[pb + J0 + nJ]) - j0 : 0;
  const int i0 = __ldg(&ppstart[pb + I0]), in = live ? __ldg(&ppstart[pb + I0 + nI]) - i0 : 0;
  double* out = C + __ldg(boff + 1);
  // UPD: HS += cof C and the sums of squares of both
  const double* hs = UPD ? U.src + __ldg(boff + 1) : nullptr;
  const i64 hsd = UPD ? U.HS - U.src : 0;  // from an entry read to the entry written
  double an = 0.0, bn = 0.0;
  auto sums = [&]() {  // the CTA's two sums, in a fixed order
    if (!UPD) return;
    __shared__ double red[GP_T / 32];
    const double a = block_sum<GP_T>(an, red), b = block_sum<GP_T>(bn, red);
    if (threadIdx.x == 0) {
      U.partial[2 * blockIdx.x] = a;
      U.partial[2 * blockIdx.x + 1] = b;
    }
  };
  if (jn == 0 && in == 0 && K == 0) {  // nothing reaches the tile pair: C = 0, HS = src
    for (int side = 0; side < (diag ? 1 : 2); ++side) {
      const int R0 = side ? J0 : I0, C0 = side ? I0 : J0, nr = side ? nJ : nI, nc = side ? nI : nJ;
      if (r < nr)
#pragma unroll 4
        for (int c = cq; c < nc; c += 4) {
          const i64 e = (R0 + r) + (i64)(C0 + c) * np;
          out[e] = 0.0;
          if (UPD) {
            const double x = hs[e];
            an += x * x;
            if (hsd) U.HS[__ldg(boff + 1) + e] = x;
          }
        }
    }
    sums();
    return;
  }
  double cof = 0.0;
  if (UPD) {
    cof = U.kidx ? c_gp_cof[*U.kidx] : U.cof;
    // HS of both tiles on its way to L2 while the tables are read: a column's
    // 64 rows are 512 bytes, five sectors' starts 128 bytes apart
    for (int i = tid; i < 5 * (nJ + (diag ? 0 : nI)); i += GP_T) {
      const int c = i / 5, s = i - 5 * c, side = c >= nJ;
      const int R0 = side ? J0 : I0, nr = side ? nJ : nI, col = side ? I0 + c - nJ : J0 + c;
      const double* p = hs + R0 + min(16 * s, nr - 1) + (i64)col * np;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
  }
  const double sg = -hA * hB;
  const int ib = diag ? 0 : jn;  // first staged term of I's columns
  for (int i = tid; i <= GP_B; i += GP_T) {
    sst[0][i] = live ? __ldg(&ppstart[pb + J0 + min(i, nJ)]) - j0 : 0;
    sst[1][i] = ib + (live ? __ldg(&ppstart[pb + I0 + min(i, nI)]) - i0 : 0);
  }
  const int K4 = (K + 3) & ~3;
  double *PAI = gsm, *PBI = PAI + GP_KMAX * GP_B, *PAJ = PBI + GP_KMAX * GP_B, *PBJ = PAJ + GP_KMAX * GP_B;
  if (K > 0) {
    const double* pA = A + __ldg(boff + 2);
    const double* pB = B + __ldg(boff + 2);
    for (int k = cq; k < K4; k += 4) {
      const i64 o = (i64)k * np;
      const bool oi = k < K && r < nI, oj = k < K && r < nJ;
      const double ai = oi ? __ldg(pA + I0 + r + o) : 0.0, bi = oi ? __ldg(pB + I0 + r + o) : 0.0;
      const double aj = oj ? __ldg(pA + J0 + r + o) : 0.0, bj = oj ? __ldg(pB + J0 + r + o) : 0.0;
      const int p = gp_pos(k, r);
      PAI[p] = ai;
      PBI[p] = sg * bi;
      PAJ[p] = aj;
      PBJ[p] = bj;
    }
  }
  for (int i = tid; i < jn; i += GP_T) {
    const int2 tm = __ldg(&ppterm[j0 + i]);
    T[i] = StagedTerm{sp_coef(L, A, tm.y), tm.x * np, 0};
  }
  if (!diag)
    for (int i = tid; i < in; i += GP_T) {
      const int2 tm = __ldg(&ppterm[i0 + i]);
      T[ib + i] = StagedTerm{sp_coef(L, A, tm.y), tm.x * np, 0};
    }
  __syncthreads();
  if (K > 0) {
    const int lane = tid & 31, wm = (tid >> 5) & 1, wn = tid >> 6;  // warp tile 32 x 16
    double acc[4][2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    for (int kk = 0; kk < K4; kk += 4) {
      const int kr = kk + (lane & 3);
#pragma unroll
      for (int side = 0; side < 2; ++side) {  // A_I B_J^T, then (s B_I) A_J^T
        const double *pa = side ? PBI : PAI, *pb2 = side ? PAJ : PBJ;
        double af[4], bf[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) af[i] = pa[gp_pos(kr, wm * 32 + i * 8 + (lane >> 2))];
#pragma unroll
        for (int j = 0; j < 2; ++j) bf[j] = pb2[gp_pos(kr, wn * 16 + j * 8 + (lane >> 2))];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) gp_dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        double* p = Tt + (wm * 32 + i * 8 + (lane >> 2)) * GP_LD + wn * 16 + j * 8 + 2 * (lane & 3);
        p[0] = -hB * acc[i][j][0];
        p[1] = -hB * acc[i][j][1];
      }
    if (in > 0) __syncthreads();
  }
  const double* X = B + __ldg(boff + 4);  // B_ppph, np x nph
  const int l = tid & 31, wid = tid >> 5;
  if (in > 0) {
#pragma unroll 1
    for (int j = 0; j < GP_B / 8; j += 4) {
      double w[4][2];
      gp_cols(T, sst[1], X + J0 + l, l < nJ, l + 32 < nJ, wid, j, w);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        double* p = Tt + (wid + 8 * (j + jj)) * GP_LD + l;
        p[0] = K > 0 ? p[0] + hB * w[jj][0] : hB * w[jj][0];
        p[32] = K > 0 ? p[32] + hB * w[jj][1] : hB * w[jj][1];
      }
    }
  }
  __syncthreads();
  const bool have = in > 0 || K > 0;
  const i64 step = (i64)8 * np;
  {
    double* o = out + (I0 + l) + (i64)(J0 + wid) * np;
    const double* ho = UPD ? hs + (I0 + l) + (i64)(J0 + wid) * np : nullptr;
    const bool ok0 = l < nI, ok1 = l + 32 < nI;
#pragma unroll 1
    for (int j = 0; j < GP_B / 8; j += 4) {
      double w[4][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
      double g[4][2];
      double* hw = UPD ? const_cast<double*>(ho) + hsd : nullptr;
      if (UPD)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {  // in flight while W is summed
          const bool in = wid + 8 * (j + jj) < nJ;
          g[jj][0] = in && ok0 ? ho[jj * step] : 0.0;
          g[jj][1] = in && ok1 ? ho[jj * step + 32] : 0.0;
        }
      if (jn > 0) gp_cols(T, sst[0], X + I0 + l, ok0, ok1, wid, j, w);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int c = wid + 8 * (j + jj);
        double *p0 = Tt + l * GP_LD + c, *p1 = p0 + 32 * GP_LD;
        const double v0 = (have ? *p0 : 0.0) - hA * w[jj][0], v1 = (have ? *p1 : 0.0) - hA * w[jj][1];
        if (c < nJ) {
          if (ok0) {
            o[0] = v0;
            if (UPD) {
              hw[jj * step] = __dadd_rn(g[jj][0], __dmul_rn(cof, v0));
              an += g[jj][0] * g[jj][0];
              bn += v0 * v0;
            }
          }
          if (ok1) {
            o[32] = v1;
            if (UPD) {
              hw[jj * step + 32] = __dadd_rn(g[jj][1], __dmul_rn(cof, v1));
              an += g[jj][1] * g[jj][1];
              bn += v1 * v1;
            }
          }
        }
        o += step;
        *p0 = sg * v0;
        *p1 = sg * v1;
      }
      if (UPD) ho += 4 * step;
    }
  }
  if (!diag) {
    __syncthreads();
    const bool ok0 = l < nJ, ok1 = l + 32 < nJ;
    double* o = out + (J0 + l) + (i64)(I0 + wid) * np;
    const double* ho = UPD ? hs + (J0 + l) + (i64)(I0 + wid) * np : nullptr;
#pragma unroll 1
    for (int j = 0; j < GP_B / 8; j += 4) {
      double g[4][2];
      double* hw = UPD ? const_cast<double*>(ho) + hsd : nullptr;
      if (UPD)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const bool in = wid + 8 * (j + jj) < nI;
          g[jj][0] = in && ok0 ? ho[jj * step] : 0.0;
          g[jj][1] = in && ok1 ? ho[jj * step + 32] : 0.0;
        }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int c = wid + 8 * (j + jj);
        if (c < nI) {
          const double v0 = Tt[c * GP_LD + l], v1 = Tt[c * GP_LD + l + 32];
          if (ok0) {
            o[0] = v0;
            if (UPD) {
              hw[jj * step] = __dadd_rn(g[jj][0], __dmul_rn(cof, v0));
              an += g[jj][0] * g[jj][0];
              bn += v0 * v0;
            }
          }
          if (ok1) {
            o[32] = v1;
            if (UPD) {
              hw[jj * step + 32] = __dadd_rn(g[jj][1], __dmul_rn(cof, v1));
              an += g[jj][1] * g[jj][1];
              bn += v1 * v1;
            }
          }
        }
        o += step;
      }
      if (UPD) ho += 4 * step;
    }
  }
  sums();
}

// Whether k_gen_pppp takes block q's pppp ladder with it: up to 16 hh pairs
// fit its panels (N <= 20 has at most 16); blocks with more keep the grouped
// GEMM, whose read-modify-write of C is then a smaller part of the work.
bool gen_ladder_fused(const qd_layout* L, int q) { return L->blk[q].x > 0 && L->blk[q].x <= GP_KMAX; }

size_t gp_smem(int terms) { return sizeof(double) * GP_B * GP_LD + sizeof(StagedTerm) * (size_t)terms; }
size_t gen_smem(int terms) { return sizeof(StagedTerm) * (size_t)terms; }
static_assert(4 * GP_KMAX * GP_B <= GP_B * GP_LD, "the panels share the tile's shared memory");

// The other five parts of a block for a generator-like A, one 64 x 64 tile
// of one part per task {q, part, ti, tj}: every output element (R, c) is
//   sum over the terms of its row pair of coef * M[idx + c ld] (M[c + idx ld] transposed)
// + sum over the terms of its column pair of coef * M[R + idx ld] (M[idx + R ld] transposed),
// M a stored part of A or B in block q with ld rows.  Term {idx, coefficient
// offset, flags, source}: flags bit 0 negate, 1 times hA, 2 times hB, 3 the
// coefficient is B's entry (else A's); source (operand << 4) | (T << 3) | slot.
// The closed forms (derived from the leg sums, each checked against the
// oracle's commutator_122 in numpy first), with s an ordering sign:
//   ppph rows (a,b): +-fA(a|b,t) B_phph((t,b|a), .);  columns (h,p):
//        -s fA(t,h) B_pppp(., (t,p)) [particles t in G(h)],
//        -s hA fA(p,t) B_pphh(., (h,t)) + s hB fB(p,t) A_pphh(., (h,t)) [holes t in G(p)]
//   pphh rows (a,b): +-fA(a|b,t) B_phhh((t,b|a), .) - s hB fppB(t,a|b) A_pphh((t,b)|(a,t), .);
//        columns (k,l): +-fA(t,k|l) B_ppph(., (l|k,t)) + s hB fhhB(k|l,t) A_pphh(., (t,l)|(k,t))
//   phhh rows (h,p): s hA fA(t,h) B_pphh((t,p), .) - s hB fB(t,h) A_pphh((t,p), .) + s fA(p,t) B_hhhh((h,t), .);
//        columns (k,l): +-fA(t,k|l) B_phph(., (l|k,t))
//   phph rows (h,p): s hA fA(t,h) B_ppph((t,p), .) + s hB fA(p,t) B_phhh(., (h,t))^T;
//        columns (k,l): -s hB fA(t,k) B_ppph((t,l), .)^T - s hA fA(l,t) B_phhh(., (k,t))
//   hhhh rows (a,b): -+hA fA(t,a|b) B_phhh((b|a,t), .);  columns (k,l): +-hB fA(t,k|l) B_phhh((l|k,t), .)^T
struct GenTables {
  const int* gbase;   // 3 * nblock: first hh, ph, pp pair of each block
  const int* rstart;  // per part: per row pair its first term (one more entry at the end)
  const int* cstart;
  const int4* rterm;
  const int4* cterm;
  int rso[6], cso[6];  // offset of each part's start array (slot order)
};

// Resolve a term for one tile: its coefficient and its source element as
// off + fixed * m (row term: fixed = output column; column term: output row).
__device__ __forceinline__ StagedTerm stage_term(const DevLayout& L, const int4& tm, int q, int4 bd, bool row_term,
                                                 const double* __restrict__ A, double hA,
                                                 const double* __restrict__ B, double hB) {
  const int opd = tm.w >> 4, slot = tm.w & 7;
  const bool tr = (tm.w >> 3) & 1;
  const int ld = part_rows(P_HHHH + slot, bd);
  const int bo = (int)__ldg(L.boff + 6 * q + slot);
  StagedTerm st;
  if (row_term != tr) {
    st.off = bo + tm.x;
    st.m = ld;
  } else {
    st.off = bo + tm.x * ld;
    st.m = 1;
  }
  st.m |= opd << 30;
  double c = __ldg(&((tm.z >> 3) & 1 ? B : A)[tm.y]);
  if (tm.z & 2) c *= hA;
  if (tm.z & 4) c *= hB;
  if (tm.z & 1) c = -c;
  st.c = c;
  return st;
}

// Sums over a lane's row terms for four columns: coef * M[c * m], two terms
// at a time (eight loads in flight).
__device__ __forceinline__ void gen_rows(const StagedTerm* T, int e, int e1, const double* __restrict__ A,
                                         const double* __restrict__ B, const i64 cj[4], double y[4]) {
  for (; e + 1 < e1; e += 2) {
    const StagedTerm ta = T[e], tb = T[e + 1];
    const i64 ma = ta.m & MULT_MASK, mb = tb.m & MULT_MASK;
    const double *pa = ((ta.m >> 30) ? B : A) + ta.off, *pb = ((tb.m >> 30) ? B : A) + tb.off;
    double va[4], vb[4];
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      va[jj] = __ldg(pa + cj[jj] * ma);
      vb[jj] = __ldg(pb + cj[jj] * mb);
    }
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      y[jj] += ta.c * va[jj];
      y[jj] += tb.c * vb[jj];
    }
  }
  if (e < e1) {
    const StagedTerm tm = T[e];
    const i64 m = tm.m & MULT_MASK;
    const double* p = ((tm.m >> 30) ? B : A) + tm.off;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) y[jj] += tm.c * __ldg(p + cj[jj] * m);
  }
}

// Columns k, k + 8, k + 16, k + 24 of a tile of n columns, past its end the last one.
__device__ __forceinline__ void gen_columns(int J0, int k, int n, i64 cj[4]) {
#pragma unroll
  for (int jj = 0; jj < 4; ++jj) cj[jj] = J0 + min(k + 8 * jj, n - 1);
}

// C_phph of the tile pair (I, J), (J, I), I <= J: the column terms of phph are
// s = -hA hB times the transposed row terms, so C(I,J) = V(I,J) + s V(J,I)^T
// with V the row terms alone (half the loads, and all along rows: a column
// term reads B_ppph across its columns), and C(J,I) = s C(I,J)^T.
__global__ void __launch_bounds__(SP_T) k_gen_phph(DevLayout L, const int4* __restrict__ tasks, GenTables G,
                                                  const double* __restrict__ A, double hA,
                                                  const double* __restrict__ B, double hB, double* __restrict__ C) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int si[SP_B + 1], sj[SP_B + 1];
  const int4 t = tasks[blockIdx.x];
  const int4 bd = __ldg(&L.blk[t.x]);
  const int q = t.x, n = bd.y, I0 = t.z * SP_B, J0 = t.w * SP_B, nI = min(SP_B, n - I0), nJ = min(SP_B, n - J0);
  const bool diag = t.z == t.w;
  constexpr int LD = SP_B + 1;
  double* Tt = sm;  // V(J,I)^T, then s C(I,J)
  StagedTerm* T = reinterpret_cast<StagedTerm*>(sm + SP_B * LD);
  const int* rs = G.rstart + G.rso[3] + __ldg(&G.gbase[L.nblock + q]);
  const int i0 = __ldg(&rs[I0]), ni = __ldg(&rs[I0 + nI]) - i0;
  const int j0 = __ldg(&rs[J0]), nj = diag ? 0 : __ldg(&rs[J0 + nJ]) - j0;
  const int tid = threadIdx.x, l = tid & 31, wid = tid >> 5;
  for (int i = tid; i <= SP_B; i += SP_T) {
    si[i] = __ldg(&rs[I0 + min(i, nI)]) - i0;
    sj[i] = (diag ? 0 : ni) + __ldg(&rs[J0 + min(i, nJ)]) - j0;
  }
  for (int i = tid; i < ni; i += SP_T) T[i] = stage_term(L, __ldg(&G.rterm[i0 + i]), q, bd, true, A, hA, B, hB);
  for (int i = tid; i < nj; i += SP_T) T[ni + i] = stage_term(L, __ldg(&G.rterm[j0 + i]), q, bd, true, A, hA, B, hB);
  __syncthreads();
  for (int k = wid; k < nI; k += 32) {  // V(J,I): lanes along the rows of J
    i64 cj[4];
    gen_columns(I0, k, nI, cj);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = l + 32 * h;
      if (r >= nJ) continue;
      double y[4] = {0.0, 0.0, 0.0, 0.0};
      gen_rows(T, sj[r], sj[r + 1], A, B, cj, y);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        if (k + 8 * jj < nI) Tt[(k + 8 * jj) * LD + r] = y[jj];
    }
  }
  __syncthreads();
  const double sg = -hA * hB;
  double* out = C + __ldg(L.boff + 6 * q + 3);
  for (int k = wid; k < nJ; k += 32) {
    i64 cj[4];
    gen_columns(J0, k, nJ, cj);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = l + 32 * h;
      if (r >= nI) continue;
      double y[4] = {0.0, 0.0, 0.0, 0.0};
      gen_rows(T, si[r], si[r + 1], A, B, cj, y);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int c = k + 8 * jj;
        if (c >= nJ) continue;
        const double v = y[jj] + sg * Tt[r * LD + c];
        out[(I0 + r) + (i64)(J0 + c) * n] = v;
        if (!diag) Tt[r * LD + c] = sg * v;  // this thread's own element
      }
    }
  }
  if (diag) return;
  __syncthreads();
  for (int c = wid; c < nI; c += 8)
    for (int r = l; r < nJ; r += 32) out[(J0 + r) + (i64)(I0 + c) * n] = Tt[c * LD + r];
}

// The tile's column terms, then its row terms, are staged once per CTA in
// shared memory (dynamic size: the most terms of any tile of the launch).
__global__ void __launch_bounds__(SP_T) k_122_gen(DevLayout L, const int4* __restrict__ tasks, GenTables G,
                                                 const double* __restrict__ A, double hA,
                                                 const double* __restrict__ B, double hB, int ladder,
                                                 double* __restrict__ C) {
  extern __shared__ __align__(16) double sgt[];
  StagedTerm* T = reinterpret_cast<StagedTerm*>(sgt);
  __shared__ int scs[SP_B + 1], srs[SP_B + 1];
  const int4 t = tasks[blockIdx.x];
  const int q = t.x, slot = t.y, I0 = t.z * SP_B, J0 = t.w * SP_B;
  const int4 bd = __ldg(&L.blk[q]);
  int cr, cc;
  part_classes(P_HHHH + slot, cr, cc);
  const int nrow = part_rows(P_HHHH + slot, bd), ncol = cc == 0 ? bd.x : (cc == 1 ? bd.y : bd.z);
  const int nrt = min(SP_B, nrow - I0), nct = min(SP_B, ncol - J0);
  const int* rs = G.rstart + G.rso[slot] + __ldg(&G.gbase[cr * L.nblock + q]) + I0;
  const int* cs = G.cstart + G.cso[slot] + __ldg(&G.gbase[cc * L.nblock + q]) + J0;
  const int c0 = __ldg(&cs[0]), nce = __ldg(&cs[nct]) - c0;
  const int r0 = __ldg(&rs[0]), nre = __ldg(&rs[nrt]) - r0;
  const int tid = threadIdx.x;
  for (int i = tid; i <= SP_B; i += SP_T) {
    scs[i] = __ldg(&cs[min(i, nct)]) - c0;
    srs[i] = nce + __ldg(&rs[min(i, nrt)]) - r0;
  }
  for (int i = tid; i < nce; i += SP_T) T[i] = stage_term(L, __ldg(&G.cterm[c0 + i]), q, bd, false, A, hA, B, hB);
  for (int i = tid; i < nre; i += SP_T) T[nce + i] = stage_term(L, __ldg(&G.rterm[r0 + i]), q, bd, true, A, hA, B, hB);
  __syncthreads();
  // a warp takes four columns at a time, its lanes the rows l and l + 32: a
  // term is read from shared memory once for the loads it feeds, and eight
  // (column terms) or four (row terms) loads are in flight together
  const int l = tid & 31, wid = tid >> 5;
  const bool ok0 = l < nrt, ok1 = l + 32 < nrt;
  const int row = I0 + l;
  double* out = C + __ldg(L.boff + 6 * q + slot) + row + (i64)J0 * nrow;
  // the ppph ladder that a generator-like A leaves: -hB A_pphh B_phhh^T
  const int K = slot == 4 && ladder && bd.x <= GP_KMAX ? bd.x : 0;
  const double* LA = A + __ldg(L.boff + 6 * q + 2) + row;
  const double* LB = B + __ldg(L.boff + 6 * q + 5) + J0;
  for (int k = wid; k < nct; k += 4 * (SP_T / 32)) {
    double y[4][2];
    int s[4], n[4], most = 0;
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const int c = min(k + 8 * jj, nct);
      s[jj] = scs[c];
      n[jj] = scs[min(c + 1, nct)] - s[jj];
      most = max(most, n[jj]);
      y[jj][0] = y[jj][1] = 0.0;
    }
    for (int i = 0; i < most; ++i) {
#pragma unroll
      for (int jj = 0; jj < 4; ++jj)
        if (i < n[jj]) {
          const StagedTerm tm = T[s[jj] + i];
          const int m = tm.m & MULT_MASK;
          const double* p = ((tm.m >> 30) ? B : A) + tm.off + (i64)row * m;
          if (ok0) y[jj][0] += tm.c * __ldg(p);
          if (ok1) y[jj][1] += tm.c * __ldg(p + 32 * m);
        }
    }
    i64 cj[4];
    gen_columns(J0, k, nct, cj);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!(h ? ok1 : ok0)) continue;
      double z[4] = {0.0, 0.0, 0.0, 0.0};
      gen_rows(T, srs[l + 32 * h], srs[l + 32 * h + 1], A, B, cj, z);
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) y[jj][h] += z[jj];
    }
#pragma unroll 2
    for (int h = 0; h < K; ++h) {
      const double a0 = ok0 ? -hB * __ldg(LA + (i64)h * nrow) : 0.0, a1 = ok1 ? -hB * __ldg(LA + (i64)h * nrow + 32) : 0.0;
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const double b = k + 8 * jj < nct ? __ldg(LB + k + 8 * jj + (i64)h * ncol) : 0.0;
        y[jj][0] += a0 * b;
        y[jj][1] += a1 * b;
      }
    }
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
      if (k + 8 * jj < nct) {
        double* o = out + (i64)(k + 8 * jj) * nrow;
        if (ok0) o[0] = y[jj][0];
        if (ok1) o[32] = y[jj][1];
      }
  }
}

// ---- the ladders with a long K that a generator-like A leaves --------------
// (matrix_mult222, src/commutators.f90:996-1130, blocks with n_h <= 16 hh pairs)
//   pphh += -B_pppp A_pphh - A_pphh B_hhhh
//   phhh += -hB B_ppph^T A_pphh
//   hhhh += V + s V^T, V = -hB B_pphh^T A_pphh, s = -hA hB
// All multiply by the n_p x n_h panel A_pphh: n_h <= 16 columns, so a 64 x 64
// tile of the grouped GEMM was three quarters padding.  Bound: reading B_pppp
// of the blocks with hh pairs once (218 MB at N=20, R=20).  Roles (task.y):
//   0  64 rows of pphh on the FP64 tensor pipe: a warp multiplies every eighth
//      group of four columns of B_pppp (a fragment is four runs of eight rows,
//      straight from global memory, sixteen fragments in flight) with the
//      panel's fragment; the eight warps' sums are added in warp order
//   1  16 rows of phhh, 2 all of hhhh: a warp per two rows, lanes along the
//      contracted index (contiguous), one warp sum per output at the end
constexpr int GL_T = 256;

// sums of v[16] over a warp: lanes 2 i and 2 i + 1 return that of v[i]
__device__ __forceinline__ double gl_sum16(double* v, int lane) {
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int half = 8 >> s, d = 16 >> s;
    const bool up = lane & d;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const double send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

template <int NB>  // groups of eight hh pairs
__device__ void gl_pphh(int np, int nh, int I0, const double* __restrict__ Bpp, const double* __restrict__ Ap,
                        const double* __restrict__ Bhh, double* __restrict__ out, double* sm) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, lr = lane >> 2, lk = lane & 3;
  const int nr = min(64, np - I0);
  double acc[8][NB][2];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int n = 0; n < NB; ++n) acc[i][n][0] = acc[i][n][1] = 0.0;
  if (Bpp) {
    int ro[8];  // rows past the block repeat its last one: their sums are not used
#pragma unroll
    for (int i = 0; i < 8; ++i) ro[i] = I0 + min(8 * i + lr, nr - 1);
    const double* pb[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) pb[n] = Ap + (i64)min(8 * n + lr, nh - 1) * np;
    constexpr int U = NB == 1 ? 2 : 1;
    auto step = [&](int k, auto tail) {  // columns k .. k + 3 and, U = 2, k + 32 .. k + 35
      double a[U][8], b[U][NB];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int kk = k + 32 * u + lk;
        const bool in = !decltype(tail)::value || kk < np;
        const double* p = Bpp + (i64)kk * np;
#pragma unroll
        for (int i = 0; i < 8; ++i) a[u][i] = in ? __ldg(p + ro[i]) : 0.0;
#pragma unroll
        for (int n = 0; n < NB; ++n) b[u][n] = in && 8 * n + lr < nh ? __ldg(pb[n] + kk) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int n = 0; n < NB; ++n) gp_dmma(acc[i][n][0], acc[i][n][1], a[u][i], b[u][n]);
    };
    int k = 4 * w;
#pragma unroll 1
    for (; k + 32 * (U - 1) + 4 <= np; k += 32 * U) step(k, std::false_type());
    if (k < np) step(k, std::true_type());
  }
  // the eight warps' sums, added in warp order through shared memory
  for (int turn = 0; turn < GL_T / 32; ++turn) {
    __syncthreads();
    if (w == turn) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int n = 0; n < NB; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            double* p = sm + (8 * n + 2 * lk + e) * 64 + 8 * i + lr;
            *p = turn == 0 ? acc[i][n][e] : *p + acc[i][n][e];
          }
    }
  }
  __syncthreads();
  for (int i = tid; i < 64 * nh; i += GL_T) {
    const int r = i & 63, h = i >> 6;
    if (r >= nr) continue;
    double s = sm[h * 64 + r];
    if (Bhh)
      for (int k = 0; k < nh; ++k) s += __ldg(Ap + I0 + r + (i64)k * np) * __ldg(Bhh + k + h * nh);
    out[(I0 + r) + (i64)h * np] -= s;
  }
}

__global__ void __launch_bounds__(GL_T, 2) k_gen_ladder(DevLayout L, const int4* __restrict__ tasks,
                                                       const double* __restrict__ A, double hA,
                                                       const double* __restrict__ B, double hB, unsigned zB,
                                                       double* __restrict__ C) {
  __shared__ double sm[64 * GP_KMAX];
  const int4 t = tasks[blockIdx.x];
  const int q = t.x;
  const int4 bd = __ldg(&L.blk[q]);
  const int nh = bd.x, nb = bd.y, np = bd.z;
  const i64* o = L.boff + 6 * q;
  const double* Ap = A + __ldg(o + 2);
  if (t.y == 0) {
    const double* Bpp = (zB >> P_PPPP) & 1u ? nullptr : B + __ldg(o + 1);
    const double* Bhh = (zB >> P_HHHH) & 1u ? nullptr : B + __ldg(o + 0);
    double* out = C + __ldg(o + 2);
    if (nh <= 8)
      gl_pphh<1>(np, nh, t.z, Bpp, Ap, Bhh, out, sm);
    else
      gl_pphh<2>(np, nh, t.z, Bpp, Ap, Bhh, out, sm);
    return;
  }
  const bool hh = t.y == 2;
  if ((zB >> (hh ? P_PPHH : P_PPPH)) & 1u) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int rows = hh ? nh : nb, r0 = t.z + 2 * w;  // at most 16 hh pairs: one CTA holds all of hhhh
  const double* x0 = B + __ldg(o + (hh ? 2 : 4)) + (i64)min(r0, rows - 1) * np;
  const double* x1 = r0 + 1 < rows ? x0 + np : x0;
  for (int half = 0; half < 2 && 8 * half < nh; ++half) {
    double v[16];  // rows r0, r0 + 1 times eight columns
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = 0.0;
    const double* a = Ap + (i64)8 * half * np;
#pragma unroll 2
    for (int k = lane; k < np; k += 32) {
      const double b0 = __ldg(x0 + k), b1 = __ldg(x1 + k);
#pragma unroll
      for (int h = 0; h < 8; ++h)
        if (8 * half + h < nh) {
          const double c = __ldg(a + k + (i64)h * np);
          v[h] += b0 * c;
          v[8 + h] += b1 * c;
        }
    }
    const double s = -hB * gl_sum16(v, lane);
    const int r = r0 + (lane >> 4), h = 8 * half + ((lane >> 1) & 7);
    if (!(lane & 1) && r < rows && h < nh) {
      if (hh)
        sm[r * 16 + h] = s;
      else
        C[__ldg(o + 5) + r + (i64)h * nb] += s;
    }
  }
  if (!hh) return;
  __syncthreads();
  const double sg = -hA * hB;
  for (int i = threadIdx.x; i < nh * nh; i += GL_T) {
    const int r = i % nh, h = i / nh;
    C[__ldg(o + 0) + r + (i64)h * nh] += sm[r * 16 + h] + sg * sm[h * 16 + r];
  }
}

// ---- particle-hole channel of commutator_222 over the same tiles ----------
// (src/commutators.f90:716-980, ME_general.f90:923-952.)  With Z = XCC - YCC
// in cross-coupled coordinates and the stored output element oriented as the
// cells (k1,k2) of S(g,h), (l1,l2) of S(g',h') -- states x = G_g[k1],
// y = G_h[k2], u = G_g'[l1], v = G_h'[l2] --
//   C += Z[(u,x),(y,v)] - Z[(u,y),(x,v)] + Z[(v,y),(x,u)] - Z[(v,x),(y,u)].
// The cc rows are group-major (all rows (i in G1, j in G2) form one run), so
// each term reads one dense sub-matrix of one cc block: rows G1 x G2 (one run
// of |G1||G2| doubles per column), columns G3 x G4.  Term t (sign (-1)^t):
//   t  rows (G1,G2)  columns (G3,G4)  element (rows; columns)
//   0  (g', g)       (h, h')          (l1,k1; k2,l2)
//   1  (g', h)       (g, h')          (l1,k2; k1,l2)
//   2  (h', h)       (g, g')          (l2,k2; k1,l1)
//   3  (h', g)       (h, g')          (l2,k1; k2,l1)
// Terms 0 and 2, and 1 and 3, lie in blocks of opposite transfer, whose sum
// prog_pandya stores in the upper one: a tile reads the terms whose block is
// the upper of its pair (two of the four, more where a transfer is zero).
// Modes (per launch bucket, by the tile's size):
//   PD_ALL    the sub-matrices of all its terms staged at once (one wait), one
//             pass over the stored cells adds their elements into C;
//   PD_SINGLE one buffer and an accumulator, the terms one after another;
//   PD_DIRECT no staging: each cell reads its elements from global memory.
// Every cell adds its terms in the order of t in all modes.  Bound: HBM and
// L2 traffic of Z and C.
enum { PD_DIRECT = 0, PD_ALL = 1, PD_SINGLE = 2 };
constexpr size_t PD_SMEM = SMEM_MAX_122 - 1024;  // beside the term list
constexpr size_t PD_SMALL = 6 * 1024, PD_MEDIUM = 20 * 1024;

// One term's sub-matrix, and the position of a cell's element in it: row =
// sk k + sl l over the term's row states, column likewise.
struct PdTerm {
  const double* zb;  // element (0, 0)
  int ldz;           // leading dimension of the cc block
  int nrow, ncol;
  int r[4], c[4];    // row and column strides of k1, k2, l1, l2
  double sgn;
};

// The tile's terms into d (at most four, in the order of t), by lanes 0 to 3
// of the first warp.
__device__ __forceinline__ void pd_terms(const DevLayout& L, const int2* __restrict__ zrow, int ng,
                                         const double* __restrict__ Z, int2 gb, int2 gk, int n1, int n2, int n3, int n4,
                                         PdTerm* d, int* nt) {
  const int t = threadIdx.x & 3;
  const bool lo = t < 2, same = t == 0 || t == 3;  // rows by l1 or l2; by k1 or k2
  const int G1 = lo ? gk.x : gk.y, G2 = same ? gb.x : gb.y, G3 = same ? gb.y : gb.x, G4 = lo ? gk.y : gk.x;
  const int2 zr = __ldg(&zrow[G1 * ng + G2]);
  const int zc = __ldg(&zrow[G3 * ng + G4]).y;
  const bool on = zr.x >= L.ncc - 1 - zr.x;  // else summed into the opposite block
  const unsigned act = __ballot_sync(0xffffffffu, on && threadIdx.x < 4);
  if (threadIdx.x == 0) *nt = __popc(act);
  if (!on || threadIdx.x >= 4) return;
  const int m2 = same ? n1 : n2, m3 = same ? n2 : n1, m1 = lo ? n3 : n4, m4 = lo ? n4 : n3;
  PdTerm& p = d[__popc(act & ((1u << t) - 1))];
  p.ldz = __ldg(&L.ccdim[zr.x]).x;
  p.zb = Z + __ldg(&L.cczoff[zr.x]) + zr.y + (i64)zc * p.ldz;
  p.nrow = m1 * m2;
  p.ncol = m3 * m4;
  p.r[0] = same ? 1 : 0;
  p.r[1] = same ? 0 : 1;
  p.r[2] = lo ? m2 : 0;
  p.r[3] = lo ? 0 : m2;
  p.c[0] = same ? 0 : m4;
  p.c[1] = same ? m4 : 0;
  p.c[2] = lo ? 0 : 1;
  p.c[3] = lo ? 1 : 0;
  p.sgn = t & 1 ? -1.0 : 1.0;
}

// copy term d's sub-matrix into dst (runs of nrow doubles, coalesced)
template <int T>
__device__ __forceinline__ void pd_stage(const PdTerm& d, double* dst, int tid) {
  const int total = d.nrow * d.ncol;
  const int2 i0 = divmod_small(tid, d.nrow), di = divmod_small(T, d.nrow);
  int fr = i0.y, fc = i0.x;
  for (int e = tid; e < total; e += T) {
    cp_async8(&dst[e], d.zb + fr + (i64)fc * d.ldz);
    fr += di.y;
    fc += di.x;
    if (fr >= d.nrow) {
      fr -= d.nrow;
      ++fc;
    }
  }
}

template <int MODE, int T>
__global__ void __launch_bounds__(T) k_pandya_tile(DevLayout L, const int* __restrict__ tasks,
                                                     const int2* __restrict__ tiles, const int4* __restrict__ gpd,
                                                     const int2* __restrict__ gpp, const int2* __restrict__ gpg,
                                                     const int2* __restrict__ zrow, int ng,
                                                     const double* __restrict__ Z, double* __restrict__ C) {
  extern __shared__ __align__(16) double smp[];
  __shared__ PdTerm d[4];
  __shared__ int snt;
  const int2 tl = __ldg(&tiles[__ldg(&tasks[blockIdx.x])]);
  const GpDesc da = load_gp(gpd, tl.x), db = load_gp(gpd, tl.y);
  const int n1 = da.n1, n2 = da.n2, n3 = db.n1, n4 = db.n2;
  const int cells = n1 * n2 * n3 * n4;
  const int pa = da.cnt(0) + da.cnt(1) + da.cnt(2), pb = db.cnt(0) + db.cnt(1) + db.cnt(2);
  const int q = da.q;
  const int4 bd = __ldg(&L.blk[q]);
  const i64* boff = L.boff + 6 * q;
  const int tid = threadIdx.x;
  if (tid < 32) pd_terms(L, zrow, ng, Z, __ldg(&gpg[tl.x]), __ldg(&gpg[tl.y]), n1, n2, n3, n4, d, &snt);
  __syncthreads();
  const int nt = snt;
  int nst = 0;  // stored cells: regions c1 >= c2
#pragma unroll 1
  for (int c1 = 0; c1 < 3; ++c1)
    for (int c2 = 0; c2 <= c1; ++c2) nst += da.cnt(c1) * db.cnt(c2);
  // shared memory: sub-matrix buffers | accumulator | row, column pairs
  double* Zs = smp;
  double* Y = smp + (MODE == PD_ALL ? nt * cells : (MODE == PD_SINGLE ? cells : 0));
  int2* pr = reinterpret_cast<int2*>(Y + (MODE == PD_SINGLE ? nst : 0));
  int2* pc = pr + pa;
  for (int i = tid; i < pa; i += T) pr[i] = __ldg(&gpp[da.pstart + i]);
  for (int i = tid; i < pb; i += T) pc[i] = __ldg(&gpp[db.pstart + i]);
  const int npass = MODE == PD_SINGLE ? nt : 1;
#pragma unroll 1
  for (int pass = 0; pass < npass; ++pass) {
    if (MODE == PD_SINGLE) {
      if (pass > 0) __syncthreads();  // the buffer is free again
      pd_stage<T>(d[pass], Zs, tid);
      cp_async_wait_all();
    } else if (MODE == PD_ALL) {
#pragma unroll 1
      for (int t = 0; t < nt; ++t) pd_stage<T>(d[t], Zs + t * cells, tid);
      cp_async_wait_all();
    }
    __syncthreads();
    int j0 = 0;  // first accumulator slot of the region
#pragma unroll 1
    for (int rg = 0; rg < 6; ++rg) {
      const int c1 = rg < 1 ? 0 : (rg < 3 ? 1 : 2), c2 = rg - (c1 * (c1 + 1)) / 2;
      const int r1 = da.cnt(c1), r2 = db.cnt(c2);
      if (r1 == 0 || r2 == 0) continue;
      const int o1 = da.off(c1), o2 = db.off(c2);
      const i64 base = __ldg(boff + slot_of(c1, c2));
      const i64 ldc = cnt_of(c1, bd);
      const int2 i0 = divmod_small(tid, r1), di = divmod_small(T, r1);
      int p = i0.y, u = i0.x;
#pragma unroll 2
      for (int e = tid; e < r1 * r2; e += T) {
        const int2 P = pr[o1 + p], Q = pc[o2 + u];
        p += di.y;
        u += di.x;
        if (p >= r1) {
          p -= r1;
          ++u;
        }
        double* out = C + base + P.x + (i64)Q.x * ldc;
        const bool last = MODE != PD_SINGLE || pass == npass - 1;
        const double old = last ? *out : 0.0;
        const int k1 = (P.y >> 17) & 15, k2 = (P.y >> 21) & 15;
        const int l1 = (Q.y >> 17) & 15, l2 = (Q.y >> 21) & 15;
        double y = MODE == PD_SINGLE && pass > 0 ? Y[j0 + e] : 0.0;
#pragma unroll 1
        for (int t = MODE == PD_SINGLE ? pass : 0; t < (MODE == PD_SINGLE ? pass + 1 : nt); ++t) {
          const PdTerm& D = d[t];
          const int row = k1 * D.r[0] + k2 * D.r[1] + l1 * D.r[2] + l2 * D.r[3];
          const int col = k1 * D.c[0] + k2 * D.c[1] + l1 * D.c[2] + l2 * D.c[3];
          const double z = MODE == PD_DIRECT ? __ldg(D.zb + row + (i64)col * D.ldz)
                                             : Zs[(MODE == PD_ALL ? t * cells : 0) + row + col * D.nrow];
          y += D.sgn * z;
        }
        if (!last) {
          Y[j0 + e] = y;
        } else {
          if ((P.y ^ Q.y) & (1 << 16)) y = -y;
          *out = old + y;
        }
      }
      j0 += r1 * r2;
    }
  }
}

// ---- host side --------------------------------------------------------------
namespace {
struct TileInfo {
  int a, b;          // group pairs
  int cells;         // nr * nc
  int nf, npair;     // F entries (double2) and pair entries of the two group pairs
  int nr, nc;
  unsigned parts;    // two-body parts the tile touches (bit = vectorize slot)
  int nst;           // stored output cells
  bool holefree;     // none of the four (m_l, m_s) groups holds a hole
};
struct PdBucket {  // one launch of the particle-hole tile kernel
  int first, count;
  size_t smem;
  int mode;  // PD_ALL, PD_SINGLE or PD_DIRECT
};
struct Bucket122 {
  int tw;       // doubles per staged cell
  int first;    // range in the task array
  int count;
  size_t smem;
  int list = 0;          // 0 one operand (sets C), 1 both operands, 2 one operand (accumulates)
  int threads = 256;    // CTA size (autotuned)
  float ms[3] = {0, 0, 0};  // measured time of the 64-, 128- and 256-thread variants
};
struct TaskSet {
  int2* d_task = nullptr;
  std::vector<Bucket122> buckets;
  bool tuned = false;
  int bounds_id = 0;           // which bucketing (see kBounds) the tuner kept
  float ms_total = 0.f;        // tuned time of this bucketing
  std::vector<TaskSet> alts;   // the other bucketings, until tuned
};
struct Plan122 {
  int4* d_gpd = nullptr;
  int2* d_gpp = nullptr;
  int2* d_tiles = nullptr;
  int* d_sbase = nullptr;
  double2* d_ftab = nullptr;
  int gmax = 0, nfent = 0;
  std::vector<TileInfo> tiles;
  std::map<std::pair<unsigned, unsigned>, TaskSet> sets;  // per (zero mask A, zero mask B)
  // particle-hole channel: groups (g, h) of each group pair, the first cc row
  // of each group pair (G1, G2) as {cc block, row}, the tasks (tile indices)
  int2* d_gpg = nullptr;
  int2* d_zrow = nullptr;
  int ng = 0;
  int* d_ptask = nullptr;
  std::vector<PdBucket> pbuckets;
  // generator-like A: term tables of k_gen_pppp / k_122_gen and their tasks
  int* d_ppbase = nullptr;   // per block: first pp pair
  int* d_ppstart = nullptr;  // per pp pair: first term (one more entry at the end)
  int2* d_ppterm = nullptr;
  int* d_gbase = nullptr;    // 3 * nblock: first hh, ph, pp pair of each block
  int* d_rstart = nullptr;   // k_122_gen row and column term starts, per slot at gen_rso / gen_cso
  int* d_cstart = nullptr;
  int4* d_rterm = nullptr;
  int4* d_cterm = nullptr;
  int gen_rso[6] = {0}, gen_cso[6] = {0};
  int4* d_sptask = nullptr;  // C_pppp tile pairs, then the k_122_gen tiles, then the C_phph tile pairs
  int* d_ftask = nullptr;  // k_122_full: tile indices, by CTA size, largest first
  struct FullBucket {
    int first, count, threads;
    size_t smem;
    bool both;                // both operands staged together
    float ms[3] = {0, 0, 0};  // measured with 64, 128 and 256 threads
  };
  std::vector<FullBucket> fbuckets;
  bool full_fits = true;  // every tile fits k_122_full's shared memory
  bool full_tuned = false;
  int4* d_ltask = nullptr;   // k_gen_ladder: {block, role, first row}, longest first
  int nsp_ladder = 0;
  int nsp_pppp = 0, nsp_gen = 0;
  int pppp_terms = 0;    // the most terms one task of k_gen_pppp stages
  size_t gen_bytes = 0, phph_bytes = 0;  // the most shared memory a task of k_122_gen, k_gen_phph needs
  int nsp_phph = 0;
};
std::map<const qd_layout*, Plan122>& plans() {
  static std::map<const qd_layout*, Plan122> m;
  return m;
}
// plans of different layouts are built and dropped from concurrent host
// threads (batched flows)
std::mutex g_plan_mutex;

size_t tile_smem(const TileInfo& t, int tw) {
  const size_t ld = (size_t)(t.nc | 1);
  const size_t tsz = ((size_t)t.nr * ld * tw + 1) & ~(size_t)1;
  return 8 * tsz + 16 * (size_t)t.nf + 8 * (size_t)t.npair;
}
size_t full_smem(const TileInfo& t, int n1, int n2, int n3, int n4, bool both) {
  const size_t tsz = ((size_t)t.nr * (t.nc | 1) + 1) & ~(size_t)1;
  return 8 * ((both ? 3 : 2) * tsz + (both ? 2 : 1) * (size_t)(full_fsz(n1) + full_fsz(n2) + full_fsz(n3) + full_fsz(n4))) +
         8 * (size_t)t.npair;
}
// a task that only writes zeros keeps just the two pair lists
size_t zero_smem(const TileInfo& t) { return 8 * (size_t)t.npair; }

}  // namespace

static int plan_122(qd_layout* L, Plan122** out) {
  std::lock_guard<std::mutex> lock(g_plan_mutex);
  auto it = plans().find(L);
  if (it != plans().end()) {
    *out = &it->second;
    return QD_OK;
  }
  Plan122 p;
  const int m = L->m;
  const int ngroup = (int)L->gstart.size() - 1;
  std::vector<int> gsz(ngroup), goff(ngroup + 1, 0), kpos(m, 0), sbase(m, 0), holes(ngroup, 0);
  for (int g = 0; g < ngroup; ++g) {
    gsz[g] = L->gstart[g + 1] - L->gstart[g];
    p.gmax = std::max(p.gmax, gsz[g]);
    goff[g + 1] = goff[g] + gsz[g] * gsz[g];
    for (int k = 0; k < gsz[g]; ++k) {
      const int s = L->gmem[L->gstart[g] + k];
      kpos[s] = k;
      if (s < L->n) {
        if (k != holes[g]) {  // holes must be the lowest members of every group
          set_error("commutator_122: holes are not the lowest states of their (ml,ms) group");
          return QD_ERR_LAYOUT;
        }
        ++holes[g];
      }
    }
  }
  if (p.gmax > 16) {  // cells of a group pair fit the 8-bit cell fields
    set_error("commutator_122: (ml,ms) group of %d states exceeds 16", p.gmax);
    return QD_ERR_ARG;
  }
  p.nfent = goff[ngroup];
  for (int s = 0; s < m; ++s) sbase[s] = goff[L->gid[s]] + kpos[s] * gsz[L->gid[s]];

  std::vector<int4> gpd;
  std::vector<int2> gpp, gpg;
  struct GpHost {
    int n1, n2, cnt[3], nf, npair;
  };
  std::vector<int> gpidx((size_t)ngroup * ngroup, -1);  // place of a group pair in `order`, within a block
  for (int q = 0; q < L->nblock; ++q) {
    const int nh = L->blk[q].x, nb = L->blk[q].y, ntot = L->blk[q].w, pb = L->pbase[q];
    // group pairs in order of first appearance; per group pair its pairs in
    // class order (pairs are enumerated [hh | ph | pp], each class by index)
    std::vector<std::pair<int, int>> order;
    std::vector<std::vector<int2>> plist;  // {w, packed cells}
    std::vector<GpHost> gh;
    for (int P = 0; P < ntot; ++P) {
      const int2 pr = L->pairs[pb + P];  // 0-based states, pr.x < pr.y
      const int c = P < nh ? 0 : (P < nh + nb ? 1 : 2);
      const int w = P - (c == 0 ? 0 : (c == 1 ? nh : nh + nb));
      const int gi = L->gid[pr.x], gj = L->gid[pr.y];
      const int g = std::min(gi, gj), h = std::max(gi, gj);
      int& at = gpidx[(size_t)g * ngroup + h];
      if (at < 0) {
        at = (int)order.size();
        order.push_back({g, h});
        plist.emplace_back();
        gh.push_back(GpHost{gsz[g], gsz[h], {0, 0, 0}, 0, 0});
      }
      const int u = at;
      int t1, t2;
      if (g != h) {
        t1 = gi == g ? pr.x : pr.y;
        t2 = gi == g ? pr.y : pr.x;
      } else {
        t1 = pr.x;
        t2 = pr.y;
      }
      const int n2c = gsz[h];
      const int r = kpos[t1] * n2c + kpos[t2];
      const int neg = t1 > t2 ? 1 : 0;
      const int rm = g == h ? kpos[t2] * n2c + kpos[t1] : -1;
      if (gsz[g] * gsz[h] > 256 || r >= 255 || rm >= 255) {
        set_error("commutator_122: group pair of %d cells exceeds the cell fields", gsz[g] * gsz[h]);
        return QD_ERR_ARG;
      }
      plist[u].push_back(int2{w, r | ((rm + 1) << 8) | (neg << 16) | (kpos[t1] << 17) | (kpos[t2] << 21)});
      gh[u].cnt[c] += 1;
    }
    for (const auto& o : order) gpidx[(size_t)o.first * ngroup + o.second] = -1;
    const int u0 = (int)gpd.size() / 2;
    for (size_t u = 0; u < order.size(); ++u) {
      const int g = order[u].first, h = order[u].second;
      GpHost& d = gh[u];
      if (d.cnt[0] > 1023 || d.cnt[1] > 1023 || d.cnt[2] > 1023) {
        set_error("commutator_122: group pair class count exceeds 1023");
        return QD_ERR_ARG;
      }
      d.nf = d.n1 * d.n1 + d.n2 * d.n2;
      d.npair = d.cnt[0] + d.cnt[1] + d.cnt[2];
      gpd.push_back(int4{q, d.n1 | (d.n2 << 8) | ((g == h ? 1 : 0) << 16), holes[g] | (holes[h] << 8), goff[g]});
      gpd.push_back(int4{goff[h], (int)gpp.size(), 0, d.cnt[0] | (d.cnt[1] << 10) | (d.cnt[2] << 20)});
      gpg.push_back(int2{g, h});
      gpp.insert(gpp.end(), plist[u].begin(), plist[u].end());
    }
    // tiles: every ordered pair of group pairs with at least one stored
    // output cell (a row class >= a column class)
    for (size_t a = 0; a < order.size(); ++a)
      for (size_t b = 0; b < order.size(); ++b) {
        const GpHost &A = gh[a], &B = gh[b];
        bool out = false;
        unsigned parts = 0;
        for (int c1 = 0; c1 < 3; ++c1)
          for (int c2 = 0; c2 < 3; ++c2)
            if (A.cnt[c1] > 0 && B.cnt[c2] > 0) {
              parts |= 1u << (c1 >= c2 ? slot_of(c1, c2) : slot_of(c2, c1));
              if (c1 >= c2) out = true;
            }
        if (!out) continue;
        TileInfo t;
        t.a = u0 + (int)a;
        t.b = u0 + (int)b;
        t.nr = A.n1 * A.n2;
        t.nc = B.n1 * B.n2;
        t.cells = t.nr * t.nc;
        t.nf = A.nf + B.nf;
        t.npair = A.npair + B.npair;
        t.parts = parts;
        t.holefree = holes[order[a].first] == 0 && holes[order[a].second] == 0 && holes[order[b].first] == 0 &&
                     holes[order[b].second] == 0;
        t.nst = 0;
        for (int c1 = 0; c1 < 3; ++c1)
          for (int c2 = 0; c2 <= c1; ++c2) t.nst += A.cnt[c1] * B.cnt[c2];
        p.tiles.push_back(t);
      }
  }
  for (const TileInfo& t : p.tiles)
    if (tile_smem(t, 1) > SMEM_MAX_122) {
      set_error("commutator_122: tile of %d cells exceeds shared memory", t.cells);
      return QD_ERR_ARG;
    }
  std::vector<int2> th(p.tiles.size());
  for (size_t i = 0; i < p.tiles.size(); ++i) th[i] = int2{p.tiles[i].a, p.tiles[i].b};
  PlanMemory mem;
  mem.add(std::move(gpd), &p.d_gpd);
  mem.add(std::move(gpp), &p.d_gpp);
  mem.add(std::move(th), &p.d_tiles);
  mem.add(std::move(sbase), &p.d_sbase);
  // generator-like A: the pp pairs' W terms (k_gen_pppp) and the row and
  // column terms of the other five parts (k_122_gen), per block
  {
    const int n = L->n, mp = L->mp;
    const int ofph = (int)L->o_fph, ofpp = (int)L->o_fpp, ofhh = (int)L->o_fhh;
    std::vector<int> gbase(3 * L->nblock), ppstart(1, 0);
    std::vector<int2> ppterm;
    // per slot: its terms and, per pair of its classes (block order), their starts
    std::vector<int> rst[6], cst[6];
    std::vector<int4> rterm_s[6], cterm_s[6];
    std::vector<int4> ptask, gtask, htask;
    // room for the most terms there can be (memory that is not touched costs
    // nothing, growing the arrays copies them several times over)
    {
      size_t pairs[3] = {0, 0, 0};
      for (int q = 0; q < L->nblock; ++q) {
        pairs[0] += L->blk[q].x;
        pairs[1] += L->blk[q].y;
        pairs[2] += L->blk[q].z;
      }
      for (int slot : {0, 2, 3, 4, 5}) {
        int cr, cc;
        part_classes(P_HHHH + slot, cr, cc);
        rterm_s[slot].reserve(pairs[cr] * 3 * p.gmax);
        cterm_s[slot].reserve(pairs[cc] * 3 * p.gmax);
      }
    }
    int cnt[3] = {0, 0, 0};
    enum { NEG = 1, MA = 2, MB = 4, CB = 8 };
    auto fA = [&](int pt, int h) { return ofph + (pt - n) + h * mp; };  // A's or B's fph(p, h)
    auto fpp = [&](int t, int b) { return ofpp + (t - n) + (b - n) * mp; };
    auto fhh = [&](int k, int t) { return ofhh + k + t * n; };
    auto src = [](int opd, int slot, int tr) { return (opd << 4) | (tr << 3) | slot; };
    for (int q = 0; q < L->nblock; ++q) {
      const int nh = L->blk[q].x, nb = L->blk[q].y, np = L->blk[q].z, pb = L->pbase[q];
      for (int c = 0; c < 3; ++c) gbase[c * L->nblock + q] = cnt[c];
      cnt[0] += nh;
      cnt[1] += nb;
      cnt[2] += np;
      // index of the pair (u, v), u < v, among the pairs of class c of this block, or -1
      auto at = [&](int c, int u, int v) {
        if (u >= v) return -1;
        const int e = L->ptab[(size_t)u * m + v];
        return e >= 0 && pt_blk(e) == q && pt_cls(e) == c ? pt_idx(e) : -1;
      };
      auto grp = [&](int x) { return std::make_pair(L->gstart[L->gid[x]], L->gstart[L->gid[x] + 1]); };
      // members t of G(x) that are holes (want_hole) or particles, excluding `skip`
      auto each = [&](int x, bool want_hole, int skip, auto fn) {
        const auto mr = grp(x);
        for (int u = mr.first; u < mr.second; ++u) {
          const int tt = L->gmem[u];
          if ((tt < n) == want_hole && tt != skip) fn(tt);
        }
      };
      // index and ordering sign of the pair {u, v}
      auto srt = [&](int c, int u, int v, int* idx, int* sg) {
        *idx = at(c, std::min(u, v), std::max(u, v));
        *sg = u < v ? 1 : -1;
        return *idx >= 0;
      };
      const auto hhp = [&](int k) { return L->pairs[pb + k]; };
      const auto php = [&](int k) { return L->pairs[pb + nh + k]; };
      const auto ppp = [&](int k) { return L->pairs[pb + nh + nb + k]; };
      int idx, sg;
      // pp pairs (a, b): W terms +fA(a,t) B_ppph(., (t,b)), -fA(b,t) B_ppph(., (t,a)), holes t
      for (int k = 0; k < np; ++k) {
        const int x0 = ppp(k).x, y0 = ppp(k).y;
        for (int side = 0; side < 2; ++side) {
          const int x = side ? y0 : x0, y = side ? x0 : y0;
          each(x, true, -1, [&](int t) {
            const int f = at(1, t, y);
            if (f >= 0) ppterm.push_back(int2{f, (t) | ((x - n) << 8) | ((side ? 1 : 0) << 20)});
          });
        }
        ppstart.push_back((int)ppterm.size());
      }
      // row terms, per slot over the pairs of its row class
      auto rows_of = [&](int slot, int k) {
        std::vector<int4>& T = rterm_s[slot];
        if (slot == 4 || slot == 2) {  // rows pp (x, y)
          const int x0 = ppp(k).x, y0 = ppp(k).y;
          for (int side = 0; side < 2; ++side) {
            const int x = side ? y0 : x0, y = side ? x0 : y0;
            each(x, true, -1, [&](int t) {
              const int f = at(1, t, y);
              if (f >= 0) T.push_back(int4{f, fA(x, t), side ? NEG : 0, src(1, slot == 4 ? 3 : 5, 0)});
            });
            if (slot == 2)  // -s hB fppB(t, x) A_pphh((t,y)) over particles t in G(x)
              each(x, false, y, [&](int t) {
                if (srt(2, side ? y : t, side ? t : y, &idx, &sg))
                  T.push_back(int4{idx, fpp(t, x), MB | CB | (sg > 0 ? NEG : 0), src(0, 2, 0)});
              });
          }
        } else if (slot == 5 || slot == 3) {  // rows ph (h, p)
          const int h = php(k).x, pt = php(k).y;
          each(h, false, pt, [&](int t) {
            if (!srt(2, t, pt, &idx, &sg)) return;
            if (slot == 5) {
              T.push_back(int4{idx, fA(t, h), MA | (sg < 0 ? NEG : 0), src(1, 2, 0)});
              T.push_back(int4{idx, fA(t, h), MB | CB | (sg > 0 ? NEG : 0), src(0, 2, 0)});
            } else {
              T.push_back(int4{idx, fA(t, h), MA | (sg < 0 ? NEG : 0), src(1, 4, 0)});
            }
          });
          each(pt, true, h, [&](int t) {
            if (!srt(0, h, t, &idx, &sg)) return;
            if (slot == 5)
              T.push_back(int4{idx, fA(pt, t), sg < 0 ? NEG : 0, src(1, 0, 0)});
            else
              T.push_back(int4{idx, fA(pt, t), MB | (sg < 0 ? NEG : 0), src(1, 5, 1)});
          });
        } else {  // slot 0, rows hh (b1, b2)
          const int b1 = hhp(k).x, b2 = hhp(k).y;
          each(b1, false, -1, [&](int t) {
            const int f = at(1, b2, t);
            if (f >= 0) T.push_back(int4{f, fA(t, b1), MA | NEG, src(1, 5, 0)});
          });
          each(b2, false, -1, [&](int t) {
            const int f = at(1, b1, t);
            if (f >= 0) T.push_back(int4{f, fA(t, b2), MA, src(1, 5, 0)});
          });
        }
      };
      auto cols_of = [&](int slot, int k) {
        std::vector<int4>& T = cterm_s[slot];
        if (slot == 4) {  // columns ph (h, p)
          const int h = php(k).x, pt = php(k).y;
          each(h, false, pt, [&](int t) {
            if (srt(2, t, pt, &idx, &sg)) T.push_back(int4{idx, fA(t, h), sg > 0 ? NEG : 0, src(1, 1, 0)});
          });
          each(pt, true, h, [&](int t) {
            if (!srt(0, h, t, &idx, &sg)) return;
            T.push_back(int4{idx, fA(pt, t), MA | (sg > 0 ? NEG : 0), src(1, 2, 0)});
            T.push_back(int4{idx, fA(pt, t), MB | CB | (sg < 0 ? NEG : 0), src(0, 2, 0)});
          });
        } else if (slot == 3) {  // none: k_gen_phph transposes the row terms
        } else {  // columns hh (k1, k2): slots 2, 5, 0
          const int k1 = hhp(k).x, k2 = hhp(k).y;
          for (int side = 0; side < 2; ++side) {
            const int kk = side ? k2 : k1, ko = side ? k1 : k2;
            each(kk, false, -1, [&](int t) {
              const int f = at(1, ko, t);
              if (f < 0) return;
              const int ng = side ? NEG : 0;
              if (slot == 2) T.push_back(int4{f, fA(t, kk), ng, src(1, 4, 0)});
              else if (slot == 5) T.push_back(int4{f, fA(t, kk), ng, src(1, 3, 0)});
              else T.push_back(int4{f, fA(t, kk), MB | ng, src(1, 5, 1)});
            });
            if (slot == 2)  // +s hB fhhB(kk, t) A_pphh(., (t,ko)) over holes t in G(kk)
              each(kk, true, ko, [&](int t) {
                if (srt(0, side ? ko : t, side ? t : ko, &idx, &sg))
                  T.push_back(int4{idx, fhh(kk, t), MB | CB | (sg < 0 ? NEG : 0), src(0, 2, 0)});
              });
          }
        }
      };
      const int rows_n[6] = {nh, 0, np, nb, np, nb}, cols_n[6] = {nh, 0, nh, nb, nb, nh};
      for (int slot : {0, 2, 3, 4, 5}) {
        int cr, cc;
        part_classes(P_HHHH + slot, cr, cc);
        const int nr = cr == 0 ? nh : (cr == 1 ? nb : np), nc = cc == 0 ? nh : (cc == 1 ? nb : np);
        for (int k = 0; k < nr; ++k) {
          rows_of(slot, k);
          rst[slot].push_back((int)rterm_s[slot].size());  // end of pair k's terms
        }
        for (int k = 0; k < nc; ++k) {
          cols_of(slot, k);
          cst[slot].push_back((int)cterm_s[slot].size());
        }
        if (rows_n[slot] > 0 && cols_n[slot] > 0)
          for (int i = 0; i < (rows_n[slot] + SP_B - 1) / SP_B; ++i)
            for (int j = slot == 3 ? i : 0; j < (cols_n[slot] + SP_B - 1) / SP_B; ++j)
              (slot == 3 ? htask : gtask).push_back(int4{q, slot, i, j});
      }
      const int tr = (np + GP_B - 1) / GP_B;
      for (int i = 0; i < tr; ++i)
        for (int j = i; j < tr; ++j) ptask.push_back(int4{q, i, j, 0});
    }
    // per slot start arrays: one entry per pair of its class (in block order) plus one
    // concatenated: per slot a start 0 then the pairs' ends, shifted by the
    // slot's first term in the joint term arrays
    std::vector<int> rall, call;
    int r0 = 0, c0 = 0;
    const auto next = [](int at, size_t n) {  // where PlanMemory places the terms of the next slot
      constexpr int A = (int)(PlanMemory::ALIGN / sizeof(int4));
      return at + ((int)n + A - 1) / A * A;
    };
    for (int slot = 0; slot < 6; ++slot) {
      p.gen_rso[slot] = (int)rall.size();
      p.gen_cso[slot] = (int)call.size();
      rall.push_back(r0);
      for (int e : rst[slot]) rall.push_back(r0 + e);
      call.push_back(c0);
      for (int e : cst[slot]) call.push_back(c0 + e);
      r0 = next(r0, rterm_s[slot].size());
      c0 = next(c0, cterm_s[slot].size());
    }
    p.nsp_pppp = (int)ptask.size();
    p.nsp_gen = (int)gtask.size();
    // the parts with many terms per element first (their CTAs run longest),
    // then ppph, whose many CTAs fill the rest
    std::stable_sort(gtask.begin(), gtask.end(), [](const int4& x, const int4& y) {
      const auto rank = [](int slot) { return slot == 5 ? 0 : (slot == 2 ? 1 : (slot == 0 ? 2 : 3)); };
      return rank(x.y) < rank(y.y);
    });
    // the most terms one task stages (its shared memory)
    p.pppp_terms = 0;
    for (const int4& tk : ptask) {
      const int q = tk.x, np = L->blk[q].z, pbq = gbase[2 * L->nblock + q];
      int ne = 0;
      for (int pass = 0; pass < (tk.y == tk.z ? 1 : 2); ++pass) {
        const int c0 = (pass == 0 ? tk.z : tk.y) * GP_B, nc = std::min(GP_B, np - c0);
        ne += ppstart[pbq + c0 + nc] - ppstart[pbq + c0];
      }
      p.pppp_terms = std::max(p.pppp_terms, ne);
    }
    p.gen_bytes = p.phph_bytes = 0;
    for (const std::vector<int4>* v : {&gtask, &htask})
      for (const int4& tk : *v) {
        const int q = tk.x, slot = tk.y;
        int cr, cc;
        part_classes(P_HHHH + slot, cr, cc);
        const int4 bd = L->blk[q];
        const int nr = cr == 0 ? bd.x : (cr == 1 ? bd.y : bd.z), nc = cc == 0 ? bd.x : (cc == 1 ? bd.y : bd.z);
        const int i0 = tk.z * SP_B, j0 = tk.w * SP_B, nrt = std::min(SP_B, nr - i0), nct = std::min(SP_B, nc - j0);
        const int* rr = rall.data() + p.gen_rso[slot] + gbase[cr * L->nblock + q];
        const int* cs = call.data() + p.gen_cso[slot] + gbase[cc * L->nblock + q];
        const int rows = rr[i0 + nrt] - rr[i0];
        if (slot == 3)  // the pair's row terms beside its transposed tile
          p.phph_bytes = std::max(p.phph_bytes, sizeof(double) * SP_B * (SP_B + 1) +
                                                    gen_smem(rows + (i0 == j0 ? 0 : rr[j0 + nct] - rr[j0])));
        else
          p.gen_bytes = std::max(p.gen_bytes, gen_smem(rows + cs[j0 + nct] - cs[j0]));
      }
    if (gp_smem(p.pppp_terms) > SMEM_MAX_122 - 1024 ||
        std::max(p.gen_bytes, p.phph_bytes) > SMEM_MAX_122 - 1024) {
      set_error("commutator_122: the terms of one tile exceed shared memory");
      return QD_ERR_ARG;
    }
    std::vector<int4> all = ptask;
    all.insert(all.end(), gtask.begin(), gtask.end());
    all.insert(all.end(), htask.begin(), htask.end());
    p.nsp_phph = (int)htask.size();
    std::vector<std::pair<i64, int4>> lt;
    for (int q = 0; q < L->nblock; ++q) {
      if (!gen_ladder_fused(L, q) || L->blk[q].z == 0) continue;
      const int4 bd = L->blk[q];
      for (int r = 0; r < bd.z; r += 64) lt.push_back({(i64)bd.z * 64, int4{q, 0, r, 0}});
      for (int r = 0; r < bd.y; r += 16) lt.push_back({(i64)bd.z * 16, int4{q, 1, r, 0}});
      lt.push_back({(i64)bd.z * 16, int4{q, 2, 0, 0}});
    }
    std::stable_sort(lt.begin(), lt.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
    std::vector<int4> ltask;
    for (const auto& x : lt) ltask.push_back(x.second);
    p.nsp_ladder = (int)ltask.size();
    mem.add(std::move(ltask), &p.d_ltask);
    std::vector<int> ppbase(L->nblock);
    for (int q = 0; q < L->nblock; ++q) ppbase[q] = gbase[2 * L->nblock + q];
    mem.add(std::move(ppbase), &p.d_ppbase);
    mem.add(std::move(ppstart), &p.d_ppstart);
    mem.add(std::move(ppterm), &p.d_ppterm);
    mem.add(std::move(gbase), &p.d_gbase);
    mem.add(std::move(rall), &p.d_rstart);
    mem.add(std::move(call), &p.d_cstart);
    for (int slot = 0; slot < 6; ++slot) mem.add(std::move(rterm_s[slot]), slot ? (int4**)nullptr : &p.d_rterm);
    for (int slot = 0; slot < 6; ++slot) mem.add(std::move(cterm_s[slot]), slot ? (int4**)nullptr : &p.d_cterm);
    mem.add(std::move(all), &p.d_sptask);
  }
  {  // k_122_full: buckets by shared memory, small tiles with fewer threads
    std::vector<std::pair<size_t, int>> v;
    for (size_t i = 0; i < p.tiles.size(); ++i) {
      const TileInfo& t = p.tiles[i];
      const int2 gb = gpg[t.a], gk = gpg[t.b];
      const size_t two = full_smem(t, gsz[gb.x], gsz[gb.y], gsz[gk.x], gsz[gk.y], true);
      v.push_back({two <= FULL_BOTH ? two : FULL_BOTH + full_smem(t, gsz[gb.x], gsz[gb.y], gsz[gk.x], gsz[gk.y], false),
                   (int)i});  // beyond FULL_BOTH: one operand at a time
    }
    std::stable_sort(v.begin(), v.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
    p.full_fits = v.empty() || v[0].first <= FULL_BOTH + SMEM_MAX_122 - 1024;
    std::vector<int> tasks;
    size_t i = 0;
    while (i < v.size()) {
      size_t lower = 0;
      for (size_t b : FULL_BOUNDS)
        if (b < v[i].first) lower = std::max(lower, b);
      Plan122::FullBucket b;
      b.first = (int)tasks.size();
      b.both = v[i].first <= FULL_BOTH;
      b.smem = b.both ? v[i].first : v[i].first - FULL_BOTH;
      b.threads = !b.both ? 256 : (b.smem <= FULL_SMALL ? 64 : 128);
      while (i < v.size() && v[i].first > lower) tasks.push_back(v[i++].second);
      b.count = (int)tasks.size() - b.first;
      // column strips together (see build_variant)
      std::stable_sort(tasks.begin() + b.first, tasks.end(), [&](int x, int y) {
        return p.tiles[x].b != p.tiles[y].b ? p.tiles[x].b < p.tiles[y].b : p.tiles[x].a < p.tiles[y].a;
      });
      p.fbuckets.push_back(b);
    }
    mem.add(std::move(tasks), &p.d_ftask);
  }
  // particle-hole channel: first cc row of each (G1, G2) and the launches
  p.ng = ngroup;
  std::vector<int2> zrow((size_t)ngroup * ngroup);
  for (int g1 = 0; g1 < ngroup; ++g1)
    for (int g2 = 0; g2 < ngroup; ++g2)
      zrow[(size_t)g1 * ngroup + g2] = L->ccmap[(size_t)L->gmem[L->gstart[g1]] * m + L->gmem[L->gstart[g2]]];
  {
    // per tile the first mode that fits: all its terms staged, one buffer,
    // none; buckets by mode, then by size interval, largest first
    struct PdT {
      int mode;
      size_t sm;
      int tile;
    };
    std::vector<PdT> lst;
    for (size_t i = 0; i < p.tiles.size(); ++i) {
      const TileInfo& t = p.tiles[i];
      const int2 gb = gpg[t.a], gk = gpg[t.b];
      int nt = 0;  // as pd_terms
      for (int k = 0; k < 4; ++k) {
        const int q = zrow[(size_t)(k < 2 ? gk.x : gk.y) * ngroup + (k == 0 || k == 3 ? gb.x : gb.y)].x;
        nt += q >= L->ncc - 1 - q;
      }
      const size_t c = (size_t)t.cells, ns = (size_t)t.nst, np = (size_t)t.npair;
      const size_t sa = 8 * (nt * c + np), s1 = 8 * (c + ns + np);
      if (sa <= PD_SMEM)
        lst.push_back({PD_ALL, sa, (int)i});
      else if (s1 <= PD_SMEM)
        lst.push_back({PD_SINGLE, s1, (int)i});
      else
        lst.push_back({PD_DIRECT, 8 * np, (int)i});
    }
    const size_t bounds[5] = {PD_SMALL, PD_MEDIUM, 48 * 1024, 112 * 1024, SMEM_MAX_122};
    auto interval = [&](size_t sm) {
      int l = 0;
      while (l < 4 && sm > bounds[l]) ++l;
      return l;
    };
    std::stable_sort(lst.begin(), lst.end(), [&](const PdT& x, const PdT& y) {
      return x.mode != y.mode ? x.mode < y.mode : x.sm > y.sm;
    });
    std::vector<int> tasks;
    size_t i = 0;
    while (i < lst.size()) {
      const int mode = lst[i].mode, l = interval(lst[i].sm);
      PdBucket b{(int)tasks.size(), 0, lst[i].sm, mode};
      while (i < lst.size() && lst[i].mode == mode && interval(lst[i].sm) == l) tasks.push_back(lst[i++].tile);
      b.count = (int)tasks.size() - b.first;
      p.pbuckets.push_back(b);
    }
    mem.add(std::move(gpg), &p.d_gpg);
    mem.add(std::move(zrow), &p.d_zrow);
    mem.add(std::move(tasks), &p.d_ptask);
  }
  mem.room(2 * (i64)p.nfent, &p.d_ftab);
  for (const void* fn : {(const void*)k_122_tile<1, 64>, (const void*)k_122_tile<2, 64>,
                         (const void*)k_122_tile<1, 128>, (const void*)k_122_tile<2, 128>,
                         (const void*)k_122_tile<1, 256>, (const void*)k_122_tile<2, 256>,
                         (const void*)k_122_full<64, true>, (const void*)k_122_full<128, true>, (const void*)k_122_full<256, true>,
                         (const void*)k_122_full<64, false>, (const void*)k_122_full<128, false>, (const void*)k_122_full<256, false>,
                         (const void*)k_pandya_tile<PD_ALL, 64>, (const void*)k_pandya_tile<PD_ALL, 128>,
                         (const void*)k_pandya_tile<PD_ALL, 256>,
                         (const void*)k_pandya_tile<PD_SINGLE, 256>, (const void*)k_pandya_tile<PD_DIRECT, 256>,
                         (const void*)k_gen_pppp<false>, (const void*)k_gen_pppp<true>, (const void*)k_122_gen, (const void*)k_gen_phph}) {
    cudaFuncAttributes fa;
    QD_CUDA(cudaFuncGetAttributes(&fa, fn));
    QD_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)SMEM_MAX_122 - (int)fa.sharedSizeBytes));
  }
  const int rc = mem.commit(L);
  if (rc) return rc;
  Plan122& kept = plans()[L];
  kept = std::move(p);
  *out = &kept;
  return QD_OK;
}

// Tasks for one pair of zero-part masks: per tile the terms it needs, in
// buckets of similar shared memory (largest first).  A tile that needs both
// terms but does not fit with both operands staged runs as a B task that
// sets C and an A task (in a later launch) that accumulates.
// Bucketings the autotuner chooses from: the size bounds (bytes of shared
// memory) that split each list into launches.  More buckets give small tiles
// more CTAs per SM; fewer keep the tiles of one column strip in one launch.
constexpr int kNumBounds = 4, kBoundsLen = 6;
const size_t kBounds[kNumBounds][kBoundsLen] = {
    {24 * 1024, 56 * 1024, 112 * 1024, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122},
    {56 * 1024, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122},
    {SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122, SMEM_MAX_122},
    {8 * 1024, 16 * 1024, 24 * 1024, 56 * 1024, 112 * 1024, SMEM_MAX_122}};

// One bucketing of the task lists: buckets by size bound (largest first),
// and within a bucket the tiles sharing a column strip (block q, column
// group pair b) together: their gathers read the same columns, whose memory
// atoms also hold neighbouring group pairs' rows, so concurrent CTAs hit in
// L2.
static int build_variant(qd_layout* L, const Plan122* p, std::vector<std::pair<size_t, int2>> lst_in[3], int bid,
                         TaskSet& ts) {
  std::vector<int2> all;
  const size_t* bounds = kBounds[bid];
  ts.bounds_id = bid;
  for (int l = 0; l < 3; ++l) {
    std::vector<std::pair<size_t, int2>> v = lst_in[l];
    std::stable_sort(v.begin(), v.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
    size_t i = 0;
    while (i < v.size()) {
      // bucket: tasks down to the next size bound below the first one
      const size_t top = v[i].first;
      size_t lower = 0;
      for (int k = 0; k < kBoundsLen; ++k)
        if (bounds[k] < top) lower = std::max(lower, bounds[k]);
      Bucket122 b;
      b.tw = l == 1 ? 2 : 1;
      b.list = l;
      b.first = (int)all.size();
      b.smem = top;
      while (i < v.size() && v[i].first > lower) all.push_back(v[i++].second);
      b.count = (int)all.size() - b.first;
      ts.buckets.push_back(b);
    }
  }
  for (const Bucket122& bk : ts.buckets)
    std::stable_sort(all.begin() + bk.first, all.begin() + bk.first + bk.count, [&](const int2& x, const int2& y) {
      const TileInfo &tx = p->tiles[x.x], &ty = p->tiles[y.x];
      return tx.b != ty.b ? tx.b < ty.b : tx.a < ty.a;
    });
  QD_CUDA(cudaMalloc(&ts.d_task, std::max<size_t>(1, all.size()) * sizeof(int2)));
  if (!all.empty()) QD_CUDA(copy_table(ts.d_task, all.data(), all.size() * sizeof(int2)));
  L->ws_bytes += (i64)(all.size() * sizeof(int2));
  return QD_OK;
}

static int task_set(qd_layout* L, Plan122* p, unsigned zA, unsigned zB, TaskSet** out) {
  std::lock_guard<std::mutex> lock(g_plan_mutex);
  auto key = std::make_pair(zA, zB);
  auto it = p->sets.find(key);
  if (it != p->sets.end()) {
    *out = &it->second;
    return QD_OK;
  }
  const unsigned one = (1u << P_FHH) | (1u << P_FPP) | (1u << P_FPH);
  const bool fa0 = (zA & one) == one, fb0 = (zB & one) == one;  // a one-body part entirely zero
  // a one-body part without hh and pp entries (the Magnus generator's) couples
  // holes to particles only: on a tile whose four groups hold no hole every
  // leg of its term sums over nothing
  const unsigned hp = (1u << P_FHH) | (1u << P_FPP);
  const bool spa = (zA & hp) == hp, spb = (zB & hp) == hp;
  const unsigned za2 = (zA >> P_HHHH) & 63u, zb2 = (zB >> P_HHHH) & 63u;
  // lists: 0 one operand (set), 1 both operands (set), 2 one operand (accumulate)
  std::vector<std::pair<size_t, int2>> lst[3];
  for (size_t i = 0; i < p->tiles.size(); ++i) {
    const TileInfo& t = p->tiles[i];
    const bool nb = !fa0 && (t.parts & ~zb2) && !(spa && t.holefree);
    const bool na = !fb0 && (t.parts & ~za2) && !(spb && t.holefree);
    const int op = (nb ? 1 : 0) | (na ? 2 : 0);
    if (op == 3) {
      if (tile_smem(t, 2) <= SMEM_MAX_122) {
        lst[1].push_back({tile_smem(t, 2), int2{(int)i, 3}});
      } else {
        lst[0].push_back({tile_smem(t, 1), int2{(int)i, 1}});
        lst[2].push_back({tile_smem(t, 1), int2{(int)i, 2 | 4}});
      }
    } else {
      lst[0].push_back({op ? tile_smem(t, 1) : zero_smem(t), int2{(int)i, op}});  // op 0: writes zeros
    }
  }
  TaskSet ts;
  for (int bid = 0; bid < kNumBounds; ++bid) {
    TaskSet& v = bid == 0 ? ts : (ts.alts.emplace_back(), ts.alts.back());
    int rc = build_variant(L, p, lst, bid, v);
    if (rc) return rc;
  }
  p->sets[key] = ts;
  *out = &p->sets[key];
  return QD_OK;
}

void drop_122_plan(const qd_layout* L) {
  std::lock_guard<std::mutex> lock(g_plan_mutex);
  auto it = plans().find(L);
  if (it == plans().end()) return;
  Plan122& p = it->second;
  for (auto& kv : p.sets) {
    if (kv.second.d_task) cudaFree(kv.second.d_task);
    for (TaskSet& t : kv.second.alts)
      if (t.d_task) cudaFree(t.d_task);
  }
  plans().erase(it);
}

// class pairs (c1 * 3 + c2, both orders) on which an operand can be non-zero
static unsigned nz_mask(unsigned zmask) {
  unsigned nz = 0;
  for (int c1 = 0; c1 < 3; ++c1)
    for (int c2 = 0; c2 < 3; ++c2) {
      const int part = c1 >= c2 ? slot_of(c1, c2) : slot_of(c2, c1);
      if (!((zmask >> (P_HHHH + part)) & 1u)) nz |= 1u << (c1 * 3 + c2);
    }
  return nz;
}

// Leg masks of one term, per launch: byte cfix (0..2) holds bit
// kh * 4 + oh * 2 + th, set when a leg with fixed class cfix can add anything
// whose fixed state has kind kh, whose other state on the same side has kind
// oh and whose summed states have kind th (1 = hole); `sparse` is the one-body
// factor's sparsity, zstaged the zero-part mask of the staged operand.
static unsigned leg_masks(int sparse, unsigned zstaged) {
  const unsigned nz = nz_mask(zstaged);
  unsigned m = sparse ? LEG_SPARSE : 0u;
  for (int cfix = 0; cfix < 3; ++cfix)
    for (int bits = 0; bits < 8; ++bits)
      if (leg_ok(sparse, (bits >> 2) & 1, bits & 1, (bits >> 1) & 1, cfix, nz)) m |= 1u << (8 * cfix + bits);
  return m;
}

static int launch_bucket(qd_layout* L, const Plan122* p, const TaskSet* ts, const Bucket122& b, int threads,
                         const qd_op* A, const qd_op* B, int spA, int spB, double* C) {
  // the B term (FA x TB) and the A term (-FB x TA)
  const unsigned legB = leg_masks(spA, B->zero_mask), legA = leg_masks(spB, A->zero_mask);
#define QD_122_LAUNCH(TW, NT)                                                                                   \
  k_122_tile<TW, NT><<<b.count, NT, b.smem, L->stream>>>(L->dev, ts->d_task + b.first, p->d_tiles, p->d_gpd,   \
                                                         p->d_gpp, p->d_ftab, p->nfent, A->d,                   \
                                                         (double)A->herm, A->zero_mask, legA, B->d,             \
                                                         (double)B->herm, B->zero_mask, legB, C)
  if (b.tw == 2) {
    if (threads == 64) QD_122_LAUNCH(2, 64); else if (threads == 128) QD_122_LAUNCH(2, 128); else QD_122_LAUNCH(2, 256);
  } else {
    if (threads == 64) QD_122_LAUNCH(1, 64); else if (threads == 128) QD_122_LAUNCH(1, 128); else QD_122_LAUNCH(1, 256);
  }
#undef QD_122_LAUNCH
  ++L->nlaunch;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// The CTA size of each bucket of one bucketing (see tune_122).
static int tune_variant(qd_layout* L, Plan122* p, TaskSet* ts, const qd_op* A, const qd_op* B, int spA, int spB,
                        double* scratch, cudaEvent_t e0, cudaEvent_t e1) {
  ts->ms_total = 0.f;
  for (Bucket122& b : ts->buckets) {
    for (int v = 0; v < 3; ++v) {
      const int threads = 64 << v;
      float best = 1e30f;
      for (int rep = 0; rep < 2; ++rep) {
        QD_CUDA(cudaEventRecord(e0, L->stream));
        TRY(launch_bucket(L, p, ts, b, threads, A, B, spA, spB, scratch));
        QD_CUDA(cudaEventRecord(e1, L->stream));
        QD_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        QD_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        best = std::min(best, ms);
      }
      b.ms[v] = best;
    }
    int v = 0;
    for (int k = 1; k < 3; ++k)
      if (b.ms[k] < b.ms[v]) v = k;
    b.threads = 64 << v;
    ts->ms_total += b.ms[v];
  }
  return QD_OK;
}

// Autotuner: the first launch of a task set times, for every bucketing
// (kBounds), every bucket with 64-, 128- and 256-thread CTAs (CUDA events, best of
// two runs each) on the real operands, writing into a scratch operator of
// the layout; it keeps the CTA size per bucket and the bucketing with the
// least total time.  Every output cell is summed by one thread in a fixed
// order whatever the bucketing or CTA size, so the choice never changes a
// result.
static int tune_122(qd_layout* L, Plan122* p, TaskSet* ts, const qd_op* A, const qd_op* B, int spA, int spB) {
  double* scratch = scratch_operator(L);
  if (!scratch) return QD_OK;  // no scratch: keep the defaults
  cudaEvent_t e0, e1;
  QD_CUDA(cudaEventCreate(&e0));
  QD_CUDA(cudaEventCreate(&e1));
  const long long n0 = L->nlaunch;
  TRY(tune_variant(L, p, ts, A, B, spA, spB, scratch, e0, e1));
  for (TaskSet& alt : ts->alts) TRY(tune_variant(L, p, &alt, A, B, spA, spB, scratch, e0, e1));
  int best = -1;
  float tbest = ts->ms_total;
  for (size_t k = 0; k < ts->alts.size(); ++k)
    if (ts->alts[k].ms_total < tbest) {
      tbest = ts->alts[k].ms_total;
      best = (int)k;
    }
  // keep the winner in *ts; the others stay in alts for the report (their task arrays are freed)
  std::vector<TaskSet> others;
  TaskSet win;
  if (best >= 0) {
    win = ts->alts[best];
    ts->alts[best] = TaskSet();
    TaskSet cur = *ts;
    cur.alts.clear();
    others.push_back(cur);
  }
  for (TaskSet& t : ts->alts)
    if (t.d_task || !t.buckets.empty()) others.push_back(t);
  if (best >= 0) {
    *ts = win;
  }
  ts->alts.clear();
  for (TaskSet& t : others) {
    if (t.d_task) cudaFree(t.d_task);
    t.d_task = nullptr;
    ts->alts.push_back(t);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  L->nlaunch = n0;  // tuning launches are not the caller's work
  ts->tuned = true;
  return QD_OK;
}

// One bucket of k_122_full on stream st.
static int launch_full(qd_layout* L, const Plan122* p, const Plan122::FullBucket& b, int threads, const qd_op* A,
                       const qd_op* B, double* C, cudaStream_t st) {
#define QD_FULL_LAUNCH(NT, BOTH)                                                                                    \
  k_122_full<NT, BOTH><<<b.count, NT, b.smem, st>>>(L->dev, p->d_ftask + b.first, p->d_tiles, p->d_gpd, p->d_gpp, \
                                                           p->d_ftab, p->nfent, A->d, (double)A->herm, A->zero_mask, \
                                                           B->d, (double)B->herm, B->zero_mask, C)
  if (b.both) {
    if (threads == 64) QD_FULL_LAUNCH(64, true); else if (threads == 128) QD_FULL_LAUNCH(128, true); else QD_FULL_LAUNCH(256, true);
  } else {
    if (threads == 64) QD_FULL_LAUNCH(64, false); else if (threads == 128) QD_FULL_LAUNCH(128, false); else QD_FULL_LAUNCH(256, false);
  }
#undef QD_FULL_LAUNCH
  ++L->nlaunch;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// The CTA size of each bucket of k_122_full, once per layout: best of two
// runs on the real operands into a workspace operator (results do not depend
// on it).  The F tables of A and B are in place.
static int tune_full(qd_layout* L, Plan122* p, const qd_op* A, const qd_op* B) {
  double* scratch = scratch_operator(L);
  if (!scratch) return QD_OK;
  cudaEvent_t e0, e1;
  QD_CUDA(cudaEventCreate(&e0));
  QD_CUDA(cudaEventCreate(&e1));
  const long long n0 = L->nlaunch;
  const int nts[3] = {64, 128, 256};
  for (Plan122::FullBucket& b : p->fbuckets) {
    int best = 0;
    for (int k = 0; k < 3; ++k) {
      b.ms[k] = 1e30f;
      for (int rep = 0; rep < 2; ++rep) {
        QD_CUDA(cudaEventRecord(e0, L->stream));
        TRY(launch_full(L, p, b, nts[k], A, B, scratch, L->stream));
        QD_CUDA(cudaEventRecord(e1, L->stream));
        QD_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        QD_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        b.ms[k] = std::min(b.ms[k], ms);
      }
      if (b.ms[k] < b.ms[best]) best = k;
    }
    b.threads = nts[best];
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  L->nlaunch = n0;  // tuning launches are not the caller's work
  p->full_tuned = true;
  return QD_OK;
}

// Text summary of the autotuned buckets: k_122_full's, then every task set's.
std::string tuning_report_122(const qd_layout* L) {
  std::lock_guard<std::mutex> lock(g_plan_mutex);
  auto it = plans().find(L);
  if (it == plans().end()) return "";
  std::string out;
  char line[256];
  if (it->second.full_tuned) {
    float sum = 0.f;
    for (const auto& b : it->second.fbuckets) sum += std::min(b.ms[0], std::min(b.ms[1], b.ms[2]));
    snprintf(line, sizeof(line), "commutator_122, legs from registers: bucketing 0 kept (%.4f ms)\n", sum);
    out += line;
    for (const auto& b : it->second.fbuckets) {
      snprintf(line, sizeof(line), "  tiles %6d smem %6zu B: 64 thr %.4f ms, 128 thr %.4f ms, 256 thr %.4f ms -> %d\n",
               b.count, b.smem, b.ms[0], b.ms[1], b.ms[2], b.threads);
      out += line;
    }
  }
  for (const auto& kv : it->second.sets) {
    const TaskSet& ts = kv.second;
    snprintf(line, sizeof(line), "commutator_122 masks A=0x%03x B=0x%03x: bucketing %d kept (%.4f ms)",
             kv.first.first, kv.first.second, ts.bounds_id, ts.ms_total);
    out += line;
    for (const TaskSet& t : ts.alts) {
      snprintf(line, sizeof(line), ", bucketing %d %.4f ms", t.bounds_id, t.ms_total);
      out += line;
    }
    out += "\n";
    for (const Bucket122& b : kv.second.buckets) {
      snprintf(line, sizeof(line),
               "  tiles %6d staged %d smem %6zu B: 64 thr %.4f ms, 128 thr %.4f ms, 256 thr %.4f ms -> %d\n",
               b.count, b.tw, b.smem, b.ms[0], b.ms[1], b.ms[2], b.threads);
      out += line;
    }
  }
  return out;
}

static bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone;
}

static int spars(const qd_op* X) {
  const unsigned hp = (1u << P_FHH) | (1u << P_FPP);
  return (X->zero_mask & hp) == hp;
}

// Whether the tiles run through k_122_full: not where a one-body factor
// couples holes to particles only and the basis is large (k_122_tile then
// skips most of the legs and tiles), nor where a tile is too large for it.
constexpr i64 FULL_SPARSE_ENTRIES = 1000000;
static bool use_full(const qd_layout* L, const Plan122* p, const qd_op* A, const qd_op* B) {
  return p->full_fits && ((!spars(A) && !spars(B)) || L->neq < FULL_SPARSE_ENTRIES);
}

// Build (and autotune on A, B) the plan and the task set of a pair of
// zero-part masks ahead of a stream capture, which must neither allocate
// nor synchronise.  A and B may be views with the masks zA, zB.
int prepare_122(qd_layout* L, const qd_op* A, const qd_op* B) {
  Plan122* p;
  int rc = plan_122(L, &p);
  if (rc) return rc;
  if (gen_like(A->zero_mask)) return QD_OK;  // no tiles
  const bool tune = !L->prof.on && !capturing(L->stream);
  TaskSet* ts = nullptr;
  const bool full = use_full(L, p, A, B);
  if (!full && (rc = task_set(L, p, A->zero_mask, B->zero_mask, &ts))) return rc;
  if (tune && (full ? !p->full_tuned : !ts->tuned && !ts->buckets.empty())) {
    // the F tables of these operands first: the timed launches read them
    const int nf = L->m * p->gmax;
    k_ftab<<<(nf + 127) / 128, 128, 0, L->stream>>>(L->dev, p->d_sbase, A->d, (double)A->herm, B->d,
                                                    (double)B->herm, p->d_ftab, p->gmax, p->nfent);
    QD_CUDA(cudaGetLastError());
    if (full)
      TRY(tune_full(L, p, A, B));
    else
      TRY(tune_122(L, p, ts, A, B, spars(A), spars(B)));
  }
  return QD_OK;
}

// Every two-body part of C for a generator-like A, and with `ladder` the
// ladders of the blocks that gen_ladder_fused names: C_pppp on stream st, the
// other parts (which no kernel of C_pppp touches) on stream st2.
static int launch_122_gen(qd_layout* L, const Plan122* p, const qd_op* A, const qd_op* B, double* C, bool ladder,
                          cudaStream_t st, cudaStream_t st2, const HsUpdate* upd) {
  const bool lad = ladder && !((A->zero_mask >> P_PPHH) & 1u);  // every ladder left has the factor A_pphh
  const double hA = (double)A->herm, hB = (double)B->herm;
  GenTables G;
  G.gbase = p->d_gbase;
  G.rstart = p->d_rstart;
  G.cstart = p->d_cstart;
  G.rterm = p->d_rterm;
  G.cterm = p->d_cterm;
  for (int k = 0; k < 6; ++k) {
    G.rso[k] = p->gen_rso[k];
    G.cso[k] = p->gen_cso[k];
  }
  if (p->nsp_gen > 0) {
    k_122_gen<<<p->nsp_gen, SP_T, p->gen_bytes, st2>>>(L->dev, p->d_sptask + p->nsp_pppp, G, A->d, hA, B->d, hB,
                                                       lad && !((B->zero_mask >> P_PHHH) & 1u), C);
    ++L->nlaunch;
  }
  if (lad && p->nsp_ladder > 0) {
    k_gen_ladder<<<p->nsp_ladder, GL_T, 0, st2>>>(L->dev, p->d_ltask, A->d, hA, B->d, hB, B->zero_mask, C);
    ++L->nlaunch;
  }
  if (p->nsp_phph > 0) {
    k_gen_phph<<<p->nsp_phph, SP_T, p->phph_bytes, st2>>>(L->dev, p->d_sptask + p->nsp_pppp + p->nsp_gen, G, A->d, hA,
                                                          B->d, hB, C);
    ++L->nlaunch;
  }
  if (p->nsp_pppp > 0) {
    const int plad = lad && !((B->zero_mask >> P_PPHH) & 1u);
    if (upd)
      k_gen_pppp<true><<<p->nsp_pppp, GP_T, gp_smem(p->pppp_terms), st>>>(L->dev, p->d_sptask, p->d_ppbase, p->d_ppstart,
                                                                        p->d_ppterm, A->d, hA, B->d, hB, B->zero_mask,
                                                                        plad, C, *upd);
    else
      k_gen_pppp<false><<<p->nsp_pppp, GP_T, gp_smem(p->pppp_terms), st>>>(
          L->dev, p->d_sptask, p->d_ppbase, p->d_ppstart, p->d_ppterm, A->d, hA, B->d, hB, B->zero_mask, plad, C,
          HsUpdate{});
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

int gen_pppp_ctas(qd_layout* L, int* n) {
  Plan122* p;
  int rc = plan_122(L, &p);
  if (rc) return rc;
  *n = p->nsp_pppp;
  return QD_OK;
}

int launch_122(qd_layout* L, const qd_op* A, const qd_op* B, double* C, bool ladder, cudaStream_t st2,
               const HsUpdate* upd) {
  Plan122* p;
  int rc = plan_122(L, &p);
  if (rc) return rc;
  if (p->tiles.empty()) return QD_OK;
  if (gen_like(A->zero_mask)) return launch_122_gen(L, p, A, B, C, ladder, L->stream, st2 ? st2 : L->stream, upd);
  const int spA = spars(A), spB = spars(B);
  const bool full = use_full(L, p, A, B);
  TaskSet* ts = nullptr;
  if (!full && (rc = task_set(L, p, A->zero_mask, B->zero_mask, &ts))) return rc;
  const int nf = L->m * p->gmax;
  k_ftab<<<(nf + 127) / 128, 128, 0, L->stream>>>(L->dev, p->d_sbase, A->d, (double)A->herm, B->d,
                                                  (double)B->herm, p->d_ftab, p->gmax, p->nfent);
  ++L->nlaunch;
  if (full) {
    if (!p->full_tuned && !L->prof.on && !capturing(L->stream)) TRY(tune_full(L, p, A, B));
    // The buckets write different tiles: every other one on the second stream,
    // after the F tables.  One after the other they leave most of a small
    // basis's chip idle (two dense operators at N=6, R=10: 154 us in one
    // stream, 146 with two); where the tiles fill the chip the caller gives
    // no second stream.
    if (st2 && st2 != L->stream && p->fbuckets.size() > 1) {
      QD_CUDA(cudaEventRecord(L->ev_side[1], L->stream));
      QD_CUDA(cudaStreamWaitEvent(st2, L->ev_side[1], 0));
    } else {
      st2 = L->stream;
    }
    for (size_t k = 0; k < p->fbuckets.size(); ++k)
      TRY(launch_full(L, p, p->fbuckets[k], p->fbuckets[k].threads, A, B, C, k & 1 ? st2 : L->stream));
    return QD_OK;
  }
  if (!ts->tuned && !L->prof.on && !capturing(L->stream)) TRY(tune_122(L, p, ts, A, B, spA, spB));
  for (const Bucket122& b : ts->buckets) TRY(launch_bucket(L, p, ts, b, b.threads, A, B, spA, spB, C));
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

int prepare_pandya(qd_layout* L) {
  Plan122* p;
  return plan_122(L, &p);
}

int launch_pandya_tiles(qd_layout* L, const double* Z, double* C) {
  Plan122* p;
  int rc = plan_122(L, &p);
  if (rc) return rc;
  for (const PdBucket& b : p->pbuckets) {
    if (b.count == 0) continue;
#define QD_PD_LAUNCH(M, T)                                                                                  \
  k_pandya_tile<M, T><<<b.count, T, b.smem, L->stream>>>(L->dev, p->d_ptask + b.first, p->d_tiles, p->d_gpd, \
                                                         p->d_gpp, p->d_gpg, p->d_zrow, p->ng, Z, C)
    // small tiles: few cells a thread, so the fixed part of a CTA weighs less
    if (b.mode == PD_SINGLE)
      QD_PD_LAUNCH(PD_SINGLE, 256);
    else if (b.mode == PD_DIRECT)
      QD_PD_LAUNCH(PD_DIRECT, 256);
    else if (b.smem <= PD_SMALL)
      QD_PD_LAUNCH(PD_ALL, 64);
    else if (b.smem <= PD_MEDIUM)
      QD_PD_LAUNCH(PD_ALL, 128);
    else
      QD_PD_LAUNCH(PD_ALL, 256);
#undef QD_PD_LAUNCH
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

}  // namespace qd
