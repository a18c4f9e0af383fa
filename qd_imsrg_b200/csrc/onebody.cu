// onebody.cu -- E0 and the one-body part of a whole commutator [A, B] (110,
// 220, 111, 121 and 221 of src/commutators.f90:12-352) in two launches, for
// operators whose one-body parts conserve (m_l, m_s) (qd_op::zero_mask bit
// CONSERVES: known on the host, so the choice costs no synchronisation).
//
// For such operators only targets (x, y) of one (m_l, m_s) group g are
// non-zero (2,800 of 176,400 at N=20, R=20).  commutator_221 takes one form
// for all of them.  For a state u and x in g let alpha_x be the stored column
// A(pp, (u,x)) when u is a hole (Apphh or Appph by the type of x) and the
// stored row A((u,x), hh) when u is a particle (Apphh or Aphhh), with the
// ordering sign of the pair; beta_x the same of B.  With S_u(x,y) =
// alpha_x . beta_y the reference's trace is
//   hole u:      C(x,y) += hA S_u(x,y) - hB S_u(y,x)
//   particle u:  C(x,y) += hB S_u(x,y) - hA S_u(y,x)
// that is C(x,y) += hA R(x,y) - hB R(y,x), R = sum_holes S_u - sum_particles S_u^T.
//
// k_one_part sums R over one hole (or a few particles) u per CTA and writes
// it per (CTA, group cell); k_one_final adds them up in a fixed order and
// adds 111 and 121.  Bound: latency of L2 reads (a column is read once per
// (u, g) and used for all |g| partners; one CTA per target re-read both
// columns of every product from L2, about |g| times the traffic, and the
// pieces ran as eleven launches; the times of both stand at launch_onebody).
#include <algorithm>
#include <memory>
#include <vector>

#include "dev_common.cuh"

namespace qd {

namespace {

constexpr int OB_T = 128;        // threads per CTA
constexpr int OB_G = 16;         // most states of a group (the pair cells of commutator_122 have the same limit)
constexpr int OB_U = 8;          // particles u per CTA
constexpr int OB_PIECE = 2048;   // entries of A.B per CTA of the E0 dots
constexpr int OB_FILL = 4096;    // one-body entries per CTA of the zero fill

// Units of k_one_part, in launch order: particle and hole units {g, u0, nu
// (0: the hole u0), row of the partial array}, then E0 pieces, then one flag CTA.
struct OneTab {
  const int4* unit;
  int nunit;
  const longlong2* piece;  // {offset, entries}
  int npiece;
  const int* gslot;        // first cell of each group: cell (x, y) = gslot[g] + x |g| + y
  const int* ghole;        // holes of each group (its lowest members)
  int nslot;
  int nrow;                // rows of the partial array: one per hole, then one per OB_U particles
  const int4* target;      // {one-body entry, x | y << 16, group, kx | ky << 16}
  int ntarget;
  int q0;                  // cross-coupled block of (hole, particle) pairs of one group
};

// element k of the vector of operator `op` for the pair (u, x) of packed
// entry e: a column over pp pairs (u a hole) or a row over hh pairs
struct OneVec {
  const double* p;
  i64 ld;
};

__device__ __forceinline__ OneVec one_vec(const DevLayout& L, const double* __restrict__ op, int e, bool hole_u) {
  const int4 bd = __ldg(&L.blk[pt_blk(e)]);
  const i64* o = L.boff + 6 * pt_blk(e);
  const int c = pt_cls(e), i = pt_idx(e);
  OneVec v;
  if (hole_u) {  // x hole: Vpphh(:, i); x particle: Vppph(:, i)
    v.p = op + __ldg(o + (c == 0 ? 2 : 4)) + (i64)i * bd.z;
    v.ld = 1;
  } else {  // x particle: Vpphh(i, :); x hole: Vphhh(i, :)
    v.p = op + __ldg(o + (c == 2 ? 2 : 5)) + i;
    v.ld = c == 2 ? bd.z : bd.y;
  }
  return v;
}

// Range [lo, hi) of a group's members whose vectors can be non-zero.
__device__ __forceinline__ int2 one_range(unsigned z, bool hole_u, int n, int h) {
  const bool hok = !((z >> (hole_u ? P_PPHH : P_PHHH)) & 1u);  // x a hole
  const bool pok = !((z >> (hole_u ? P_PPPH : P_PPHH)) & 1u);  // x a particle
  return make_int2(hok ? 0 : h, pok ? n : h);
}

// v[16] of every lane summed over the warp; lane 2 i (and 2 i + 1) returns
// the sum of v[i] (16 shuffles of a double instead of 80)
__device__ __forceinline__ double warp_sum16(double* v, int lane) {
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

__global__ void __launch_bounds__(OB_T) k_one_part(DevLayout L, OneTab T, const double* __restrict__ A,
                                                   const double* __restrict__ B, unsigned zA, unsigned zB,
                                                   double* __restrict__ partial, double* __restrict__ epart,
                                                   int* __restrict__ flag) {
  __shared__ double red[OB_T / 32][OB_G * OB_G];
  __shared__ const double* vp[OB_T / 32][2][OB_G];
  __shared__ double vs[OB_T / 32][OB_G];
  __shared__ i64 vl[OB_T / 32][OB_G];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int b = blockIdx.x;
  if (b >= T.nunit) {
    b -= T.nunit;
    if (b < T.npiece) {  // 110 + 220: dot product of one piece of fph or Vpphh
      const longlong2 pc = T.piece[b];
      double s = 0.0;
      for (int i = tid; i < (int)pc.y; i += OB_T) s += A[pc.x + i] * B[pc.x + i];
      s = block_sum<OB_T>(s, red[0]);
      if (tid == 0) epart[b] = s;
      return;
    }
    // 121: whether a (hole, particle) entry of one group is non-zero in A or B
    const int base = __ldg(&L.cchp_base[T.q0]), nb = __ldg(&L.ccdim[T.q0]).y;
    int any = 0;
    for (int k = tid; k < nb; k += OB_T) {
      const int2 ia = __ldg(&L.cchp[base + k]);
      const i64 f = L.o_fph + (ia.y - L.n) + (i64)ia.x * L.mp;
      any |= A[f] != 0.0 || B[f] != 0.0;
    }
    any = __syncthreads_or(any);
    if (tid == 0) *flag = any;
    return;
  }
  const int4 un = T.unit[b];
  const int g = un.x, gs = __ldg(&L.gstart[g]), n = __ldg(&L.gstart[g + 1]) - gs, h = __ldg(&T.ghole[g]);
  const bool hole_u = un.z == 0;
  const int2 ra = one_range(zA, hole_u, n, h), rb = one_range(zB, hole_u, n, h);
  const int na = max(0, ra.y - ra.x), nb = max(0, rb.y - rb.x);
  double* out = partial + (i64)un.w * T.nslot + __ldg(&T.gslot[g]);
  for (int i = tid; i < n * n; i += OB_T)
#pragma unroll
    for (int k = 0; k < OB_T / 32; ++k) red[k][i] = 0.0;
  if (hole_u) {
    const int u = un.y;
    __shared__ int sK;
    if (tid == 0) sK = 0;
    __syncthreads();
    if (tid < n) {
      const int x = __ldg(&L.gmem[gs + tid]);
      vp[0][0][tid] = vp[0][1][tid] = nullptr;
      vs[0][tid] = 0.0;
      if (x != u) {
        const int e = __ldg(&L.ptab[u * L.m + x]);
        vp[0][0][tid] = one_vec(L, A, e, true).p;
        vp[0][1][tid] = one_vec(L, B, e, true).p;
        vs[0][tid] = pt_swap(e) ? -1.0 : 1.0;
        sK = __ldg(&L.blk[pt_blk(e)]).z;  // every pair (u, x in g) lies in one block
      }
    }
    __syncthreads();
    const int K = sK;
    for (int x0 = 0; x0 < na && K > 0; x0 += 4)
      for (int y0 = 0; y0 < nb; y0 += 4) {
        const double *pa[4], *pb[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          pa[i] = x0 + i < na ? vp[0][0][ra.x + x0 + i] : nullptr;
          pb[i] = y0 + i < nb ? vp[0][1][rb.x + y0 + i] : nullptr;
        }
        double acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.0;
#pragma unroll 2
        for (int k = tid; k < K; k += OB_T) {
          double a[4], c[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a[i] = pa[i] ? pa[i][k] : 0.0;
            c[i] = pb[i] ? pb[i][k] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[4 * i + j] += a[i] * c[j];
        }
        const double s = warp_sum16(acc, lane);
        const int x = ra.x + x0 + (lane >> 3), y = rb.x + y0 + ((lane >> 1) & 3);
        if (!(lane & 1) && x < ra.y && y < rb.y) red[w][x * n + y] = vs[0][x] * vs[0][y] * s;
      }
  } else {
    // one particle u per warp at a time; a lane owns the cells lane, lane + 32, ...
    constexpr int MAXC = OB_G * OB_G / 32;
    double acc[MAXC];
#pragma unroll
    for (int c = 0; c < MAXC; ++c) acc[c] = 0.0;
    const int cells = na * nb;
    for (int j = w; j < un.z; j += OB_T / 32) {
      const int u = un.y + j;
      int K = 0;
      __syncwarp();
      if (lane < n) {
        const int x = __ldg(&L.gmem[gs + lane]);
        vs[w][lane] = 0.0;
        if (x != u) {
          const int e = __ldg(&L.ptab[u * L.m + x]);
          const OneVec va = one_vec(L, A, e, false), vb = one_vec(L, B, e, false);
          vp[w][0][lane] = va.p;
          vp[w][1][lane] = vb.p;
          vl[w][lane] = va.ld;
          vs[w][lane] = pt_swap(e) ? -1.0 : 1.0;
          K = __ldg(&L.blk[pt_blk(e)]).x;
        }
      }
      __syncwarp();
      K = __reduce_max_sync(0xffffffffu, K);
      if (K == 0) continue;
#pragma unroll
      for (int c = 0; c < MAXC; ++c) {
        const int cell = lane + 32 * c;
        if (cell >= cells) continue;
        const int x = ra.x + cell / nb, y = rb.x + cell % nb;
        const double sg = vs[w][x] * vs[w][y];
        if (sg == 0.0) continue;  // x or y is u itself
        const double *p = vp[w][0][x], *r = vp[w][1][y];
        const i64 lp = vl[w][x], lr = vl[w][y];
        double s = 0.0;
#pragma unroll 4
        for (int k = 0; k < K; ++k) s += p[k * lp] * r[k * lr];
        acc[c] += sg * s;
      }
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < MAXC; ++c) {
      const int cell = lane + 32 * c;
      if (cell < cells) red[w][(rb.x + cell % nb) * n + ra.x + cell / nb] = -acc[c];  // R holds -S_u^T
    }
  }
  __syncthreads();
  for (int i = tid; i < n * n; i += OB_T) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < OB_T / 32; ++k) s += red[k][i];
    out[i] = s;
  }
}

// 111 for the target (x, y) of one group, the sums over that group's members
// (the others are exact zeros): the two products of state z.  zA, zB: a
// product with a part known to be zero is left out.
__device__ __forceinline__ double one_111(const DevLayout& L, const double* __restrict__ A, double hA,
                                          const double* __restrict__ B, double hB, unsigned zA, unsigned zB, int x,
                                          int y, int z) {
  const int n = L.n, mp = L.mp;
  const unsigned HH = 1u << P_FHH, PP = 1u << P_FPP, PH = 1u << P_FPH;
  auto fhh = [&](const double* f, int i, int j) { return f[L.o_fhh + i + (i64)j * n]; };
  auto fpp = [&](const double* f, int a, int b) { return f[L.o_fpp + (a - n) + (i64)(b - n) * mp]; };
  auto fph = [&](const double* f, int a, int i) { return f[L.o_fph + (a - n) + (i64)i * mp]; };
  const double sg = -hA * hB;
  if (x < n) {  // V + sg V^T, V = Afhh Bfhh - hB Bfph^T Afph
    if (z < n) return ((zA | zB) & HH) ? 0.0 : fhh(A, x, z) * fhh(B, z, y) + sg * (fhh(A, y, z) * fhh(B, z, x));
    return ((zA | zB) & PH) ? 0.0 : -hB * (fph(B, z, x) * fph(A, z, y) + sg * (fph(B, z, y) * fph(A, z, x)));
  }
  if (y >= n) {  // V + sg V^T, V = hB Afph Bfph^T - Bfpp Afpp
    if (z < n) return ((zA | zB) & PH) ? 0.0 : hB * (fph(A, x, z) * fph(B, y, z) + sg * (fph(A, y, z) * fph(B, x, z)));
    return ((zA | zB) & PP) ? 0.0 : -(fpp(B, x, z) * fpp(A, z, y) + sg * (fpp(B, y, z) * fpp(A, z, x)));
  }
  double s = 0.0;
  if (z < n) {
    if (!((zA & PH) | (zB & HH))) s += fph(A, x, z) * fhh(B, z, y);
    if (!((zB & PH) | (zA & HH))) s -= fph(B, x, z) * fhh(A, z, y);
  } else {
    if (!((zA & PP) | (zB & PH))) s += fpp(A, x, z) * fph(B, z, y);
    if (!((zB & PP) | (zA & PH))) s -= fpp(B, x, z) * fph(A, z, y);
  }
  return s;
}

// Stored part (as a P_* bit) with pairs of classes hi >= lo.
__device__ __forceinline__ unsigned one_part_bit(int c1, int c2) {
  const int hi = max(c1, c2), lo = min(c1, c2);
  return 1u << (hi == 0 ? P_HHHH : (hi == 1 ? (lo == 0 ? P_PHHH : P_PHPH)
                                            : (lo == 0 ? P_PPHH : (lo == 1 ? P_PPPH : P_PPPP))));
}

// One warp per target of one group; the CTAs after them write the other
// one-body entries (zero) and, the last one, E0.
__global__ void __launch_bounds__(OB_T) k_one_final(DevLayout L, OneTab T, const double* __restrict__ A, double hA,
                                                    const double* __restrict__ B, double hB, unsigned zA, unsigned zB,
                                                    const double* __restrict__ partial,
                                                    const double* __restrict__ epart, const int* __restrict__ flag,
                                                    double* __restrict__ C) {
  constexpr int W = OB_T / 32;
  const int tid = threadIdx.x, lane = tid & 31;
  const int ntc = (T.ntarget + W - 1) / W;
  const int n = L.n, mp = L.mp;
  if ((int)blockIdx.x >= ntc) {
    const int b = blockIdx.x - ntc;
    const i64 n1 = (i64)n * n + (i64)mp * mp + (i64)mp * n;
    if ((i64)b * OB_FILL < n1) {
      const i64 e1 = min(n1, (i64)(b + 1) * OB_FILL);
      for (i64 t = (i64)b * OB_FILL + tid; t < e1; t += OB_T) {
        int x, y;
        if (t < (i64)n * n) {
          x = (int)t % n;
          y = (int)t / n;
        } else {
          int r = (int)(t - (i64)n * n);
          const bool pp = r < mp * mp;
          if (!pp) r -= mp * mp;
          x = n + r % mp;
          y = r / mp + (pp ? n : 0);
        }
        if (__ldg(&L.gid[x]) != __ldg(&L.gid[y])) C[L.o_fhh + t] = 0.0;
      }
      return;
    }
    __shared__ double red[W];
    double s = 0.0;
    for (int i = tid; i < T.npiece; i += OB_T) s += epart[i];
    s = block_sum<OB_T>(s, red);
    if (tid == 0) C[0] = (hA - hB) * s;
    return;
  }
  const int it = blockIdx.x * W + (tid >> 5);
  if (it >= T.ntarget) return;
  const int4 tg = __ldg(&T.target[it]);
  const int x = tg.y & 0xFFFF, y = tg.y >> 16, g = tg.z, kx = tg.w & 0xFFFF, ky = tg.w >> 16;
  const int gs = __ldg(&L.gstart[g]), ng = __ldg(&L.gstart[g + 1]) - gs;
  double s = 0.0;
  // 221: R(x,y) and R(y,x) over the partial rows
  {
    const i64 sl = __ldg(&T.gslot[g]);
    const i64 xy = sl + kx * ng + ky, yx = sl + ky * ng + kx;
    for (int c = lane; c < T.nrow; c += 32)
      s += hA * partial[c * (i64)T.nslot + xy] - hB * partial[c * (i64)T.nslot + yx];
  }
  // 121 (src/commutators.f90:73-134) over the (hole, particle) pairs of one group
  if (*flag) {
    const bool px = x >= n, py = y >= n;
    const unsigned part1 = one_part_bit(px ? 2 : 1, py ? 1 : 0), part2 = one_part_bit(px ? 1 : 0, py ? 2 : 1);
    const bool b1 = !(zB & part1), a1 = !(zA & part1), b2 = !(zB & part2), a2 = !(zA & part2);
    const int base = __ldg(&L.cchp_base[T.q0]), nb = __ldg(&L.ccdim[T.q0]).y;
    for (int k = lane; k < nb; k += 32) {
      const int2 ia = __ldg(&L.cchp[base + k]);
      const int i = ia.x, a = ia.y;
      const i64 f = L.o_fph + (a - n) + (i64)i * mp;
      const double fa = A[f], fb = B[f];
      const PairPos p1 = dv_pos(L, __ldg(&L.ptab[a * L.m + x]), __ldg(&L.ptab[i * L.m + y]));  // <a x|i y>
      const PairPos p2 = dv_pos(L, __ldg(&L.ptab[i * L.m + x]), __ldg(&L.ptab[a * L.m + y]));  // <i x|a y>
      const double t1 = b1 ? fa * hA * dv_at(p1, B, hB) : 0.0;
      const double t2 = a1 ? fb * hB * dv_at(p1, A, hA) : 0.0;
      const double t3 = b2 ? -fa * dv_at(p2, B, hB) : 0.0;
      const double t4 = a2 ? fb * dv_at(p2, A, hA) : 0.0;
      s += (t1 - t2) + (t3 + t4);
    }
  }
  if (lane < ng) s += one_111(L, A, hA, B, hB, zA, zB, x, y, __ldg(&L.gmem[gs + lane]));
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) C[L.o_fhh + tg.x] = s;
}

}  // namespace

// Tables and buffers of one layout, built on first use.
struct OneBody {
  OneTab tab{};
  double* d_partial = nullptr;
  double* d_epart = nullptr;
  int* d_flag = nullptr;
  int grid1 = 0, grid2 = 0;
  bool usable = true;  // every group fits the kernel's cells
};

void onebody_free(qd_layout* L) {
  delete L->onebody;
  L->onebody = nullptr;
}

static int onebody_plan(qd_layout* L) {
  if (L->onebody) return QD_OK;
  std::unique_ptr<OneBody> p(new OneBody());  // the layout's when complete: a failure leaves no plan
  const int m = L->m, n = L->n, mp = L->mp, ng = (int)L->gstart.size() - 1;
  std::vector<int> gslot(ng + 1, 0), ghole(ng, 0), kpos(m, 0);
  for (int g = 0; g < ng; ++g) {
    const int sz = L->gstart[g + 1] - L->gstart[g];
    if (sz > OB_G) p->usable = false;
    gslot[g + 1] = gslot[g] + sz * sz;
    for (int k = 0; k < sz; ++k) {
      const int s = L->gmem[L->gstart[g] + k];
      kpos[s] = k;
      if (s < n) {
        if (k != ghole[g]) p->usable = false;  // holes are not the group's lowest members
        ++ghole[g];
      }
    }
  }
  if (m > 0x7FFF || m == 0) p->usable = false;
  if (!p->usable) {
    L->onebody = p.release();
    return QD_OK;
  }
  // hole units first: they are the longer ones
  std::vector<int4> unit;
  const int npu = (mp + OB_U - 1) / OB_U;
  for (int u = 0; u < n; ++u)
    for (int g = 0; g < ng; ++g) unit.push_back(int4{g, u, 0, u});
  for (int c = 0; c < npu; ++c)
    for (int g = 0; g < ng; ++g) unit.push_back(int4{g, n + c * OB_U, std::min(OB_U, mp - c * OB_U), n + c});
  const int nrow = n + npu;
  std::vector<longlong2> piece;
  auto add = [&](i64 o, i64 len) {
    for (i64 k = 0; k < len; k += OB_PIECE) piece.push_back(longlong2{o + k, std::min<i64>(OB_PIECE, len - k)});
  };
  add(L->o_fph, (i64)mp * n);
  for (int q = 0; q < L->nblock; ++q) add(L->boff[6 * q + 2], (i64)L->blk[q].x * L->blk[q].z);
  std::vector<int4> target;
  const i64 nhh = (i64)n * n, npp = (i64)mp * mp;
  for (i64 t = 0; t < nhh + npp + (i64)mp * n; ++t) {
    int x, y;
    if (t < nhh) {
      x = (int)(t % n);
      y = (int)(t / n);
    } else if (t < nhh + npp) {
      x = n + (int)((t - nhh) % mp);
      y = n + (int)((t - nhh) / mp);
    } else {
      x = n + (int)((t - nhh - npp) % mp);
      y = (int)((t - nhh - npp) / mp);
    }
    if (L->gid[x] == L->gid[y]) target.push_back(int4{(int)t, x | (y << 16), L->gid[x], kpos[x] | (kpos[y] << 16)});
  }
  OneTab& T = p->tab;
  T.nunit = (int)unit.size();
  T.npiece = (int)piece.size();
  T.ntarget = (int)target.size();
  T.nslot = gslot[ng];
  T.nrow = nrow;
  T.q0 = L->ccmap[0].x;  // (0, 0): no transfer
  const i64 n1 = nhh + npp + (i64)mp * n;
  p->grid1 = T.nunit + T.npiece + 1;
  p->grid2 = (T.ntarget + OB_T / 32 - 1) / (OB_T / 32) + (int)((n1 + OB_FILL - 1) / OB_FILL) + 1;
  PlanMemory mem;
  mem.add(unit, &T.unit);
  mem.add(piece, &T.piece);
  mem.add(gslot, &T.gslot);
  mem.add(ghole, &T.ghole);
  mem.add(target, &T.target);
  // k_one_part writes every partial sum, dot and the flag before k_one_final reads them
  mem.room((i64)nrow * T.nslot, &p->d_partial);
  mem.room(T.npiece, &p->d_epart);
  mem.room(1, &p->d_flag);
  const int rc = mem.commit(L);
  if (!rc) L->onebody = p.release();
  return rc;
}

// Tables and buffers of the layout for onebody (ahead of a stream capture,
// which must not allocate).
int prepare_onebody(qd_layout* L) { return onebody_plan(L); }

// E0 and the one-body part of C = [A, B]; *done = false (and nothing
// launched) when A or B may couple different (m_l, m_s), or a group is too
// large: the caller then runs the pieces one by one.  Measured on the whole
// stage (CUDA events), piece by piece and fused: [Omega, X] at N=20, R=20
// 403 and 68 us, at N=6, R=10 90 and 19 us; two dense operators at N=20, R=20
// 593 and 123 us.
int launch_onebody(qd_layout* L, const qd_op* A, const qd_op* B, double* C, bool* done) {
  *done = false;
  if (!(A->zero_mask & B->zero_mask & CONSERVES)) return QD_OK;
  int rc = onebody_plan(L);
  if (rc) return rc;
  const OneBody* p = L->onebody;
  if (!p->usable) return QD_OK;
  k_one_part<<<p->grid1, OB_T, 0, L->stream>>>(L->dev, p->tab, A->d, B->d, A->zero_mask, B->zero_mask, p->d_partial,
                                               p->d_epart, p->d_flag);
  k_one_final<<<p->grid2, OB_T, 0, L->stream>>>(L->dev, p->tab, A->d, (double)A->herm, B->d, (double)B->herm,
                                                A->zero_mask, B->zero_mask, p->d_partial, p->d_epart, p->d_flag, C);
  L->nlaunch += 2;
  QD_CUDA(cudaGetLastError());
  *done = true;
  return QD_OK;
}

}  // namespace qd
