// kernels_alg.cu -- bandwidth-bound kernels of the commutator engine:
// axpy (add_arrays), deterministic FP64 reductions (commutator_110/220 traces,
// mat_2_norm, MBPT2, HF_E2), the White generator, the BCH term's update with
// its norms and exit test, and the Pandya transform of an operator (calc_cc).
#include <algorithm>
#include <vector>

#include "dev_common.cuh"

namespace qd {

// BCH_EXPAND's truncated coefficients cof(1..11) (magnus_IMSRG.f90:265-267),
// for terms whose coefficient is picked on the device (whole BCH step in one
// graph): term k (0-based) adds cof[k] * INT2.
__constant__ double c_bch_cof[11] = QD_BCH_COF;

// ---------------------------------------------------------------------------
// add_arrays (src/ME_general.f90:592-618): c = sa*a + sb*b over the whole
// vectorize array (E0 included).  double2-vectorised when all three pointers
// share 16-byte alignment.  Products and sum are rounded separately (no FMA
// contraction), as in the reference's build, so the result is bit-identical.
// ---------------------------------------------------------------------------
__global__ void k_axpy(const double* __restrict__ a, double sa, const double* __restrict__ b, double sb,
                       double* __restrict__ c, i64 n) {
  i64 stride = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    c[i] = __dadd_rn(__dmul_rn(sa, a[i]), __dmul_rn(sb, b[i]));
}
__global__ void k_axpy2(const double2* __restrict__ a, double sa, const double2* __restrict__ b, double sb,
                        double2* __restrict__ c, i64 n2) {
  i64 stride = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += stride) {
    double2 x = a[i], y = b[i];
    c[i] = make_double2(__dadd_rn(__dmul_rn(sa, x.x), __dmul_rn(sb, y.x)),
                       __dadd_rn(__dmul_rn(sa, x.y), __dmul_rn(sb, y.y)));
  }
}

// zero every entry of op outside the parts in `keep` (bit P_* per part, bit
// P_COUNT for E0)
__global__ void k_keep_parts(DevLayout L, double* __restrict__ op, unsigned keep) {
  const i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= L.neq) return;
  int part;
  if (e < L.o_fhh)
    part = P_COUNT;
  else if (e < L.o_fpp)
    part = P_FHH;
  else if (e < L.o_fph)
    part = P_FPP;
  else if (e < L.o2)
    part = P_FPH;
  else
    part = P_HHHH + (__ldg(L.s2id + find_seg(L.s2off, L.ns2, e)) & 7);
  if (!((keep >> part) & 1u)) op[e] = 0.0;
}

int launch_keep_parts(qd_layout* L, double* op, unsigned keep) {
  if (L->neq > 0) k_keep_parts<<<(unsigned)((L->neq + 255) / 256), 256, 0, L->stream>>>(L->dev, op, keep);
  ++L->nlaunch;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

__global__ void __launch_bounds__(256) k_axpy_gen(DevLayout L, const double* a, double sa, const double* b, double sb,
                                                  double* c) {
  const i64 n1 = (i64)L.mp * L.n, n = 1 + n1 + L.pcnt[P_PPHH - P_HHHH];
  const i64 stride = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    i64 pos = i == 0 ? 0 : L.o_fph + i - 1;
    if (i > n1) {
      int q, row, col;
      part_elem(L, P_PPHH - P_HHHH, i - 1 - n1, q, pos, row, col);
    }
    c[pos] = __dadd_rn(__dmul_rn(sa, a[pos]), __dmul_rn(sb, b[pos]));
  }
}

int launch_axpy_gen(qd_layout* L, const double* a, double sa, const double* b, double sb, double* c) {
  const i64 n = 1 + (i64)L->mp * L->n + L->dev.pcnt[P_PPHH - P_HHHH];
  k_axpy_gen<<<(unsigned)std::min<i64>(148 * 8, (n + 255) / 256), 256, 0, L->stream>>>(L->dev, a, sa, b, sb, c);
  ++L->nlaunch;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

int launch_axpy(qd_layout* L, const double* a, double sa, const double* b, double sb, double* c, i64 n) {
  const int threads = 256, blocks = 148 * 8;
  if ((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0) {
    k_axpy2<<<blocks, threads, 0, L->stream>>>((const double2*)a, sa, (const double2*)b, sb, (double2*)c, n / 2);
    ++L->nlaunch;
    if (n & 1) {
      k_axpy<<<1, 32, 0, L->stream>>>(a + n - 1, sa, b + n - 1, sb, c + n - 1, 1);
      ++L->nlaunch;
    }
  } else {
    k_axpy<<<blocks, threads, 0, L->stream>>>(a, sa, b, sb, c, n);
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// ---------------------------------------------------------------------------
// Deterministic two-stage reductions.  Stage 1: RED_BLOCKS CTAs, fixed
// element->thread assignment, fixed tree -> partial[b].  Stage 2: one CTA sums
// the partials in a fixed order and writes scale*sum (+ add*out) to *out.
// ---------------------------------------------------------------------------
struct RedDotRange {  // sum a[i]*b[i] (or a[i]^2) over [o, o+n)
  const double* a;
  const double* b;
  i64 o;
  __device__ double operator()(i64 i) const {
    double x = a[o + i];
    return x * (b ? b[o + i] : x);
  }
};

struct RedDotPart {  // sum over all entries of one two-body part: a*b (or a^2)
  DevLayout L;
  const double* a;
  const double* b;
  int p;
  __device__ double operator()(i64 e) const {
    int q, row, col;
    i64 pos;
    part_elem(L, p, e, q, pos, row, col);
    double x = a[pos];
    return x * (b ? b[pos] : x);
  }
};

// MBPT2 (src/HFQDmod.f90:325-362): Vpphh^2 / (fhh(h1,h1)+fhh(h2,h2)-(fpp(p1,p1)+fpp(p2,p2)))
struct RedMBPT2 {
  DevLayout L;
  const double* h;
  __device__ double operator()(i64 e) const {
    int q, row, col;
    i64 pos;
    part_elem(L, P_PPHH - P_HHHH, e, q, pos, row, col);
    int2 pp = block_pair(L, q, 2, row), hh = block_pair(L, q, 0, col);
    const int n = L.n, mp = L.mp;
    double f12 = h[L.o_fpp + (pp.x - n) + (i64)(pp.x - n) * mp] + h[L.o_fpp + (pp.y - n) + (i64)(pp.y - n) * mp];
    double denom = h[L.o_fhh + hh.x + (i64)hh.x * n] + h[L.o_fhh + hh.y + (i64)hh.y * n] - f12;
    double x = h[pos];
    return x * x / denom;
  }
};

struct RedGenSquares {  // squares of fph, then of Vpphh
  DevLayout L;
  const double* a;
  i64 n1;
  __device__ double operator()(i64 e) const {
    i64 pos = L.o_fph + e;
    if (e >= n1) {
      int q, row, col;
      part_elem(L, P_PPHH - P_HHHH, e - n1, q, pos, row, col);
    }
    return a[pos] * a[pos];
  }
};

// HF_E2 trace: sum over blocks of Vhhhh(j,j)
struct RedHHTrace {
  DevLayout L;
  const double* h;
  __device__ double operator()(i64 e) const {
    int q, row, col;
    i64 pos;
    part_elem(L, P_HHHH - P_HHHH, e, q, pos, row, col);
    return row == col ? h[pos] : 0.0;
  }
};

template <class F>
__global__ void __launch_bounds__(RED_THREADS) k_reduce(F f, i64 n, double* __restrict__ partial) {
  __shared__ double sh[RED_THREADS / 32];
  double s = 0.0;
  i64 stride = (i64)gridDim.x * blockDim.x;
  for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) s += f(i);
  s = block_sum<RED_THREADS>(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// out = scale * sum(partial) + add * (*out), or its square root
__global__ void k_reduce_final(const double* __restrict__ partial, int np, double scale, double add, bool root,
                               double* __restrict__ out) {
  __shared__ double sh[RED_THREADS / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) s += partial[i];
  s = block_sum<RED_THREADS>(s, sh);
  if (threadIdx.x == 0) {
    const double v = scale * s + (add != 0.0 ? add * (*out) : 0.0);
    *out = root ? sqrt(v) : v;
  }
}

int ensure_reduction(qd_layout* L) {
  if (!L->d_red) {
    QD_CUDA(cudaMalloc(&L->d_red, sizeof(double) * (RED_BLOCKS + 64)));
    L->ws_bytes += sizeof(double) * (RED_BLOCKS + 64);
  }
  if (!L->h_red) QD_CUDA(cudaMallocHost(&L->h_red, sizeof(double) * 64));
  return QD_OK;
}

template <class F>
static int reduce_to(qd_layout* L, const F& f, i64 n, double scale, double add, double* dout, bool root = false) {
  int rc = ensure_reduction(L);
  if (rc) return rc;
  if (n > 0) {
    const int blocks = (int)std::min<i64>(RED_BLOCKS, (n + RED_THREADS - 1) / RED_THREADS);
    k_reduce<F><<<blocks, RED_THREADS, 0, L->stream>>>(f, n, L->d_red);
    k_reduce_final<<<1, RED_THREADS, 0, L->stream>>>(L->d_red, blocks, scale, add, root, dout);
    L->nlaunch += 2;
  } else {
    k_reduce_final<<<1, RED_THREADS, 0, L->stream>>>(L->d_red, 0, scale, add, root, dout);
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// Device scalar slots in d_red beyond the partials
double* red_slot(qd_layout* L, int k) { return L->d_red + RED_BLOCKS + k; }

int reduce_dot_range(qd_layout* L, const double* a, const double* b, i64 o, i64 n, double scale, double add,
                     double* dout) {
  return reduce_to(L, RedDotRange{a, b, o}, n, scale, add, dout);
}
int reduce_dot_part(qd_layout* L, const double* a, const double* b, int part, double scale, double add, double* dout) {
  int p = part - P_HHHH;
  return reduce_to(L, RedDotPart{L->dev, a, b, p}, L->dev.pcnt[p], scale, add, dout);
}
int reduce_mbpt2(qd_layout* L, const double* h, double* dout) {
  return reduce_to(L, RedMBPT2{L->dev, h}, L->dev.pcnt[P_PPHH - P_HHHH], 1.0, 0.0, dout);
}
int reduce_hhtrace(qd_layout* L, const double* h, double* dout) {
  return reduce_to(L, RedHHTrace{L->dev, h}, L->dev.pcnt[0], 1.0, 0.0, dout);
}
// mat_2_norm (src/ME_general.f90:2112-2138): sqrt of the sum of squares of
// every stored one- and two-body entry (E0 excluded), sqrt on the device.
// The entries are summed in vectorize order by the fixed two-stage tree; the
// reference's order (fph, fpp, fhh, then per block hhhh, pppp, pphh, phph,
// phhh, ppph) differs only in rounding.
int reduce_norm(qd_layout* L, const double* a, unsigned zmask, double* dout) {
  if (gen_like(zmask))  // a generator: its other parts add exact zeros
    return reduce_to(L, RedGenSquares{L->dev, a, (i64)L->mp * L->n}, (i64)L->mp * L->n + L->dev.pcnt[P_PPHH - P_HHHH],
                     1.0, 0.0, dout, true);
  return reduce_to(L, RedDotRange{a, nullptr, L->o_fhh}, L->neq - L->o_fhh, 1.0, 0.0, dout, true);
}

// ---------------------------------------------------------------------------
// One BCH_EXPAND term update in one pass (magnus_IMSRG.f90:298-316):
//   c = sa*a + sb*b  (add_arrays, bit-identical: no FMA contraction)
// together with mat_2_norm of both inputs, |a| = |INT1| (HS before the
// update) and |b| = |INT2|, over every stored entry but E0.  Fixed grid and
// fixed element -> thread assignment: deterministic.  Partial sums: 2 per
// CTA (a, b).
// ---------------------------------------------------------------------------
constexpr int AXN_BLOCKS = 4 * 148, AXN_THREADS = 256;


// The last CTA of an update to finish adds the np pairs of partial sums in a
// fixed order, writes out[0] = |a|, out[1] = |b| and, inside a step graph,
// BCH_EXPAND's exit test (magnus_IMSRG.f90:316): after the term whose
// coefficient index is *kidx, continue while |INT2| cof / |INT1| >= conv and
// fewer than 11 terms ran; the answer sets the graph's loop condition (and,
// for the first term of a two-term loop body, the condition of the second),
// and *kidx advances by one, without the two more launches that a final sum
// and the test would be.  Every CTA calls this after
// its partial sums are written; count returns to zero for the next launch.
__device__ __forceinline__ void axn_finish(const double2* partial, int np, unsigned* count, double* out, int* kidx,
                                           const BchDecide& D) {
  __shared__ double sh[AXN_THREADS / 32];
  __shared__ bool last;
  __threadfence();
  if (threadIdx.x == 0) last = atomicAdd(count, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0, b = 0.0;
#pragma unroll 8
  for (int i = threadIdx.x; i < np; i += AXN_THREADS) {
    const double2 v = __ldcg(partial + i);
    a += v.x;
    b += v.y;
  }
  a = block_sum<AXN_THREADS>(a, sh);
  b = block_sum<AXN_THREADS>(b, sh);
  if (threadIdx.x != 0) return;
  *count = 0;
  const double n1 = sqrt(a), n2 = sqrt(b);
  out[0] = n1;
  out[1] = n2;
  if (!D.on) return;
  const int k = *kidx;
  const bool stop = n2 * c_bch_cof[k] / n1 < D.conv;  // NaN continues, as the host test does
  const unsigned go = (!stop && k + 1 < 11) ? 1u : 0u;
  *kidx = k + 1;
  cudaGraphSetConditional(D.hloop, go);
  if (D.set_next) cudaGraphSetConditional(D.hnext, go);
}

// 16-byte accesses: the arrays are 16-byte aligned (cudaMalloc) and walked
// as pairs of entries; entry 0 (E0) is left out of the norms, an odd last
// entry is handled by thread 0.
__global__ void __launch_bounds__(AXN_THREADS) k_axpy_norms(const double* a, double sa,
                                                            const double* __restrict__ b, double sb,
                                                            double* c, i64 n, i64 o1, double2* partial,
                                                            int* kidx, unsigned* count, double* out, BchDecide D) {
  __shared__ double sh[AXN_THREADS / 32];
  if (kidx) sb = c_bch_cof[*kidx];  // coefficient of the term the device counter names
  double an = 0.0, bn = 0.0;
  const i64 stride = (i64)gridDim.x * blockDim.x;
  const i64 n2 = n >> 1;
  const double2* a2 = reinterpret_cast<const double2*>(a);
  const double2* b2 = reinterpret_cast<const double2*>(b);
  double2* c2 = reinterpret_cast<double2*>(c);
  for (i64 j = (i64)blockIdx.x * blockDim.x + threadIdx.x; j < n2; j += stride) {
    const double2 x = a2[j], y = b2[j];
    c2[j] = make_double2(__dadd_rn(__dmul_rn(sa, x.x), __dmul_rn(sb, y.x)),
                         __dadd_rn(__dmul_rn(sa, x.y), __dmul_rn(sb, y.y)));
    if (2 * j >= o1) {
      an += x.x * x.x;
      bn += y.x * y.x;
    }
    if (2 * j + 1 >= o1) {
      an += x.y * x.y;
      bn += y.y * y.y;
    }
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    const double x = a[n - 1], y = b[n - 1];
    c[n - 1] = __dadd_rn(__dmul_rn(sa, x), __dmul_rn(sb, y));
    if (n - 1 >= o1) {
      an += x * x;
      bn += y * y;
    }
  }
  an = block_sum<AXN_THREADS>(an, sh);
  bn = block_sum<AXN_THREADS>(bn, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(an, bn);
  axn_finish(partial, gridDim.x, count, out, kidx, D);
}

// {sums of one-pass updates | their CTA counter}
static int ensure_axn(qd_layout* L) {
  if (L->d_axn) return QD_OK;
  const size_t bytes = sizeof(double2) * (AXN_BLOCKS + 1);
  double* p = nullptr;
  QD_CUDA(cudaMalloc(&p, bytes));
  const cudaError_t e = cudaMemsetAsync(p, 0, bytes, L->stream);
  if (e != cudaSuccess) {  // the counter has to be zero before the first update
    cudaFree(p);
    return cuda_fail(e, "cudaMemsetAsync(update sums)");
  }
  L->d_axn = p;
  L->ws_bytes += (i64)bytes;
  return QD_OK;
}
static unsigned* axn_count(qd_layout* L) { return reinterpret_cast<unsigned*>(L->d_axn + 2 * AXN_BLOCKS); }

int launch_axpy_norms(qd_layout* L, const double* a, double sa, const double* b, double sb, double* c,
                      double* dout2, int* kidx, const BchDecide& D) {
  int rc = ensure_axn(L);
  if (rc) return rc;
  if ((((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) != 0) {
    set_error("launch_axpy_norms: operator arrays must be 16-byte aligned");
    return QD_ERR_ARG;
  }
  // a CTA per two rounds of its threads at least: small bases need few
  const int blocks = (int)std::max<i64>(1, std::min<i64>(AXN_BLOCKS, L->neq / (4 * AXN_THREADS)));
  k_axpy_norms<<<blocks, AXN_THREADS, 0, L->stream>>>(a, sa, b, sb, c, L->neq, L->o_fhh, (double2*)L->d_axn, kidx,
                                                      axn_count(L), dout2, D);
  ++L->nlaunch;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// The update outside Vpppp, whose entries k_gen_pppp updates where it makes
// them (reading C_pppp back costs as much as writing it): one CTA per piece
// of at most AXR_PIECE entries.  Bound: HBM, 24 bytes an entry.  At N=20,
// R=20 the one-pass update of all 61.9 M entries takes 230 us; Vpppp is 88%
// of them.
constexpr int AXR_PIECE = 4096;
__global__ void __launch_bounds__(AXN_THREADS) k_axpy_norms_rest(const longlong2* __restrict__ piece,
                                                                 const double* src, double* hs,
                                                                 const double* __restrict__ b, double sb, int* kidx, i64 o1, double2* partial,
                                                                 int first, unsigned* count, double* out,
                                                                 BchDecide D) {
  __shared__ double sh[AXN_THREADS / 32];
  if (kidx) sb = c_bch_cof[*kidx];
  const longlong2 p = piece[blockIdx.x];
  double an = 0.0, bn = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < (int)p.y; i += AXN_THREADS) {
    const i64 e = p.x + i;
    const double x = src[e], y = b[e];
    hs[e] = __dadd_rn(x, __dmul_rn(sb, y));
    if (e >= o1) {
      an += x * x;
      bn += y * y;
    }
  }
  an = block_sum<AXN_THREADS>(an, sh);
  bn = block_sum<AXN_THREADS>(bn, sh);
  if (threadIdx.x == 0) partial[first + blockIdx.x] = make_double2(an, bn);
  axn_finish(partial, first + gridDim.x, count, out, kidx, D);  // the first sums are k_gen_pppp's
}

int prepare_hs_update(qd_layout* L) {
  int rc = ensure_axn(L);
  if (rc || L->d_axp) return rc;
  if ((rc = gen_pppp_ctas(L, &L->naxp))) return rc;
  std::vector<longlong2> v;
  auto add = [&](i64 o, i64 e) {
    for (; o < e; o += AXR_PIECE) v.push_back(longlong2{o, std::min<i64>(AXR_PIECE, e - o)});
  };
  i64 o = 0;
  for (int q = 0; q < L->nblock; ++q) {
    add(o, L->boff[6 * q + 1]);
    o = L->boff[6 * q + 2];
  }
  add(o, L->neq);
  PlanMemory mem;
  mem.add(v, &L->d_axrest);
  mem.room(2 * (i64)(L->naxp + (int)v.size()), &L->d_axp);
  L->naxrest = (int)v.size();
  return mem.commit(L);
}

int hs_update_begin(qd_layout* L, const double* src, double* HS, double cof, int* kidx, HsUpdate* upd) {
  int rc = prepare_hs_update(L);
  if (rc) return rc;
  upd->src = src;
  upd->HS = HS;
  upd->cof = cof;
  upd->kidx = kidx;
  upd->partial = L->d_axp;
  return QD_OK;
}

int launch_axpy_norms_rest(qd_layout* L, const double* b, const HsUpdate& u, double* dout2, const BchDecide& D) {
  k_axpy_norms_rest<<<L->naxrest, AXN_THREADS, 0, L->stream>>>(L->d_axrest, u.src, u.HS, b, u.cof, u.kidx, L->o_fhh,
                                                               (double2*)u.partial, L->naxp, axn_count(L), dout2, D);
  ++L->nlaunch;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// ---------------------------------------------------------------------------
// build_white (src/IMSRG_tools.f90:377-434)
// ---------------------------------------------------------------------------
__global__ void k_white_1b(DevLayout L, double* __restrict__ gen, const double* __restrict__ h, double herm) {
  i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  const int n = L.n, mp = L.mp;
  if (e >= (i64)mp * n) return;
  int a = (int)(e % mp), i = (int)(e / mp);  // fph(a,i), a particle-local
  int as = n + a;
  double d = h[L.o_fpp + a + (i64)a * mp] - h[L.o_fhh + i + (i64)i * n] - dv_elem(L, h, herm, as, i, as, i);
  gen[L.o_fph + e] = h[L.o_fph + e] / d;
}

__global__ void k_white_2b(DevLayout L, double* __restrict__ gen, const double* __restrict__ h, double herm) {
  i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= L.pcnt[P_PPHH - P_HHHH]) return;
  int q, row, col;
  i64 pos;
  part_elem(L, P_PPHH - P_HHHH, e, q, pos, row, col);
  int2 p = block_pair(L, q, 2, row), hh = block_pair(L, q, 0, col);
  const int n = L.n, mp = L.mp;
  double efs = h[L.o_fpp + (p.x - n) + (i64)(p.x - n) * mp];
  efs = efs + h[L.o_fpp + (p.y - n) + (i64)(p.y - n) * mp];
  efs = efs - h[L.o_fhh + hh.x + (i64)hh.x * n];
  efs = efs - h[L.o_fhh + hh.y + (i64)hh.y * n];
  // the six diagonal elements, read side by side
  const int xs[6] = {p.x, hh.x, p.x, p.x, p.y, p.y}, ys[6] = {p.y, hh.y, hh.x, hh.y, hh.x, hh.y};
  double v[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const int e = __ldg(&L.ptab[xs[k] * L.m + ys[k]]);
    v[k] = dv_at(dv_pos(L, e, e), h, herm);
  }
  const double Aph = v[0] + v[1] - v[2] - v[3] - v[4] - v[5];
  gen[pos] = h[pos] / (efs + Aph);
}

int launch_white(qd_layout* L, double* gen, const double* h, int herm) {
  i64 n1 = (i64)L->mp * L->n;
  if (n1 > 0) {
    k_white_1b<<<(unsigned)((n1 + 255) / 256), 256, 0, L->stream>>>(L->dev, gen, h, (double)herm);
    ++L->nlaunch;
  }
  i64 n2 = L->dev.pcnt[P_PPHH - P_HHHH];
  if (n2 > 0) {
    k_white_2b<<<(unsigned)((n2 + 255) / 256), 256, 0, L->stream>>>(L->dev, gen, h, (double)herm);
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// ---------------------------------------------------------------------------
// calc_cc (src/commutators.f90:1135-1159): X_q(r,nb) = v_elem(j,k,i,l,H)
// with (i,j) the r-th row pair and (k,l) the nb-th (hole,particle) column pair.
// One thread per row and CC_COLS columns of a block: a row's pair is read once
// for all of them, the columns' reads overlap, and nothing is searched (a
// thread per element with a binary search for its block, both operators at
// N=20, R=20: 320 us; eight columns and 256 rows a CTA through dv_elem's
// branches 215 us, and 46 instead of 17 us at N=6, R=10; this one 195 and 17).
// ---------------------------------------------------------------------------
constexpr int CC_T = 128, CC_ROWS = 128, CC_COLS = 4;
__global__ void __launch_bounds__(CC_T) k_calc_cc(DevLayout L, const int4* __restrict__ tasks,
                                                  const double* __restrict__ h, double herm, double* __restrict__ X) {
  const int4 t = tasks[blockIdx.x];
  const int q = t.x;
  const int2 d = __ldg(&L.ccdim[q]);
  const int2* ab = L.ccab + __ldg(&L.ccab_base[q]);
  const int2* hp = L.cchp + __ldg(&L.cchp_base[q]) + t.z;
  const int nc = min(CC_COLS, d.y - t.z), r1 = min(t.y + CC_ROWS, d.x);
  double* x = X + __ldg(L.ccxoff + q) + (i64)t.z * d.x;
  for (int r = t.y + threadIdx.x; r < r1; r += CC_T) {
    const int2 ij = __ldg(ab + r);
    double v[CC_COLS];
    int e1[CC_COLS], e2[CC_COLS];
#pragma unroll
    for (int c = 0; c < CC_COLS; ++c) {
      const int2 kl = __ldg(hp + min(c, nc - 1));
      e1[c] = __ldg(&L.ptab[ij.y * L.m + kl.x]);
      e2[c] = __ldg(&L.ptab[ij.x * L.m + kl.y]);
    }
#pragma unroll
    for (int c = 0; c < CC_COLS; ++c) v[c] = dv_at(dv_pos(L, e1[c], e2[c]), h, herm);
#pragma unroll
    for (int c = 0; c < CC_COLS; ++c)
      if (c < nc) x[r + (i64)c * d.x] = v[c];
  }
}

int launch_calc_cc(qd_layout* L, const qd_op* H, double* X) {
  if (L->xsize <= 0) return QD_OK;
  if (!L->d_cctask) {
    std::vector<int4> v;
    for (int q = 0; q < L->ncc; ++q)
      for (int c = 0; c < L->ccdim[q].y; c += CC_COLS)
        for (int r = 0; r < L->ccdim[q].x; r += CC_ROWS) v.push_back(int4{q, r, c, 0});
    void* p = nullptr;
    QD_CUDA(cudaMalloc(&p, sizeof(int4) * std::max<size_t>(1, v.size())));
    L->dev_allocs.push_back(p);
    QD_CUDA(copy_table(p, v.data(), sizeof(int4) * v.size()));
    L->ncctask = (int)v.size();
    L->d_cctask = (const int4*)p;
  }
  if (L->ncctask > 0) {
    k_calc_cc<<<L->ncctask, CC_T, 0, L->stream>>>(L->dev, L->d_cctask, H->d, (double)H->herm, X);
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// Device memory of the particle-hole channel: Z and the tile plan that
// re-couples it (built here, ahead of any stream capture).
int ensure_z(qd_layout* L) {
  if (!L->d_z && L->zsize > 0) {
    QD_CUDA(cudaMalloc(&L->d_z, sizeof(double) * L->zsize));
    L->ws_bytes += sizeof(double) * L->zsize;
  }
  return prepare_pandya(L);
}

}  // namespace qd
