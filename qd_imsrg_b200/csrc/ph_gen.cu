// ph_gen.cu -- the particle-hole channel of [A, B] for a generator-like A
// (construct_cc_ints and the re-coupling of commutator_222,
// src/commutators.f90:716-980, src/ME_general.f90:923-952).
//
// In general Z = hB P - hA P^T with P = X_A X_B^T per cross-coupled block and
//   C(xy,uv) += Z[(u,x),(y,v)] - Z[(u,y),(x,v)] + Z[(v,y),(x,u)] - Z[(v,x),(y,u)].
// When A holds only Vpphh, X_A[(i,j),(k,l)] = A(jk,il) with k a hole and l a
// particle is zero unless i is a particle and j a hole, so only the (particle,
// hole) rows of P exist (a twentieth of them at N=12, R=15), and of the
// stored parts only four receive anything.  With p, h particles and holes:
//   pphh: hA (P[(x,v),(u,y)] + P[(y,u),(v,x)] - P[(y,v),(u,x)] - P[(x,u),(v,y)])
//   ppph: hA (P[(y,u),(v,x)] - P[(x,u),(v,y)])      phhh: hA (P[(y,u),(v,x)] - P[(y,v),(u,x)])
//   phph: hA P[(y,u),(v,x)] - hB P[(v,x),(y,u)]
// Per block q: Y = X_B (rows s) times X'_A^T, X'_A the (particle, hole) rows,
// stored [s + row r]: r x r_ph values in place of r x r.  Bound: latency and
// L2 gathers; the operands are small.  Measured at N=12, R=15 (one dGam):
// products 0.34 ms and re-coupling 0.33 ms in the general form, 0.083 ms for
// all three kernels of this one.
#include <algorithm>
#include <memory>
#include <vector>

#include "dev_common.cuh"

namespace qd {

namespace {

constexpr int PG_R = 64, PG_C = 32, PG_T = 256;

struct PhTab {
  const int4* task;     // {block, slot, row tile, column tile}
  const i64* phbase;    // per (particle, hole): its row's first value in Y, [particle + hole (m - n)]
  const int4* xtask;    // {cross-coupled block, column, -, -} of X'_A
  const i64* xoff;      // start of X'_A of a cross-coupled block
};

// X'_A[(p,h), (k,l)] = A(h k, p l) = hA A_pphh: one CTA per column (k,l) of a
// block, threads along its (particle, hole) rows, which are the (hole,
// particle) columns of the opposite block.
__global__ void __launch_bounds__(128) k_xa_gen(DevLayout L, PhTab T, const double* __restrict__ A, double hA,
                                                double* __restrict__ X) {
  const int4 t = T.xtask[blockIdx.x];
  const int q = t.x, c = t.y, qr = t.z;  // qr: the block of the opposite transfer
  const int2 kl = __ldg(&L.cchp[__ldg(&L.cchp_base[q]) + c]);
  const int base = __ldg(&L.cchp_base[qr]), rows = __ldg(&L.ccdim[qr]).y;
  double* x = X + __ldg(&T.xoff[q]) + (i64)c * rows;
  for (int r = threadIdx.x; r < rows; r += 128) {
    const int2 hp = __ldg(&L.cchp[base + r]);
    x[r] = dv_elem(L, A, hA, hp.x, kl.x, hp.y, kl.y);
  }
}

// C += the re-coupled Y.  A warp takes one column (u,v) at a time, its lanes
// rows (x,y); four columns' reads are in flight together.
__global__ void __launch_bounds__(PG_T) k_ph_gen(DevLayout L, PhTab T, const double* __restrict__ Y, double hA,
                                                 double hB, double* __restrict__ C) {
  const int4 t = T.task[blockIdx.x];
  const int q = t.x, slot = t.y, n = L.n, mp = L.mp, m = L.m;
  const int4 bd = __ldg(&L.blk[q]);
  int cr, cc;
  part_classes(P_HHHH + slot, cr, cc);
  const int nr = cr == 1 ? bd.y : bd.z, nc = cc == 0 ? bd.x : bd.y;
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r0 = t.z * PG_R, c0 = t.w * PG_C, ncol = min(PG_C, nc - c0);
  double* out = C + __ldg(L.boff + 6 * q + slot);
  auto P = [&](int p, int h, int s1, int s2) {  // Y[(p,h), (s1,s2)]
    return __ldg(Y + __ldg(&T.phbase[(p - n) + (i64)h * mp]) + __ldg(&L.ccmap[s1 * m + s2]).y);
  };
#pragma unroll
  for (int half = 0; half < PG_R / 32; ++half) {
    const int row = r0 + l + 32 * half;
    if (row >= nr) return;
    const int2 xy = block_pair(L, q, cr, row);
    const int x = xy.x, y = xy.y;
    // columns w, w + 8, w + 16, w + 24 of the tile, past its end the last one
    double v[PG_C / 8], old[PG_C / 8];
#pragma unroll
    for (int j = 0; j < PG_C / 8; ++j) {
      const int col = c0 + min(w + 8 * j, ncol - 1);
      const int2 uv = block_pair(L, q, cc, col);
      const int u = uv.x, s = uv.y;
      old[j] = out[row + (i64)col * nr];
      double z = hA * P(y, u, s, x);
      if (slot == 2)
        z = hA * P(x, s, u, y) - hA * P(y, s, u, x) + z - hA * P(x, u, s, y);
      else if (slot == 4)
        z -= hA * P(x, u, s, y);
      else if (slot == 5)
        z -= hA * P(y, s, u, x);
      else
        z -= hB * P(s, x, y, u);
      v[j] = z;
    }
#pragma unroll
    for (int j = 0; j < PG_C / 8; ++j)
      if (w + 8 * j < ncol) out[row + (i64)(c0 + w + 8 * j) * nr] = old[j] + v[j];
  }
}

}  // namespace

struct PhGen {
  PhTab tab{};
  int ntask = 0, nxtask = 0;
  double* d_xa = nullptr;
  double* d_y = nullptr;
  GemmProgram prog;
};

void ph_gen_free(qd_layout* L) {
  if (!L->ph_gen) return;
  L->ph_gen->prog.clear_device();
  delete L->ph_gen;
  L->ph_gen = nullptr;
}

// Tables, the products' program and the buffers of L (ahead of a stream
// capture, which must not allocate).
int prepare_ph_gen(qd_layout* L) {
  if (L->ph_gen) return QD_OK;
  std::unique_ptr<PhGen> p(new PhGen());  // the layout's when complete: a failure leaves no plan
  const int n = L->n, mp = L->mp, m = L->m;
  std::vector<i64> phbase((size_t)std::max(1, mp * n), 0), xoff(std::max(1, L->ncc), 0), yoff(std::max(1, L->ncc), 0);
  std::vector<int4> xtask, task;
  std::vector<PhProduct> prod;
  i64 xa = 0, ys = 0;
  for (int q = 0; q < L->ncc; ++q) {
    // opposite transfer: blocks run over ML, then MS, symmetric about zero
    const int qr = L->ncc - 1 - q, r = L->ccdim[q].x, nb = L->ccdim[q].y, rows = L->ccdim[qr].y;
    xoff[q] = xa;
    yoff[q] = ys;
    if (r == 0 || rows == 0) continue;
    for (int c = 0; c < nb; ++c) xtask.push_back(int4{q, c, qr, 0});
    for (int k = 0; k < rows; ++k) {
      const int2 hp = L->cchp[L->cchp_base[qr] + k];
      phbase[(hp.y - n) + (size_t)hp.x * mp] = ys + (i64)k * r;
      if (L->ccmap[(size_t)hp.y * m + hp.x].x != q) {
        set_error("particle-hole tables: pair (%d, %d) is not in the opposite block", hp.y, hp.x);
        return QD_ERR_LAYOUT;
      }
    }
    prod.push_back(PhProduct{r, rows, nb, ys, L->ccxoff[q], xa});
    xa += (i64)rows * nb;
    ys += (i64)rows * r;
  }
  for (int q = 0; q < L->nblock; ++q) {
    const int nh = L->blk[q].x, nb = L->blk[q].y, np = L->blk[q].z;
    const int rows[6] = {0, 0, np, nb, np, nb}, cols[6] = {0, 0, nh, nb, nb, nh};
    for (int slot = 2; slot < 6; ++slot)
      for (int i = 0; i * PG_R < rows[slot]; ++i)
        for (int j = 0; j * PG_C < cols[slot]; ++j) task.push_back(int4{q, slot, i, j});
  }
  p->ntask = (int)task.size();
  p->nxtask = (int)xtask.size();
  PlanMemory mem;
  mem.add(task, &p->tab.task);
  mem.add(phbase, &p->tab.phbase);
  mem.add(xtask, &p->tab.xtask);
  mem.add(xoff, &p->tab.xoff);
  mem.room(xa, &p->d_xa);
  mem.room(ys, &p->d_y);
  int rc = build_ph_products(L, prod, p->prog);
  if (!rc) rc = prepare_program(L, p->prog, 0u, 0u);
  if (!rc) rc = mem.commit(L);
  if (rc) {
    p->prog.clear_device();
    return rc;
  }
  L->ph_gen = p.release();
  return QD_OK;
}

// The products of the particle-hole channel of [A, B] for a generator-like A,
// XB the cross-coupled matrices of B.
int launch_ph_gen_products(qd_layout* L, const qd_op* A, const double* XB, double hB) {
  int rc = prepare_ph_gen(L);
  if (rc) return rc;
  PhGen* p = L->ph_gen;
  const double hA = (double)A->herm;
  if (p->nxtask > 0) {
    k_xa_gen<<<p->nxtask, 128, 0, L->stream>>>(L->dev, p->tab, A->d, hA, p->d_xa);
    ++L->nlaunch;
  }
  const double* bufs[NBUF] = {nullptr, nullptr, p->d_xa, XB, nullptr, nullptr, p->d_y};
  if ((rc = run_program_f64(L, p->prog, bufs, hA, hB, 0u, 0u))) return rc;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// Their re-coupling into C.
int launch_ph_gen(qd_layout* L, double hA, double hB, double* C) {
  PhGen* p = L->ph_gen;
  if (p->ntask > 0) {
    k_ph_gen<<<p->ntask, PG_T, 0, L->stream>>>(L->dev, p->tab, p->d_y, hA, hB, C);
    ++L->nlaunch;
  }
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

}  // namespace qd
