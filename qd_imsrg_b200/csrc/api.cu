// api.cu -- extern "C" entry points (include/qd_imsrg.h).
//
// Host orchestration of the reference's call sequences on device-resident
// operators; every numeric step is a kernel on the layout's stream.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <utility>
#include <vector>

#include "dev_common.cuh"

namespace qd {
const char* last_error();
void drop_122_plan(const qd_layout* L);
}  // namespace qd

using namespace qd;

// Layout-owned workspaces used by qd_commutator (allocated on first use).
namespace {
struct Workspace {
  qd_op* w1 = nullptr;
  qd_op* w2 = nullptr;
  qd_cc* ca = nullptr;
  qd_cc* cb = nullptr;
  // Magnus flow: ETA, G, DG, ETA0, G0, HS0, INT1, INT2, AD, w1, w2 and HCC,
  // OCC, allocated by the first flow on the layout and kept
  qd_op* flow[11] = {nullptr};
  qd_cc* flow_cc[2] = {nullptr};
  qd_op* eta = nullptr;  // dGam's generator
  qd_op* eomq = nullptr;  // EOM matvec: excitation operator, second commutator
  qd_op* eomt = nullptr;
};
std::map<const qd_layout*, Workspace>& workspaces() {
  static std::map<const qd_layout*, Workspace> m;
  return m;
}
std::mutex g_ws_mutex;  // workspaces of different layouts from concurrent host threads

#define CHECK(cond, code, ...)    \
  do {                            \
    if (!(cond)) {                \
      qd::set_error(__VA_ARGS__); \
      return code;                \
    }                             \
  } while (0)
#define TRY(x)               \
  do {                       \
    int rc_ = (x);           \
    if (rc_) return rc_;     \
  } while (0)

int use_device(const qd_layout* L) {
  if (L->device == QD_HOST_ONLY) {
    qd::set_error("layout was created host-only (QD_HOST_ONLY)");
    return QD_ERR_STATE;
  }
  QD_CUDA(cudaSetDevice(L->device));
  return QD_OK;
}

int op_new(qd_layout* L, int herm, qd_op** out) {
  qd_op* op = new qd_op();
  op->L = L;
  op->herm = herm;
  cudaError_t e = cudaMalloc(&op->d, sizeof(double) * L->neq);
  if (e != cudaSuccess) {
    delete op;
    return cuda_fail(e, "cudaMalloc(operator)");
  }
  ++L->children;
  QD_CUDA(cudaMemsetAsync(op->d, 0, sizeof(double) * L->neq, L->stream));
  op->zero_mask = ALL_PARTS | CONSERVES;
  *out = op;
  return QD_OK;
}

// Tear down a layout's device state and the layout itself.
void layout_finish(qd_layout* L) {
  drop_122_plan(L);
  drop_eom_plans(L);
  layout_free_device(L);
  delete L;
}

// A layout destroyed while operators or cross-coupled matrices still refer
// to it (e.g. a garbage collector finalising the layout first) stays alive
// until the last of them is freed.
void release_child(qd_layout* L) {
  if (--L->children == 0 && L->closing) layout_finish(L);
}

void op_free(qd_op* op) {
  if (!op) return;
  qd_layout* L = op->L;
  if (op->d) cudaFree(op->d);
  delete op;
  release_child(L);
}

void cc_free(qd_cc* c) {
  if (!c) return;
  qd_layout* L = c->L;
  if (c->d) cudaFree(c->d);
  delete c;
  release_child(L);
}

int cc_new(qd_layout* L, double herm, qd_cc** out) {
  qd_cc* c = new qd_cc();
  c->L = L;
  c->herm = herm;
  if (L->xsize > 0) {
    cudaError_t e = cudaMalloc(&c->d, sizeof(double) * L->xsize);
    if (e != cudaSuccess) {
      delete c;
      return cuda_fail(e, "cudaMalloc(cc)");
    }
  }
  ++L->children;
  if (c->d) QD_CUDA(cudaMemsetAsync(c->d, 0, sizeof(double) * L->xsize, L->stream));
  *out = c;
  return QD_OK;
}

int scalar_out(qd_layout* L, const double* dslot, double* out) {
  QD_CUDA(cudaMemcpyAsync(L->h_red, dslot, sizeof(double), cudaMemcpyDeviceToHost, L->stream));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  *out = L->h_red[0];
  return QD_OK;
}

int same_layout(const qd_op* a, const qd_op* b) {
  CHECK(a && b, QD_ERR_ARG, "null operator handle");
  CHECK(a->L == b->L, QD_ERR_ARG, "operators belong to different layouts");
  // an operand whose raw pointer the caller holds may have been written since
  // its mask was set (by an upload, a copy, a result): nothing is known zero
  for (const qd_op* o : {a, b})
    if (o->exposed) const_cast<qd_op*>(o)->zero_mask = 0;
  return QD_OK;
}

// Operators of one role pair (G/G0, HS/HS0, ETA/ETA0, INT2/AD) trade buffers
// instead of copying: "G0 = G" becomes a swap after which G's buffer is
// rewritten.
void swap_ops(qd_op* a, qd_op* b) {
  std::swap(a->d, b->d);
  std::swap(a->zero_mask, b->zero_mask);
  std::swap(a->exposed, b->exposed);
}

// zero mask of a host vector: parts that are identically zero
unsigned host_zero_mask(const qd_layout* L, const double* v) {
  auto zero = [&](i64 o, i64 n) {
    for (i64 i = 0; i < n; ++i)
      if (v[o + i] != 0.0) return false;
    return true;
  };
  unsigned m = 0;
  if (zero(L->o_fhh, (i64)L->n * L->n)) m |= 1u << P_FHH;
  if (zero(L->o_fpp, (i64)L->mp * L->mp)) m |= 1u << P_FPP;
  if (zero(L->o_fph, (i64)L->mp * L->n)) m |= 1u << P_FPH;
  for (int p = 0; p < 6; ++p) {
    bool z = true;
    for (int q = 0; q < L->nblock && z; ++q) {
      i64 nh = L->blk[q].x, nb = L->blk[q].y, np = L->blk[q].z;
      i64 sz[6] = {nh * nh, np * np, np * nh, nb * nb, np * nb, nb * nh};
      z = zero(L->boff[6 * q + p], sz[p]);
    }
    if (z) m |= 1u << (P_HHHH + p);
  }
  const int n = L->n, mp = L->mp;
  bool cons = true;
  for (int j = 0; j < L->m && cons; ++j)
    for (int i = 0; i < L->m && cons; ++i) {
      if (L->gid[i] == L->gid[j] || (i < n && j >= n)) continue;
      const i64 e = i < n ? L->o_fhh + i + (i64)j * n
                          : (j < n ? L->o_fph + (i - n) + (i64)j * mp : L->o_fpp + (i - n) + (i64)(j - n) * mp);
      cons = v[e] == 0.0;
    }
  if (cons) m |= CONSERVES;
  return m;
}

// CONSERVES of a commutator: both operands conserve (m_l, m_s)
unsigned conserves(const qd_op* a, const qd_op* b) { return a->zero_mask & b->zero_mask & CONSERVES; }

// RAII stage timer: records an event pair around a stage when profiling is on
struct StageTimer {
  qd_layout* L;
  int id;
  cudaEvent_t a = nullptr, b = nullptr;
  StageTimer(qd_layout* l, int i) : L(l), id(i) {
    if (L->prof.on && cudaEventCreate(&a) == cudaSuccess && cudaEventCreate(&b) == cudaSuccess)
      cudaEventRecord(a, L->stream);
  }
  void cancel() {  // nothing was launched
    if (a) cudaEventDestroy(a);
    if (b) cudaEventDestroy(b);
    a = b = nullptr;
  }
  ~StageTimer() {
    if (L->prof.on && a && b) {
      cudaEventRecord(b, L->stream);
      L->prof.pending[id].push_back({a, b});
    }
  }
};

void prof_collect(qd_layout* L) {
  for (int s = 0; s < S_COUNT; ++s) {
    for (auto& pr : L->prof.pending[s]) {
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, pr.first, pr.second) == cudaSuccess) {
        L->prof.ms[s] += ms;
        L->prof.count[s] += 1;
      }
      cudaEventDestroy(pr.first);
      cudaEventDestroy(pr.second);
    }
    L->prof.pending[s].clear();
  }
}

// ---- the stages of one commutator [A,B] -> C ------------------------------
int stage_e0(qd_layout* L, const qd_op* A, const qd_op* B, double* dout, double add) {
  StageTimer tm(L, S_E0);
  const double dh = (double)(A->herm - B->herm);
  TRY(reduce_dot_range(L, A->d, B->d, L->o_fph, (i64)L->mp * L->n, dh, add, dout));
  TRY(reduce_dot_part(L, A->d, B->d, P_PPHH, dh, 1.0, dout));
  return QD_OK;
}

int stage_111(qd_layout* L, const qd_op* A, const qd_op* B, qd_op* C) {
  StageTimer tm(L, S_111);
  const double* bufs[7] = {A->d, B->d, nullptr, nullptr, C->d, nullptr, nullptr};
  TRY(run_program(L, L->prog_111, bufs, (double)A->herm, (double)B->herm, A->zero_mask, B->zero_mask));
  C->zero_mask = (C->zero_mask & ~(ONE_BODY | CONSERVES)) | conserves(A, B);
  return QD_OK;
}

// commutator_221 with the reference's visible intermediates w1, w2
int stage_221(qd_layout* L, const qd_op* A, const qd_op* B, qd_op* C, qd_op* w1, qd_op* w2) {
  StageTimer tm(L, S_221);
  QD_CUDA(cudaMemsetAsync(w1->d, 0, sizeof(double) * L->neq, L->stream));
  QD_CUDA(cudaMemsetAsync(w2->d, 0, sizeof(double) * L->neq, L->stream));
  const double* bufs[7] = {A->d, B->d, nullptr, nullptr, w1->d, w2->d, nullptr};
  TRY(run_program(L, L->prog_221, bufs, (double)A->herm, (double)B->herm, A->zero_mask, B->zero_mask));
  w1->zero_mask = 0;
  w2->zero_mask = 0;
  TRY(launch_221_trace(L, A, B, w1, w2, C->d));
  return QD_OK;
}

// Whether a whole commutator takes its ladders with 122 (a split-form layout
// keeps every ladder in the split form), and the ladders left then.
bool ladder_in_122(const qd_layout* L, const qd_op* A) { return gen_like(A->zero_mask) && L->split_slices == 0; }
GemmProgram& ladder_program(qd_layout* L, const qd_op* A) {
  return ladder_in_122(L, A) ? L->prog_ladder_gen : L->prog_ladder;
}

// From here on a BCH term's update of HS runs where C_pppp is made: reading
// C_pppp back then costs more than the slower kernel does.  Whole flows with
// the update in one pass and split (ms, medians of 24, three runs within 0.3%):
// N=20 R=12 (1.7 M entries) 6.90 and 7.33, N=12 R=14 (5.4 M) 10.63 and 10.88,
// N=12 R=15 (8.7 M) 14.49 and 14.55, N=20 R=16 (13 M) 19.48 and 19.05, N=6 R=16
// (14 M) 14.41 and 13.70, N=20 R=20 (62 M) 61.1 and 57.9: equal near 9 M.
constexpr i64 SPLIT_UPDATE_ENTRIES = 8000000;
// Whether a BCH term's update of HS runs where C_pppp is made: C_pppp must be
// final there (no ladder left to the grouped GEMM; the particle-hole channel
// adds nothing to it, see launch_pandya_tiles).
bool splits_update(qd_layout* L, const qd_op* G) {
  return L->neq >= SPLIT_UPDATE_ENTRIES && ladder_in_122(L, G) && L->prog_ladder_gen.probs.empty();
}

int stage_ladders(qd_layout* L, const qd_op* A, const qd_op* B, qd_op* C, GemmProgram& ladders) {
  const double* bufs[7] = {A->d, B->d, nullptr, nullptr, C->d, nullptr, nullptr};
  StageTimer tm(L, S_LADDER);
  return run_program(L, ladders, bufs, (double)A->herm, (double)B->herm, A->zero_mask, B->zero_mask);
}

// construct_cc_ints: Z of the cross-coupled matrices, and its re-coupling into C
int stage_ph_product(qd_layout* L, const qd_cc* HCC, const qd_cc* ETACC) {
  TRY(ensure_z(L));
  const double* zb[7] = {nullptr, nullptr, ETACC->d, HCC->d, nullptr, nullptr, L->d_z};
  StageTimer tm(L, S_PANDYA_GEMM);
  return run_program(L, L->prog_pandya, zb, ETACC->herm, HCC->herm, 0u, 0u);
}
int stage_ph_recouple(qd_layout* L, qd_op* C) {
  StageTimer tm(L, S_PANDYA_GATHER);
  return launch_pandya_tiles(L, L->d_z, C->d);
}

int stage_222(qd_layout* L, const qd_op* A, const qd_op* B, qd_op* C, const qd_cc* HCC, const qd_cc* ETACC) {
  TRY(stage_ladders(L, A, B, C, L->prog_ladder));
  if (HCC && ETACC && HCC->filled && ETACC->filled && L->zsize > 0) {
    CHECK(std::fabs(HCC->herm) == 1.0 && std::fabs(ETACC->herm) == 1.0, QD_ERR_ARG,
          "cross-coupled herm must be +1 or -1");
    TRY(stage_ph_product(L, HCC, ETACC));
    TRY(stage_ph_recouple(L, C));
  }
  C->zero_mask = 0;
  return QD_OK;
}

int white(qd_op* gen, const qd_op* H) {
  TRY(launch_white(H->L, gen->d, H->d, H->herm));
  gen->zero_mask &= ~((1u << P_FPH) | (1u << P_PPHH)) & (conserves(H, H) ? ~0u : ~CONSERVES);
  return QD_OK;
}

// E0 and the one-body part of C = [A, B] (110, 220, 111, 121, 221): two
// launches when both operands conserve (m_l, m_s), piece by piece otherwise.
int stage_one_body(qd_layout* L, const qd_op* A, const qd_op* B, qd_op* C) {
  // the split form keeps the pieces: its 111 is a product of slices
  if (L->split_slices == 0) {
    bool done = false;
    StageTimer tm(L, S_221);
    TRY(launch_onebody(L, A, B, C->d, &done));
    if (done) return QD_OK;
    tm.cancel();
  }
  TRY(stage_e0(L, A, B, C->d, 0.0));
  TRY(stage_111(L, A, B, C));
  {
    StageTimer tm(L, S_121);
    TRY(launch_121(L, A, B, C->d));
  }
  StageTimer tm(L, S_221);
  return launch_221_fused(L, A, B, C->d);
}

// Branches of one commutator beside the layout's stream.  E0 and the
// one-body part, and for a generator-like A the parts other than C_pppp,
// depend on nothing else of the commutator; their kernels leave much of the
// chip idle (latency-bound, or a last wave of few CTAs), which the other
// branches fill.  Measured with and without branches (us): generator-like A
// N=6 R=8 27 and 48, N=12 R=12 62 and 83, N=20 R=16 176 and 222; two dense
// operators N=6 R=8 151 and 163, N=12 R=14 (5.4 M entries) 1215 and 1235,
// N=20 R=16 (13 M) 3158 and 3109: there the tiles of 122 fill the chip and
// the one-body kernels only disturb them.
constexpr i64 FORK_ENTRIES = 8000000;

struct Branches {
  qd_layout* L = nullptr;
  bool on = false;
  int used = 0;  // bit k: branch k has work
  int open = 0;  // bit k: branch k may have work
  int fork(qd_layout* l, const qd_op* A) {
    L = l;
    if (L->prof.on || (!gen_like(A->zero_mask) && L->neq >= FORK_ENTRIES)) return QD_OK;
    bool use;
    TRY(use_branches(L, &use));
    if (!use) return QD_OK;
    QD_CUDA(cudaEventRecord(L->ev_fork, L->stream));
    on = true;
    // The split form's programs (111, the products, the ladders) share one set
    // of slices and accumulators on the layout (run_program_split): they stay
    // in order on the main stream, and only 122, which uses none of these,
    // runs beside them (all in one stream and 122 beside: [Omega, X] with three
    // slices at N=6, R=15 328 and 276 us, two dense operators with three at
    // N=6, R=10 364 and 347 us).
    open = L->split_slices > 0 ? 1 << 1 : (1 << qd_layout::NSIDE) - 1;
    return QD_OK;
  }
  // stream of branch k (the main one without branches)
  int side(int k, cudaStream_t* st) {
    const bool go = on && ((open >> k) & 1);
    *st = go ? L->side[k] : L->stream;
    if (go && !((used >> k) & 1)) {
      QD_CUDA(cudaStreamWaitEvent(*st, L->ev_fork, 0));
      used |= 1 << k;
    }
    return QD_OK;
  }
  // wait for one branch, or for all (which ends the branches)
  int join(int one = -1) {
    if (!on) return QD_OK;
    on = one >= 0;
    for (int k = 0; k < qd_layout::NSIDE; ++k) {
      if (!((used >> k) & 1) || (one >= 0 && k != one)) continue;
      used &= ~(1 << k);
      QD_CUDA(cudaEventRecord(L->ev_side[k], L->side[k]));
      QD_CUDA(cudaStreamWaitEvent(L->stream, L->ev_side[k], 0));
    }
    return QD_OK;
  }
  // an error path: the main stream still waits for what was launched
  ~Branches() {
    if (on) join();
  }
};

// The layout's launches go to another stream while this lives.
struct OnStream {
  qd_layout* L;
  cudaStream_t keep;
  OnStream(qd_layout* l, cudaStream_t s) : L(l), keep(l->stream) { L->stream = s; }
  ~OnStream() { L->stream = keep; }
};

// upd: also the BCH update of HS.  fill_acc: the caller can see ACC, which a
// generator-like A's particle-hole channel does not need (see ph_gen.cu).
int commutator_seq(qd_layout* L, const qd_op* A, const qd_op* B, qd_op* C, qd_op* w1, qd_op* w2, qd_cc* ACC,
                   qd_cc* BCC, bool pandya, const HsUpdate* upd = nullptr, bool fill_acc = true) {
  (void)w1;  // workspaces of the whole commutator: the fused 221 leaves them untouched
  (void)w2;
  TRY(build_programs(L));
  const bool gen = gen_like(A->zero_mask);
  const bool ph_short = pandya && gen && L->split_slices == 0 && L->ncc > 0;
  Branches br;
  cudaStream_t side;
  TRY(br.fork(L, A));
  if (pandya) {
    TRY(br.side(2, &side));
    OnStream os(L, side);
    StageTimer tm(L, S_CALC_CC);
    if (!ph_short || fill_acc) TRY(launch_calc_cc(L, A, ACC->d));
    ACC->filled = true;
    ACC->herm = A->herm;
    TRY(launch_calc_cc(L, B, BCC->d));
    BCC->filled = true;
    BCC->herm = B->herm;
  }
  const bool ph_full = pandya && !ph_short && L->zsize > 0;
  if (ph_short || ph_full) {
    TRY(br.side(2, &side));
    OnStream os(L, side);
    if (ph_short) {
      StageTimer tm(L, S_PANDYA_GEMM);
      TRY(launch_ph_gen_products(L, A, BCC->d, (double)B->herm));
    } else {
      TRY(stage_ph_product(L, BCC, ACC));
    }
  }
  {
    TRY(br.side(0, &side));
    OnStream os(L, side);
    TRY(stage_one_body(L, A, B, C));
  }
  {
    TRY(br.side(1, &side));
    StageTimer tm(L, S_122);
    TRY(launch_122(L, A, B, C->d, ladder_in_122(L, A), side, upd));
  }
  GemmProgram& ladders = ladder_program(L, A);
  TRY(br.join(1));  // the rest adds to the two-body parts
  if (!ladders.probs.empty()) TRY(stage_ladders(L, A, B, C, ladders));
  TRY(br.join());
  if (ph_short) {
    StageTimer tm(L, S_PANDYA_GATHER);
    TRY(launch_ph_gen(L, (double)A->herm, (double)B->herm, C->d));
  }
  if (ph_full) TRY(stage_ph_recouple(L, C));
  C->zero_mask = conserves(A, B);
  return QD_OK;
}

int get_ws(qd_layout* L, Workspace** out) {
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  Workspace& w = workspaces()[L];
  if (!w.w1) TRY(op_new(L, 1, &w.w1));
  if (!w.w2) TRY(op_new(L, 1, &w.w2));
  if (!w.ca) TRY(cc_new(L, -1.0, &w.ca));
  if (!w.cb) TRY(cc_new(L, 1.0, &w.cb));
  *out = &w;
  return QD_OK;
}

void drop_ws(const qd_layout* L) {
  Workspace w;
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    auto& m = workspaces();
    auto it = m.find(L);
    if (it == m.end()) return;
    w = it->second;
    m.erase(it);
  }
  op_free(w.w1);
  op_free(w.w2);
  cc_free(w.ca);
  cc_free(w.cb);
  for (qd_op* o : w.flow) op_free(o);
  for (qd_cc* c : w.flow_cc) cc_free(c);
  op_free(w.eta);
  op_free(w.eomq);
  op_free(w.eomt);
}

}  // namespace

int qd::make_branches(qd_layout* L) {
  if (L->ev_fork) return QD_OK;
  for (int k = 0; k < qd_layout::NSIDE; ++k) {  // a call after a failed one makes what is missing
    if (!L->side[k]) QD_CUDA(cudaStreamCreateWithFlags(&L->side[k], cudaStreamNonBlocking));
    if (!L->ev_side[k]) QD_CUDA(cudaEventCreateWithFlags(&L->ev_side[k], cudaEventDisableTiming));
  }
  QD_CUDA(cudaEventCreateWithFlags(&L->ev_fork, cudaEventDisableTiming));
  return QD_OK;
}

// Whether the calling launch may use the side streams.  Making them takes
// about 200 us; a call without them takes 10 to 40 us longer.  So the first
// calls go without: a layout that is used once or twice, as in a scan over
// dots, never pays for them (first commutator at N=2, R=3 780 and 580 us, first
// EOM product at N=12, R=10 1280 and 1100).  A step graph makes them for its
// capture, since it is replayed.
int qd::use_branches(qd_layout* L, bool* use) {
  constexpr int SERIAL_CALLS = 2;
  *use = L->ev_fork != nullptr;
  if (*use) return QD_OK;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  QD_CUDA(cudaStreamIsCapturing(L->stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) return QD_OK;  // no stream or event is created inside a capture
  if (L->serial_calls++ < SERIAL_CALLS) return QD_OK;
  TRY(make_branches(L));
  *use = true;
  return QD_OK;
}

// A workspace operator of the layout that the full commutator never reads
// or writes (the reference's w1/w2, which the fused 221 replaces), for the
// autotuner's timed launches; NULL if none is allocated yet.
double* qd::scratch_operator(qd_layout* L) {
  std::lock_guard<std::mutex> lock(g_ws_mutex);
  auto it = workspaces().find(L);
  if (it == workspaces().end()) return nullptr;
  const Workspace& w = it->second;
  for (qd_op* o : {w.w1, w.w2, w.flow[9], w.flow[10]})
    if (o) return o->d;
  return nullptr;
}

namespace {

const double kCof[11] = QD_BCH_COF;

}  // namespace

extern "C" {

const char* qd_last_error(void) { return qd::last_error(); }
const char* qd_version(void) { return "qd_imsrg_b200 0.1 (sm_100a, FP64 DMMA)"; }

int qd_layout_create(int nbody, int emax, const double* eig, int device, qd_layout** out) {
  CHECK(out, QD_ERR_ARG, "qd_layout_create: null output");
  *out = nullptr;
  if (device == QD_HOST_ONLY) {
    qd_layout* L = new qd_layout();
    L->device = QD_HOST_ONLY;
    int rc = layout_build(L, nbody, emax, eig);
    if (rc) {
      delete L;
      return rc;
    }
    *out = L;
    return QD_OK;
  }
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    qd::set_error("qd_layout_create: no CUDA device");
    return QD_ERR_NODEVICE;
  }
  qd_layout* L = new qd_layout();
  if (device < 0) {
    cudaGetDevice(&L->device);
  } else {
    L->device = device;
  }
  int rc = layout_build(L, nbody, emax, eig);
  if (rc) {
    delete L;
    return rc;
  }
  if ((rc = use_device(L)) || (rc = layout_upload(L))) {
    layout_free_device(L);
    delete L;
    return rc;
  }
  cudaError_t e = cudaStreamCreateWithFlags(&L->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    layout_free_device(L);
    delete L;
    return cuda_fail(e, "cudaStreamCreate");
  }
  L->own_stream = true;
  if ((rc = ensure_reduction(L))) {
    layout_free_device(L);
    delete L;
    return rc;
  }
  *out = L;
  return QD_OK;
}

int qd_layout_destroy(qd_layout* L) {
  if (!L) return QD_OK;
  if (L->device == QD_HOST_ONLY) {
    delete L;
    return QD_OK;
  }
  cudaSetDevice(L->device);
  cudaStreamSynchronize(L->stream);
  drop_ws(L);
  if (L->children > 0)
    L->closing = true;  // the last operator or cc freed finishes the teardown
  else
    layout_finish(L);
  (void)cudaGetLastError();
  return QD_OK;
}

int qd_layout_info(const qd_layout* L, int* nbody, int* msp, int* nblock, int64_t* neq, int* ncc) {
  CHECK(L, QD_ERR_ARG, "null layout");
  if (nbody) *nbody = L->n;
  if (msp) *msp = L->m;
  if (nblock) *nblock = L->nblock;
  if (neq) *neq = L->neq;
  if (ncc) *ncc = L->ncc;
  return QD_OK;
}

int qd_layout_blocks(const qd_layout* L, int* d) {
  CHECK(L && d, QD_ERR_ARG, "null argument");
  for (int q = 0; q < L->nblock; ++q) {
    d[5 * q + 0] = L->blk[q].x;
    d[5 * q + 1] = L->blk[q].y;
    d[5 * q + 2] = L->blk[q].z;
    int MS = -2 + 2 * (q / (4 * L->emax - 3));
    int ML = 2 - 2 * L->emax + q % (4 * L->emax - 3);
    d[5 * q + 3] = ML;
    d[5 * q + 4] = MS;
  }
  return QD_OK;
}

int qd_layout_offsets(const qd_layout* L, int64_t* off6) {
  CHECK(L && off6, QD_ERR_ARG, "null argument");
  for (size_t i = 0; i < L->boff.size(); ++i) off6[i] = L->boff[i];
  return QD_OK;
}

int qd_layout_pairs(const qd_layout* L, int q, int kind, int* out, int* count) {
  CHECK(L && q >= 0 && q < L->nblock && kind >= 0 && kind <= 2, QD_ERR_ARG, "qd_layout_pairs: bad arguments");
  int nh = L->blk[q].x, nb = L->blk[q].y, np = L->blk[q].z;
  int base = L->pbase[q] + (kind == 0 ? 0 : (kind == 1 ? nh : nh + nb));
  int cnt = kind == 0 ? nh : (kind == 1 ? nb : np);
  if (count) *count = cnt;
  if (out)
    for (int k = 0; k < cnt; ++k) {
      out[2 * k] = L->pairs[base + k].x + 1;
      out[2 * k + 1] = L->pairs[base + k].y + 1;
    }
  return QD_OK;
}

int qd_layout_set_stream(qd_layout* L, void* stream) {
  CHECK(L, QD_ERR_ARG, "null layout");
  TRY(use_device(L));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  if (L->own_stream && L->stream) cudaStreamDestroy(L->stream);
  if (stream) {
    L->stream = (cudaStream_t)stream;
    L->own_stream = false;
  } else {
    QD_CUDA(cudaStreamCreateWithFlags(&L->stream, cudaStreamNonBlocking));
    L->own_stream = true;
  }
  return QD_OK;
}

int qd_layout_set_split(qd_layout* L, int slices) {
  CHECK(L, QD_ERR_ARG, "null layout");
  CHECK(slices >= 0 && slices <= 8, QD_ERR_ARG, "qd_layout_set_split: slices must be 0..8");
  L->split_slices = slices;
  return QD_OK;
}

int qd_layout_set_graphs(qd_layout* L, int enable) {
  CHECK(L, QD_ERR_ARG, "null layout");
  if (!enable && L->graphs) {
    TRY(use_device(L));
    QD_CUDA(cudaStreamSynchronize(L->stream));
    graphs_free(L);
  }
  L->use_graphs = enable != 0;
  return QD_OK;
}

int qd_layout_graph_stats(const qd_layout* L, int64_t* captured, int64_t* replays) {
  CHECK(L, QD_ERR_ARG, "null layout");
  if (captured) *captured = L->graphs_captured;
  if (replays) *replays = L->graph_replays;
  return QD_OK;
}

int qd_layout_get_split(const qd_layout* L, int* slices) {
  CHECK(L && slices, QD_ERR_ARG, "null argument");
  *slices = L->split_slices;
  return QD_OK;
}

int qd_layout_synchronize(qd_layout* L) {
  CHECK(L, QD_ERR_ARG, "null layout");
  TRY(use_device(L));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  return QD_OK;
}

int qd_layout_profile(qd_layout* L, int enable) {
  CHECK(L, QD_ERR_ARG, "null layout");
  TRY(use_device(L));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  prof_collect(L);
  for (int s = 0; s < S_COUNT; ++s) {
    L->prof.ms[s] = 0.0;
    L->prof.count[s] = 0;
  }
  L->prof.on = enable != 0;
  return QD_OK;
}

int qd_layout_profile_read(qd_layout* L, double* ms, int64_t* counts, int nstage) {
  CHECK(L, QD_ERR_ARG, "null layout");
  TRY(use_device(L));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  prof_collect(L);
  for (int s = 0; s < nstage && s < S_COUNT; ++s) {
    if (ms) ms[s] = L->prof.ms[s];
    if (counts) counts[s] = L->prof.count[s];
  }
  return QD_OK;
}

int qd_layout_tuning(const qd_layout* L, char* buf, int64_t len, int64_t* needed) {
  CHECK(L, QD_ERR_ARG, "null layout");
  const std::string r = tuning_report_122(L);
  if (needed) *needed = (int64_t)r.size() + 1;
  if (buf && len > 0) {
    const size_t n = std::min<size_t>((size_t)len - 1, r.size());
    std::memcpy(buf, r.data(), n);
    buf[n] = 0;
  }
  return QD_OK;
}

int qd_layout_launches(const qd_layout* L, int64_t* n) {
  CHECK(L && n, QD_ERR_ARG, "null argument");
  *n = L->nlaunch;
  return QD_OK;
}

int qd_layout_workspace_bytes(const qd_layout* L, int64_t* bytes) {
  CHECK(L && bytes, QD_ERR_ARG, "null argument");
  *bytes = L->ws_bytes;
  return QD_OK;
}

int qd_op_create(qd_layout* L, int herm, qd_op** out) {
  CHECK(L && out, QD_ERR_ARG, "null argument");
  TRY(use_device(L));
  return op_new(L, herm, out);
}

int qd_op_destroy(qd_op* op) {
  if (!op) return QD_OK;
  cudaSetDevice(op->L->device);
  cudaStreamSynchronize(op->L->stream);
  op_free(op);
  (void)cudaGetLastError();  // teardown errors are not reported; do not leave them pending
  return QD_OK;
}

int qd_op_upload(qd_op* op, const double* v, int64_t neq) {
  CHECK(op && v, QD_ERR_ARG, "null argument");
  CHECK(neq == op->L->neq, QD_ERR_ARG, "qd_op_upload: %lld entries given, layout has %lld", (long long)neq,
        (long long)op->L->neq);
  TRY(use_device(op->L));
  QD_CUDA(cudaMemcpyAsync(op->d, v, sizeof(double) * neq, cudaMemcpyHostToDevice, op->L->stream));
  op->zero_mask = host_zero_mask(op->L, v);
  QD_CUDA(cudaStreamSynchronize(op->L->stream));
  return QD_OK;
}

int qd_op_upload_device(qd_op* op, const double* v, int64_t neq) {
  CHECK(op && v, QD_ERR_ARG, "null argument");
  CHECK(neq == op->L->neq, QD_ERR_ARG, "qd_op_upload_device: size mismatch");
  TRY(use_device(op->L));
  QD_CUDA(cudaMemcpyAsync(op->d, v, sizeof(double) * neq, cudaMemcpyDeviceToDevice, op->L->stream));
  op->zero_mask = 0;
  return QD_OK;
}

int qd_op_download(const qd_op* op, double* v, int64_t neq) {
  CHECK(op && v, QD_ERR_ARG, "null argument");
  CHECK(neq == op->L->neq, QD_ERR_ARG, "qd_op_download: size mismatch");
  TRY(use_device(op->L));
  QD_CUDA(cudaMemcpyAsync(v, op->d, sizeof(double) * neq, cudaMemcpyDeviceToHost, op->L->stream));
  QD_CUDA(cudaStreamSynchronize(op->L->stream));
  return QD_OK;
}

int qd_op_set_herm(qd_op* op, int herm) {
  CHECK(op && (herm == 1 || herm == -1), QD_ERR_ARG, "herm must be +1 or -1");
  op->herm = herm;
  return QD_OK;
}
int qd_op_get_herm(const qd_op* op, int* herm) {
  CHECK(op && herm, QD_ERR_ARG, "null argument");
  *herm = op->herm;
  return QD_OK;
}
int qd_op_device_ptr(qd_op* op, double** dptr) {
  CHECK(op && dptr, QD_ERR_ARG, "null argument");
  *dptr = op->d;
  op->zero_mask = 0;  // the caller may write through the pointer
  op->exposed = true;
  return QD_OK;
}

int qd_random_operator(const qd_layout* L, int herm, uint64_t seed, double sigma, int conserve, double* v,
                       int64_t neq) {
  CHECK(L && v && neq == L->neq, QD_ERR_ARG, "qd_random_operator: bad arguments");
  CHECK(herm == 1 || herm == -1, QD_ERR_ARG, "herm must be +1 or -1");
  fill_random(L, herm, seed, sigma, conserve, v);
  return QD_OK;
}

int qd_add_arrays(const qd_op* r1, double s1, const qd_op* r2, double s2, qd_op* r3) {
  TRY(same_layout(r1, r2));
  TRY(same_layout(r1, r3));
  qd_layout* L = r1->L;
  TRY(use_device(L));
  // two generators into one that already holds zeros elsewhere (euler_step)
  if (std::isfinite(s1) && std::isfinite(s2) && gen_like(r1->zero_mask & r2->zero_mask & r3->zero_mask))
    TRY(launch_axpy_gen(L, r1->d, s1, r2->d, s2, r3->d));
  else
    TRY(launch_axpy(L, r1->d, s1, r2->d, s2, r3->d, L->neq));
  unsigned m1 = s1 == 0.0 ? ALL_PARTS | CONSERVES : r1->zero_mask, m2 = s2 == 0.0 ? ALL_PARTS | CONSERVES : r2->zero_mask;
  r3->zero_mask = m1 & m2;
  return QD_OK;
}

int qd_copy_arrays(const qd_op* r1, qd_op* r2) {
  TRY(same_layout(r1, r2));
  if (r1 == r2) return QD_OK;
  TRY(use_device(r1->L));
  QD_CUDA(cudaMemcpyAsync(r2->d, r1->d, sizeof(double) * r1->L->neq, cudaMemcpyDeviceToDevice, r1->L->stream));
  r2->zero_mask = r1->zero_mask;
  return QD_OK;
}

int qd_set_to_zero(qd_op* r1) {
  CHECK(r1, QD_ERR_ARG, "null operator");
  TRY(use_device(r1->L));
  QD_CUDA(cudaMemsetAsync(r1->d, 0, sizeof(double) * r1->L->neq, r1->L->stream));
  r1->zero_mask = ALL_PARTS | CONSERVES;
  return QD_OK;
}

int qd_mat_2_norm(const qd_op* r, double* out) {
  CHECK(r && out, QD_ERR_ARG, "null argument");
  qd_layout* L = r->L;
  TRY(use_device(L));
  TRY(reduce_norm(L, r->d, r->exposed ? 0u : r->zero_mask, red_slot(L, 0)));
  return scalar_out(L, red_slot(L, 0), out);
}

int qd_commutator_110(const qd_op* r1, const qd_op* r2, double* c) {
  TRY(same_layout(r1, r2));
  CHECK(c, QD_ERR_ARG, "null output");
  qd_layout* L = r1->L;
  TRY(use_device(L));
  TRY(reduce_dot_range(L, r1->d, r2->d, L->o_fph, (i64)L->mp * L->n, (double)(r1->herm - r2->herm), 0.0,
                       red_slot(L, 0)));
  return scalar_out(L, red_slot(L, 0), c);
}

int qd_commutator_220(const qd_op* r1, const qd_op* r2, double* c) {
  TRY(same_layout(r1, r2));
  CHECK(c, QD_ERR_ARG, "null output");
  qd_layout* L = r1->L;
  TRY(use_device(L));
  TRY(reduce_dot_part(L, r1->d, r2->d, P_PPHH, (double)(r1->herm - r2->herm), 0.0, red_slot(L, 0)));
  return scalar_out(L, red_slot(L, 0), c);
}

int qd_commutator_111(const qd_op* r1, const qd_op* r2, qd_op* r3) {
  TRY(same_layout(r1, r2));
  TRY(same_layout(r1, r3));
  TRY(use_device(r1->L));
  TRY(build_programs(r1->L));
  return stage_111(r1->L, r1, r2, r3);
}

int qd_commutator_121(const qd_op* r1, const qd_op* r2, qd_op* r3) {
  TRY(same_layout(r1, r2));
  TRY(same_layout(r1, r3));
  TRY(use_device(r1->L));
  TRY(launch_121(r1->L, r1, r2, r3->d));
  r3->zero_mask &= ~ONE_BODY & (conserves(r1, r2) ? ~0u : ~CONSERVES);
  return QD_OK;
}

int qd_commutator_221(const qd_op* r1, const qd_op* r2, qd_op* r3, qd_op* w1, qd_op* w2) {
  TRY(same_layout(r1, r2));
  TRY(same_layout(r1, r3));
  TRY(same_layout(r1, w1));
  TRY(same_layout(r1, w2));
  TRY(use_device(r1->L));
  TRY(build_programs(r1->L));
  TRY(stage_221(r1->L, r1, r2, r3, w1, w2));
  r3->zero_mask &= ~ONE_BODY;
  return QD_OK;
}

int qd_commutator_122(const qd_op* r1, const qd_op* r2, qd_op* r3) {
  TRY(same_layout(r1, r2));
  TRY(same_layout(r1, r3));
  TRY(use_device(r1->L));
  TRY(launch_122(r1->L, r1, r2, r3->d, false));
  r3->zero_mask &= ONE_BODY | CONSERVES;
  return QD_OK;
}

int qd_commutator_222(const qd_op* r1, const qd_op* r2, qd_op* r3, qd_op* w1, const qd_cc* HCC, const qd_cc* ETACC) {
  (void)w1;
  TRY(same_layout(r1, r2));
  TRY(same_layout(r1, r3));
  TRY(use_device(r1->L));
  TRY(build_programs(r1->L));
  unsigned keep = r3->zero_mask & (ONE_BODY | CONSERVES);
  TRY(stage_222(r1->L, r1, r2, r3, HCC, ETACC));
  r3->zero_mask = keep;
  return QD_OK;
}

int qd_commutator(const qd_op* A, const qd_op* B, qd_op* C, unsigned flags) {
  TRY(same_layout(A, B));
  TRY(same_layout(A, C));
  CHECK(C != A && C != B, QD_ERR_ARG, "qd_commutator: output aliases an input");
  qd_layout* L = A->L;
  TRY(use_device(L));
  Workspace* w;
  TRY(get_ws(L, &w));
  return commutator_seq(L, A, B, C, w->w1, w->w2, w->ca, w->cb, (flags & QD_PANDYA) != 0, nullptr, false);
}

// dGam (src/gs_IMSRG.f90:223-273): ETA = build_white(H) on a zeroed
// operator, HCC = calc_cc(H) (herm +1), ETACC = calc_cc(ETA) (herm -1),
// DER = [ETA, H] with every term: 110+220 into E0, 111, 121, 221, 122, 222
// with the particle-hole channel (the reference's order).
int qd_dgam(const qd_op* H, qd_op* DER, qd_cc* HCC, qd_cc* ETACC) {
  TRY(same_layout(H, DER));
  CHECK(H != DER, QD_ERR_ARG, "qd_dgam: DER aliases H");
  qd_layout* L = H->L;
  CHECK((!HCC || HCC->L == L) && (!ETACC || ETACC->L == L), QD_ERR_ARG, "qd_dgam: cross-coupled matrix of another layout");
  TRY(use_device(L));
  Workspace* w;
  TRY(get_ws(L, &w));
  if (!w->eta) TRY(op_new(L, -1, &w->eta));
  qd_op* eta = w->eta;
  eta->herm = -1;
  QD_CUDA(cudaMemsetAsync(eta->d, 0, sizeof(double) * L->neq, L->stream));
  eta->zero_mask = ALL_PARTS | CONSERVES;
  TRY(white(eta, H));
  TRY(commutator_seq(L, eta, H, DER, w->w1, w->w2, ETACC ? ETACC : w->ca, HCC ? HCC : w->cb, true, nullptr,
                     ETACC != nullptr));
  return QD_OK;
}

// EOM matrix-vector product (matvec_prod, src/EOM_IMSRG.f90:551-649, with
// HQ_comm_1b/2b, src/commutators.f90:1162-1272) for the scalar target
// (M_L, M_S) = (0, 0): the particle-hole and pphh parts of [H, Q] for the
// excitation operator Q (its fph and Vpphh).  The layout stores each
// operator with herm = +-1, so Q = (Q+ + Q-)/2, Q+- the same amplitudes as
// herm +-1 operators, and [H, Q] is the average of two full commutators with
// the particle-hole channel; every other part of HQ is zero.
int qd_eom_matvec(const qd_op* H, const qd_op* Q, qd_op* HQ) {
  TRY(same_layout(H, Q));
  TRY(same_layout(H, HQ));
  CHECK(HQ != H && HQ != Q, QD_ERR_ARG, "qd_eom_matvec: HQ aliases an input");
  qd_layout* L = H->L;
  TRY(use_device(L));
  Workspace* w;
  TRY(get_ws(L, &w));
  if (!w->eomq) TRY(op_new(L, 1, &w->eomq));
  if (!w->eomt) TRY(op_new(L, 1, &w->eomt));
  const unsigned exc = (1u << P_FPH) | (1u << P_PPHH);
  qd_op* X = w->eomq;
  QD_CUDA(cudaMemcpyAsync(X->d, Q->d, sizeof(double) * L->neq, cudaMemcpyDeviceToDevice, L->stream));
  TRY(launch_keep_parts(L, X->d, exc));
  X->zero_mask = (ALL_PARTS & ~exc) | (Q->zero_mask & (exc | CONSERVES));
  X->herm = 1;
  TRY(commutator_seq(L, H, X, HQ, w->w1, w->w2, w->cb, w->ca, true, nullptr, false));
  X->herm = -1;
  TRY(commutator_seq(L, H, X, w->eomt, w->w1, w->w2, w->cb, w->ca, true, nullptr, false));
  TRY(launch_axpy(L, HQ->d, 0.5, w->eomt->d, 0.5, HQ->d, L->neq));
  TRY(launch_keep_parts(L, HQ->d, exc));
  HQ->herm = 1;
  HQ->zero_mask = (ALL_PARTS & ~exc) | conserves(H, X);
  return QD_OK;
}

int qd_cc_create(qd_layout* L, double herm, qd_cc** out) {
  CHECK(L && out, QD_ERR_ARG, "null argument");
  TRY(use_device(L));
  return cc_new(L, herm, out);
}
int qd_cc_destroy(qd_cc* cc) {
  if (!cc) return QD_OK;
  cudaSetDevice(cc->L->device);
  cudaStreamSynchronize(cc->L->stream);
  cc_free(cc);
  (void)cudaGetLastError();
  return QD_OK;
}
int qd_cc_set_herm(qd_cc* cc, double herm) {
  CHECK(cc, QD_ERR_ARG, "null cc");
  cc->herm = herm;
  return QD_OK;
}
int qd_calc_cc(const qd_op* H, qd_cc* HCC) {
  CHECK(H && HCC && H->L == HCC->L, QD_ERR_ARG, "qd_calc_cc: bad arguments");
  TRY(use_device(H->L));
  TRY(launch_calc_cc(H->L, H, HCC->d));
  HCC->filled = true;
  return QD_OK;
}
int qd_cc_download(const qd_cc* cc, double* host, int64_t n, int64_t* needed) {
  CHECK(cc, QD_ERR_ARG, "null cc");
  if (needed) *needed = cc->L->xsize;
  if (!host) return QD_OK;
  CHECK(n >= cc->L->xsize, QD_ERR_ARG, "qd_cc_download: buffer too small");
  const qd_layout* L = cc->L;
  TRY(use_device(L));
  if (L->xsize == 0) return QD_OK;
  // device rows are group-major; the host gets the reference's (i, j) row order
  std::vector<double> tmp((size_t)L->xsize);
  QD_CUDA(cudaMemcpyAsync(tmp.data(), cc->d, sizeof(double) * L->xsize, cudaMemcpyDeviceToHost, L->stream));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  for (int q = 0; q < L->ncc; ++q) {
    const int r = L->ccdim[q].x, nb = L->ccdim[q].y, rb = L->ccab_base[q];
    const i64 xo = L->ccxoff[q];
    for (int c = 0; c < nb; ++c)
      for (int t = 0; t < r; ++t) host[xo + L->ccref[rb + t] + (i64)c * r] = tmp[xo + t + (i64)c * r];
  }
  return QD_OK;
}

int qd_build_white(qd_op* gen, const qd_op* H) {
  TRY(same_layout(gen, H));
  TRY(use_device(H->L));
  return white(gen, H);
}

int qd_mbpt2(const qd_op* H, double* out) {
  CHECK(H && out, QD_ERR_ARG, "null argument");
  TRY(use_device(H->L));
  TRY(reduce_mbpt2(H->L, H->d, red_slot(H->L, 0)));
  return scalar_out(H->L, red_slot(H->L, 0), out);
}

int qd_hf_e2(qd_op* H, double* out) {
  CHECK(H, QD_ERR_ARG, "null operator");
  qd_layout* L = H->L;
  TRY(use_device(L));
  double tr;
  TRY(reduce_hhtrace(L, H->d, red_slot(L, 0)));
  TRY(scalar_out(L, red_slot(L, 0), &tr));
  double sm2 = 0.0;
  for (int i = 0; i < L->n; ++i) sm2 = sm2 + L->eig[i];
  double e = sm2 - tr;
  QD_CUDA(cudaMemcpyAsync(H->d, &e, sizeof(double), cudaMemcpyHostToDevice, L->stream));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  if (out) *out = e;
  return QD_OK;
}

// ---- one BCH term, replayed as a CUDA graph --------------------------------
// A term is INT2 = [G, AD], HS += cof INT2 with |HS| and |INT2| into
// red_slot(1) and their copy to h_red[1..2].  Its launches depend only on the
// buffers, the zero-part masks, herm, the flags, the slice count and cof, so
// a term seen before on the same key is captured once (thread-local capture
// mode, after an eager run has built every plan and workspace) and replayed
// with one cudaGraphLaunch.  A capture that fails leaves the key eager.
namespace {
struct TermKey {
  const void* p[9];  // G, AD, INT2, HS, w1, w2, OCC, HCC, source of HS
  unsigned mg, mad, mhs;
  int gh, term, flags, split;
  bool operator<(const TermKey& o) const { return std::memcmp(this, &o, sizeof(TermKey)) < 0; }
};
struct TermGraph {
  int seen = 0;
  bool failed = false;
  cudaGraphExec_t exec = nullptr;
  long long launches = 0;
};
using TermGraphs = std::map<TermKey, TermGraph>;

// HS = src + cof [G, AD]: src is HS, or for the first term H (= AD).
int bch_term(qd_layout* L, const qd_op* G, const qd_op* AD, qd_op* INT2, const qd_op* src, qd_op* HS, qd_op* w1,
             qd_op* w2, qd_cc* HCC, qd_cc* OCC, bool pandya, bool first, double cof, int* kidx = nullptr, const BchDecide& dec = BchDecide{}) {
  HsUpdate upd;
  const bool split = splits_update(L, G);
  if (split) TRY(hs_update_begin(L, src->d, HS->d, cof, kidx, &upd));
  TRY(commutator_seq(L, G, AD, INT2, w1, w2, pandya ? OCC : nullptr, pandya ? HCC : nullptr, pandya,
                     split ? &upd : nullptr, first));  // Omega's matrices once a series
  {
    StageTimer tm(L, S_GLUE);
    if (split)
      TRY(launch_axpy_norms_rest(L, INT2->d, upd, red_slot(L, 1), dec));
    else
      TRY(launch_axpy_norms(L, src->d, 1.0, INT2->d, cof, HS->d, red_slot(L, 1), kidx, dec));
  }
  if (!kidx)  // host decides: copy both norms back
    QD_CUDA(cudaMemcpyAsync(L->h_red + 1, red_slot(L, 1), 2 * sizeof(double), cudaMemcpyDeviceToHost, L->stream));
  return QD_OK;
}
}  // namespace

static int bch_term_graph(qd_layout* L, const qd_op* G, const qd_op* AD, qd_op* INT2, const qd_op* src, qd_op* HS,
                          qd_op* w1, qd_op* w2, qd_cc* HCC, qd_cc* OCC, bool pandya, int term, double cof) {
  if (!L->use_graphs || L->prof.on) return bch_term(L, G, AD, INT2, src, HS, w1, w2, HCC, OCC, pandya, term == 2, cof);
  if (!L->graphs) L->graphs = new TermGraphs();
  TermKey k;
  std::memset(&k, 0, sizeof(k));
  k.p[0] = G->d;
  k.p[1] = AD->d;
  k.p[2] = INT2->d;
  k.p[3] = HS->d;
  k.p[4] = w1->d;
  k.p[5] = w2->d;
  k.p[6] = OCC ? OCC->d : nullptr;
  k.p[7] = HCC ? HCC->d : nullptr;
  k.p[8] = src->d;
  k.mg = G->zero_mask;
  k.mad = AD->zero_mask;
  k.mhs = HS->zero_mask;
  k.gh = G->herm;
  k.term = term;
  k.flags = pandya ? 1 : 0;
  k.split = L->split_slices;
  TermGraph& tg = (*reinterpret_cast<TermGraphs*>(L->graphs))[k];
  if (tg.exec) {
    QD_CUDA(cudaGraphLaunch(tg.exec, L->stream));
    L->nlaunch += tg.launches;
    ++L->graph_replays;
    INT2->zero_mask = conserves(G, AD);  // what the captured commutator_seq leaves on the host side
    if (pandya) {
      OCC->filled = true;
      OCC->herm = G->herm;
      HCC->filled = true;
      HCC->herm = AD->herm;
    }
    return QD_OK;
  }
  if (tg.failed || tg.seen == 0) {
    ++tg.seen;
    return bch_term(L, G, AD, INT2, src, HS, w1, w2, HCC, OCC, pandya, term == 2, cof);
  }
  // second sight: capture, instantiate, launch
  const long long n0 = L->nlaunch;
  cudaGraph_t graph = nullptr;
  int rc = QD_OK;
  cudaError_t e = cudaStreamBeginCapture(L->stream, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    rc = bch_term(L, G, AD, INT2, src, HS, w1, w2, HCC, OCC, pandya, term == 2, cof);
    e = cudaStreamEndCapture(L->stream, &graph);
  }
  if (e == cudaSuccess && rc == QD_OK && graph) e = cudaGraphInstantiate(&tg.exec, graph, 0);
  if (graph) cudaGraphDestroy(graph);
  if (e != cudaSuccess || rc != QD_OK || !tg.exec) {
    (void)cudaGetLastError();
    if (tg.exec) cudaGraphExecDestroy(tg.exec);
    tg.exec = nullptr;
    tg.failed = true;
    L->nlaunch = n0;
    return bch_term(L, G, AD, INT2, src, HS, w1, w2, HCC, OCC, pandya, term == 2, cof);
  }
  tg.launches = L->nlaunch - n0;
  ++L->graphs_captured;
  QD_CUDA(cudaGraphLaunch(tg.exec, L->stream));
  return QD_OK;
}

}  // extern "C"

namespace {
// ---- a whole BCH_EXPAND as one CUDA graph --------------------------------
// The exit test runs on the device (k_bch_decide), so the term loop is a
// graph "while" node and a BCH step needs one host synchronisation (for the
// term count) instead of one per term.  Layout of the graph:
//   prologue: INT2 = [G, H]; HS = H + cof(1) INT2; decide
//   while (go): INT2' = [G, INT2]; HS += cof INT2'; decide (sets go, more)
//               if (more): INT2 = [G, INT2']; HS += cof INT2; decide (sets go)
// The two buffers of INT2 and AD alternate between the two halves of the
// loop body, so no operator is copied.  The term coefficient comes from a
// device counter (the number of terms so far), which the host reads back.
// Built like the per-term graphs: a key seen once runs eagerly (which builds
// every plan and workspace), the second time it is captured; a capture that
// fails leaves the key eager.
struct StepKey {
  const void* p[9];  // G, HS, H, INT2, AD, w1, w2, OCC, HCC data
  unsigned mg, mh;
  int gh, hh, flags, split;
  bool operator<(const StepKey& o) const { return std::memcmp(this, &o, sizeof(StepKey)) < 0; }
};
struct StepGraph {
  int seen = 0;
  bool failed = false;
  cudaGraphExec_t exec = nullptr;
  long long first = 0, per_term = 0;  // launches of the prologue and of one later term
};
using StepGraphs = std::map<StepKey, StepGraph>;

// Whether the first term can read H in place of copies in AD and HS: H is
// none of the buffers written, and Hermitian as BCH_EXPAND takes AD to be.
bool reads_h(const qd_op* H, const qd_op* HS, const double* P, const double* Q) {
  return H->herm == 1 && H->d != HS->d && H->d != P && H->d != Q;
}

int* bch_counter(qd_layout* L) { return reinterpret_cast<int*>(red_slot(L, 16)); }

// A conditional node of `type` on handle h after the current dependencies of
// a stream capturing into graph g; *body receives its body graph.
int add_conditional(cudaStream_t st, cudaGraph_t g, cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type,
                    cudaGraph_t* body) {
  cudaStreamCaptureStatus cs;
  const cudaGraphNode_t* deps = nullptr;
  size_t nd = 0;
  QD_CUDA(cudaStreamGetCaptureInfo(st, &cs, nullptr, nullptr, &deps, &nd));
  cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};  // aggregate: the rest zero
  cp.conditional.handle = h;
  cp.conditional.type = type;
  cp.conditional.size = 1;
  cudaGraphNode_t node;
  QD_CUDA(cudaGraphAddNode(&node, g, deps, nd, &cp));
  QD_CUDA(cudaStreamUpdateCaptureDependencies(st, &node, 1, cudaStreamSetCaptureDependencies));
  *body = cp.conditional.phGraph_out[0];
  return QD_OK;
}

// Capture the step graph: P (INT2's buffer) and Q (AD's buffer) alternate.
int capture_step(qd_layout* L, qd_op* HS, const qd_op* G, const qd_op* H, double* P, double* Q, qd_op* w1,
                 qd_op* w2, qd_cc* HCC, qd_cc* OCC, bool pandya, cudaGraphExec_t* exec, long long* first,
                 long long* per_term) {
  const double conv = (double)1e-5f;
  int* k = bch_counter(L);
  cudaStream_t st = L->stream;
  qd_op ad = *H, out = *H;  // host views of the two buffers (herm +1, as BCH_EXPAND sets)
  ad.herm = out.herm = 1;
  ad.exposed = out.exposed = false;
  cudaGraph_t g = nullptr;
  QD_CUDA(cudaGraphCreate(&g, 0));
  int rc = QD_OK;
  cudaGraph_t body = nullptr, body2 = nullptr, cap = nullptr;
  cudaGraphConditionalHandle hloop, hmore;
  const long long n0 = L->nlaunch;
  do {
    if (cudaGraphConditionalHandleCreate(&hloop, g, 0, 0) != cudaSuccess) { rc = QD_ERR_CUDA; break; }
    if (cudaStreamBeginCaptureToGraph(st, g, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      rc = QD_ERR_CUDA;
      break;
    }
    // prologue: term 1 into P, of H itself unless that is one of the buffers
    const bool direct = reads_h(H, HS, P, Q);
    int r2 = QD_OK;
    if (cudaMemsetAsync(k, 0, sizeof(int), st) != cudaSuccess ||
        (!direct && (cudaMemcpyAsync(HS->d, H->d, sizeof(double) * L->neq, cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
                     cudaMemcpyAsync(Q, H->d, sizeof(double) * L->neq, cudaMemcpyDeviceToDevice, st) != cudaSuccess)))
      r2 = QD_ERR_CUDA;
    ad.d = direct ? H->d : Q;
    ad.zero_mask = H->zero_mask;
    out.d = P;
    HS->zero_mask = H->zero_mask;
    if (!r2)
      r2 = bch_term(L, G, &ad, &out, direct ? &ad : HS, HS, w1, w2, HCC, OCC, pandya, true, 0.0, k,
                    BchDecide{hloop, hloop, 1, 0, conv});
    *first = L->nlaunch - n0;
    if (!r2) r2 = add_conditional(st, g, hloop, cudaGraphCondTypeWhile, &body);
    if (cudaStreamEndCapture(st, &cap) != cudaSuccess || r2) {
      rc = r2 ? r2 : QD_ERR_CUDA;
      break;
    }
    // loop body, first half: AD = P, INT2 = Q; then "more" guards the second half
    if (cudaGraphConditionalHandleCreate(&hmore, body, 0, 0) != cudaSuccess ||
        cudaStreamBeginCaptureToGraph(st, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      rc = QD_ERR_CUDA;
      break;
    }
    const long long n1 = L->nlaunch;
    ad.d = P;
    ad.zero_mask = conserves(G, H);
    out.d = Q;
    r2 = bch_term(L, G, &ad, &out, HS, HS, w1, w2, HCC, OCC, pandya, false, 0.0, k, BchDecide{hloop, hmore, 1, 1, conv});
    *per_term = L->nlaunch - n1;
    if (!r2) r2 = add_conditional(st, body, hmore, cudaGraphCondTypeIf, &body2);
    if (cudaStreamEndCapture(st, &cap) != cudaSuccess || r2) {
      rc = r2 ? r2 : QD_ERR_CUDA;
      break;
    }
    // second half: AD = Q, INT2 = P
    if (cudaStreamBeginCaptureToGraph(st, body2, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal) !=
        cudaSuccess) {
      rc = QD_ERR_CUDA;
      break;
    }
    ad.d = Q;
    out.d = P;
    r2 = bch_term(L, G, &ad, &out, HS, HS, w1, w2, HCC, OCC, pandya, false, 0.0, k, BchDecide{hloop, hloop, 1, 0, conv});
    if (cudaStreamEndCapture(st, &cap) != cudaSuccess || r2) {
      rc = r2 ? r2 : QD_ERR_CUDA;
      break;
    }
    if (cudaGraphInstantiate(exec, g, 0) != cudaSuccess) rc = QD_ERR_CUDA;
  } while (false);
  if (rc) {  // leave no capture open and no error pending
    cudaStreamCaptureStatus cs;
    if (cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
      cudaGraph_t junk = nullptr;
      cudaStreamEndCapture(st, &junk);
      if (junk) cudaGraphDestroy(junk);
    }
    (void)cudaGetLastError();
    *exec = nullptr;
  }
  cudaGraphDestroy(g);
  L->nlaunch = n0;
  return rc;
}

// The eager BCH_EXPAND loop (per-term graphs where enabled).
int bch_eager(qd_layout* L, qd_op* HS, const qd_op* G, const qd_op* H, qd_op* INT2, qd_op* AD, qd_op* w1, qd_op* w2,
              qd_cc* HCC, qd_cc* OCC, bool pandya, int* nterms);

// Launch the whole step as a graph when possible (bch_step_finish waits for
// it); *launched = false leaves it to the caller.
int bch_step_launch(qd_layout* L, qd_op* HS, const qd_op* G, const qd_op* H, qd_op* INT2, qd_op* AD, qd_op* w1,
                    qd_op* w2, qd_cc* HCC, qd_cc* OCC, bool pandya, bool* launched) {
  *launched = false;
  if (!L->use_graphs || L->prof.on || L->split_slices > 0) return QD_OK;
  if (!L->step_graphs) L->step_graphs = new StepGraphs();
  StepKey key;
  std::memset(&key, 0, sizeof(key));
  const void* ptrs[9] = {G->d, HS->d, H->d, INT2->d, AD->d, w1->d, w2->d, OCC ? OCC->d : nullptr,
                         HCC ? HCC->d : nullptr};
  for (int i = 0; i < 9; ++i) key.p[i] = ptrs[i];
  key.mg = G->zero_mask;
  key.mh = H->zero_mask;
  key.gh = G->herm;
  key.hh = H->herm;
  key.flags = pandya ? 1 : 0;
  key.split = L->split_slices;
  StepGraph& sg = (*reinterpret_cast<StepGraphs*>(L->step_graphs))[key];
  double* P = INT2->d;
  double* Q = AD->d;
  if (!sg.exec) {
    if (sg.failed || sg.seen++ == 0) return QD_OK;  // eager (first sight builds plans for H's masks)
    // plans and task lists of the later terms ([G, X] with X a full operator)
    qd_op full = *H;  // H as a full operator: the masks of AD in the later terms
    full.zero_mask = conserves(G, H);
    TRY(prepare_program(L, ladder_program(L, G), G->zero_mask, full.zero_mask));
    TRY(prepare_program(L, L->prog_111, G->zero_mask, full.zero_mask));
    TRY(prepare_program(L, L->prog_pandya, 0u, 0u));
    TRY(prepare_onebody(L));
    TRY(prepare_hs_update(L));
    if (!L->ev_fork) TRY(make_branches(L));
    TRY(prepare_122(L, G, &full));
    TRY(prepare_program(L, ladder_program(L, G), G->zero_mask, H->zero_mask));
    TRY(prepare_program(L, L->prog_111, G->zero_mask, H->zero_mask));
    TRY(prepare_122(L, G, H));
    if (pandya) TRY(gen_like(G->zero_mask) ? prepare_ph_gen(L) : ensure_z(L));
    QD_CUDA(cudaStreamSynchronize(L->stream));
    if (capture_step(L, HS, G, H, P, Q, w1, w2, HCC, OCC, pandya, &sg.exec, &sg.first, &sg.per_term)) {
      sg.failed = true;
      return QD_OK;
    }
    ++L->graphs_captured;
  }
  QD_CUDA(cudaGraphLaunch(sg.exec, L->stream));
  int* hk = reinterpret_cast<int*>(L->h_red + 16);
  QD_CUDA(cudaMemcpyAsync(hk, bch_counter(L), sizeof(int), cudaMemcpyDeviceToHost, L->stream));
  L->step_first = sg.first;
  L->step_per_term = sg.per_term;
  *launched = true;
  return QD_OK;
}

// Wait for a launched step and leave the host-side state of the eager loop:
// HS and the workspaces hold full operators, the two workspace buffers keep
// their handles.
int bch_step_finish(qd_layout* L, qd_op* HS, const qd_op* G, const qd_op* H, qd_op* INT2, qd_op* AD, qd_cc* HCC,
                    qd_cc* OCC, bool pandya, int* nterms) {
  QD_CUDA(cudaStreamSynchronize(L->stream));
  const int terms = *reinterpret_cast<int*>(L->h_red + 16);
  L->nlaunch += L->step_first + L->step_per_term * (terms - 1);
  ++L->graph_replays;
  HS->zero_mask = INT2->zero_mask = AD->zero_mask = conserves(G, H);
  if (pandya) {
    OCC->filled = true;
    OCC->herm = G->herm;
    HCC->filled = true;
    HCC->herm = 1;
  }
  *nterms = terms;
  return QD_OK;
}

}  // namespace

extern "C" {

int qd_bch_expand(qd_op* HS, const qd_op* G, const qd_op* H, qd_op* INT1, qd_op* INT2, qd_op* AD, qd_op* w1,
                  qd_op* w2, qd_cc* HCC, qd_cc* OCC, unsigned flags, int* nterms) {
  TRY(same_layout(HS, G));
  TRY(same_layout(HS, H));
  TRY(same_layout(HS, INT2));
  TRY(same_layout(HS, AD));
  TRY(same_layout(HS, w1));
  TRY(same_layout(HS, w2));
  (void)INT1;  // not written: the norm of INT1 (= HS before the update) is taken from HS itself
  qd_layout* L = HS->L;
  TRY(use_device(L));
  TRY(build_programs(L));
  const bool pandya = (flags & QD_PANDYA) != 0;
  CHECK(!pandya || (HCC && OCC), QD_ERR_ARG, "qd_bch_expand: QD_PANDYA needs HCC and OCC");
  INT2->herm = 1;
  AD->herm = 1;
  bool done = false;
  int count = 0;
  TRY(bch_step_launch(L, HS, G, H, INT2, AD, w1, w2, HCC, OCC, pandya, &done));
  if (done)
    TRY(bch_step_finish(L, HS, G, H, INT2, AD, HCC, OCC, pandya, &count));
  else
    TRY(bch_eager(L, HS, G, H, INT2, AD, w1, w2, HCC, OCC, pandya, &count));
  if (nterms) *nterms = count;
  return QD_OK;
}

}  // extern "C"

namespace {
int bch_eager(qd_layout* L, qd_op* HS, const qd_op* G, const qd_op* H, qd_op* INT2, qd_op* AD, qd_op* w1, qd_op* w2,
              qd_cc* HCC, qd_cc* OCC, bool pandya, int* nterms) {
  const double conv = (double)1e-5f;  // "conv = 1e-5" is a real(4) literal in the reference
  double* const p0 = INT2->d;
  const bool direct = reads_h(H, HS, INT2->d, AD->d);
  if (!direct) {
    TRY(qd_copy_arrays(H, HS));
    TRY(qd_copy_arrays(H, INT2));
  }
  HS->zero_mask = H->zero_mask;
  int count = 0;
  for (int i = 2; i <= 12; ++i) {
    swap_ops(INT2, AD);  // AD = previous term; INT2 becomes the output buffer
    const double cof = kCof[i - 2];
    const bool first = direct && i == 2;
    TRY(bch_term_graph(L, G, first ? H : AD, INT2, first ? H : HS, HS, w1, w2, HCC, OCC, pandya, i, cof));
    ++count;
    HS->zero_mask &= INT2->zero_mask;
    QD_CUDA(cudaStreamSynchronize(L->stream));
    const double n1 = L->h_red[1], n2 = L->h_red[2];
    if (n2 * cof / n1 < conv) break;
  }
  if (INT2->d != p0) {  // the workspaces keep their buffers (contents unspecified)
    swap_ops(INT2, AD);
  }
  if (nterms) *nterms = count;
  return QD_OK;
}
}  // namespace

extern "C" {

int qd_magnus_expand(qd_op* DG, const qd_op* G, const qd_op* ETA) {
  (void)G;
  return qd_copy_arrays(ETA, DG);
}

int qd_euler_step(qd_op* G, const qd_op* DG, double* s, double stp) {
  TRY(qd_add_arrays(G, 1.0, DG, stp, G));
  if (s) *s = *s + stp;
  return QD_OK;
}

}  // extern "C"

// ---- the Magnus flow as a stepping object (s_evolve, magnus_IMSRG.f90:194-248)
struct qd_flow {
  qd_layout* L = nullptr;
  const qd_op* HAM = nullptr;
  qd_op* HS = nullptr;
  double* hs_home = nullptr;  // the caller's HS buffer (HS and HS0 trade buffers during the flow)
  unsigned flags = 0;
  qd_op *ETA = nullptr, *G = nullptr, *DG = nullptr, *ETA0 = nullptr, *G0 = nullptr, *HS0 = nullptr;
  qd_op *INT1 = nullptr, *INT2 = nullptr, *AD = nullptr, *w1 = nullptr, *w2 = nullptr;
  qd_cc *HCC = nullptr, *OCC = nullptr;
  double s = 0.0, stp = (double)0.7f;  // "stp=.7" is a real(4) literal
  double nrm1 = 0.0, crit = 0.0, E0 = 0.0;
  int iteration = 0, rejected = 0, comms = 0, rows = 0;
};

namespace {
const double kConvCriteria = (double)1e-9f;  // real(4) literal in the reference

int flow_eta_norm(qd_flow* f, const qd_op* op, double* out) { return qd_mat_2_norm(op, out); }

// Give the caller's HS its own buffer back (copying the current contents).
int flow_home_hs(qd_flow* f) {
  if (f->HS->d == f->hs_home) return QD_OK;
  QD_CUDA(cudaMemcpyAsync(f->hs_home, f->HS->d, sizeof(double) * f->L->neq, cudaMemcpyDeviceToDevice, f->L->stream));
  const unsigned zero = f->HS->zero_mask;
  swap_ops(f->HS, f->HS0);  // HS0 held hs_home: after the swap HS->d == hs_home again
  f->HS->zero_mask = f->HS0->zero_mask = zero;  // both buffers hold HS now
  return QD_OK;
}

int flow_e0(qd_flow* f, double* e0) {
  qd_layout* L = f->L;
  QD_CUDA(cudaMemcpyAsync(L->h_red + 8, f->HS->d, sizeof(double), cudaMemcpyDeviceToHost, L->stream));
  QD_CUDA(cudaStreamSynchronize(L->stream));
  *e0 = L->h_red[8];
  return QD_OK;
}
}  // namespace

extern "C" {

int qd_flow_create(const qd_op* HAM, qd_op* HS, unsigned flags, qd_flow** out) {
  CHECK(out, QD_ERR_ARG, "qd_flow_create: null output");
  *out = nullptr;
  TRY(same_layout(HAM, HS));
  CHECK(HAM != HS, QD_ERR_ARG, "qd_flow_create: HS must not alias HAM");
  qd_layout* L = HAM->L;
  TRY(use_device(L));
  // workspaces: allocated by the first flow on this layout and kept (they
  // hold 11 operators; freeing them per flow would cost a device sync each)
  Workspace* ws;
  {
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    ws = &workspaces()[L];
  }
  const int fherm[11] = {-1, -1, -1, -1, -1, 1, 1, 1, 1, 1, 1};
  for (int k = 0; k < 11; ++k)
    if (!ws->flow[k]) TRY(op_new(L, fherm[k], &ws->flow[k]));
  if (!ws->flow_cc[0]) TRY(cc_new(L, 1.0, &ws->flow_cc[0]));
  if (!ws->flow_cc[1]) TRY(cc_new(L, -1.0, &ws->flow_cc[1]));
  qd_flow* f = new qd_flow();
  f->L = L;
  f->HAM = HAM;
  f->HS = HS;
  f->flags = flags;
  qd_op** o = ws->flow;
  f->ETA = o[0]; f->G = o[1]; f->DG = o[2]; f->ETA0 = o[3]; f->G0 = o[4]; f->HS0 = o[5];
  f->INT1 = o[6]; f->INT2 = o[7]; f->AD = o[8]; f->w1 = o[9]; f->w2 = o[10];
  f->HCC = ws->flow_cc[0];
  f->OCC = ws->flow_cc[1];
  for (int k = 0; k < 11; ++k) o[k]->herm = fherm[k];
  f->HCC->herm = 1.0;
  f->OCC->herm = -1.0;
  f->HCC->filled = f->OCC->filled = false;  // run_magnus never fills them (the Pandya option does, per commutator)
  f->hs_home = HS->d;
  int rc = QD_OK;
  // the generator and the Magnus operator start from zero (allocate_everything);
  // ETA0 too, as ETA and ETA0 trade buffers and build_white writes only fph
  // and Vpphh
  for (qd_op* z : {f->ETA, f->ETA0, f->G}) {
    if (cudaMemsetAsync(z->d, 0, sizeof(double) * L->neq, L->stream) != cudaSuccess) rc = QD_ERR_CUDA;
    z->zero_mask = ALL_PARTS | CONSERVES;
  }
  if (!rc) rc = qd_copy_arrays(HAM, HS);
  HS->herm = 1;
  if (!rc) rc = white(f->ETA, HS);
  if (!rc) rc = flow_eta_norm(f, f->ETA, &f->nrm1);
  if (!rc) rc = qd_mbpt2(HAM, &f->crit);
  if (!rc) rc = flow_e0(f, &f->E0);
  if (rc) {
    delete f;
    return rc;
  }
  f->crit = std::fabs(f->crit);
  *out = f;
  return QD_OK;
}

int qd_flow_warm_start(qd_flow* f, const qd_op* G, double s) {
  CHECK(f && G, QD_ERR_ARG, "qd_flow_warm_start: null argument");
  CHECK(G->L == f->L, QD_ERR_ARG, "qd_flow_warm_start: Omega on another layout");
  CHECK(G != f->G, QD_ERR_ARG, "qd_flow_warm_start: pass a copy of the flow's own Omega");
  TRY(use_device(f->L));
  TRY(qd_copy_arrays(G, f->G));
  f->G->herm = -1;
  f->s = s;
  int terms = 0;
  TRY(qd_bch_expand(f->HS, f->G, f->HAM, f->INT1, f->INT2, f->AD, f->w1, f->w2, f->HCC, f->OCC, f->flags, &terms));
  f->comms += terms;
  TRY(white(f->ETA, f->HS));
  double mb;
  TRY(qd_mbpt2(f->HS, &mb));
  f->crit = std::fabs(mb);
  TRY(flow_e0(f, &f->E0));
  CHECK(std::isfinite(f->E0) && std::isfinite(f->crit), QD_ERR_NAN, "qd_flow_warm_start: non-finite state");
  return QD_OK;
}

}  // extern "C"

namespace {
// s_evolve's loop body in two halves around BCH_EXPAND (the batched flows run
// the BCH of several instances between them).  flow_begin returns
// *converged = true (and fills info) when there is nothing to do.
int flow_begin(qd_flow* f, qd_flow_step_info* inf, bool* converged) {
  std::memset(inf, 0, sizeof(*inf));
  *converged = f->crit <= kConvCriteria;
  if (*converged) {
    inf->s = f->s;
    inf->E0 = f->E0;
    inf->nrm1 = f->nrm1;
    inf->crit = f->crit;
    inf->converged = 1;
    return QD_OK;
  }
  // G0 = G; MAGNUS_EXPAND: DG = ETA; euler_step: G = G + stp DG.  G and G0
  // trade buffers and G = 1 G0 + stp ETA is written in one pass (the same
  // arithmetic as add_arrays(G, 1, DG, stp, G) with DG = ETA).
  swap_ops(f->G, f->G0);
  TRY(qd_add_arrays(f->G0, 1.0, f->ETA, f->stp, f->G));
  f->s = f->s + f->stp;
  swap_ops(f->HS, f->HS0);  // HS0 = HS: BCH_EXPAND rewrites every entry of HS
  return QD_OK;
}

int flow_end_launch(qd_flow* f) {
  swap_ops(f->ETA, f->ETA0);  // ETA0 = ETA: build_white rewrites fph and Vpphh, the rest stays 0
  TRY(white(f->ETA, f->HS));
  // |ETA|, MBPT2 (used if the step is accepted) and E0 in one synchronisation
  qd_layout* L = f->L;
  TRY(reduce_norm(L, f->ETA->d, f->ETA->exposed ? 0u : f->ETA->zero_mask, red_slot(L, 4)));
  TRY(reduce_mbpt2(L, f->HS->d, red_slot(L, 5)));
  QD_CUDA(cudaMemcpyAsync(L->h_red + 4, red_slot(L, 4), 2 * sizeof(double), cudaMemcpyDeviceToHost, L->stream));
  QD_CUDA(cudaMemcpyAsync(L->h_red + 8, f->HS->d, sizeof(double), cudaMemcpyDeviceToHost, L->stream));
  return QD_OK;
}

int flow_end_finish(qd_flow* f, int terms, qd_flow_step_info* inf) {
  qd_layout* L = f->L;
  f->comms += terms;
  QD_CUDA(cudaStreamSynchronize(L->stream));
  const double nrm2 = L->h_red[4], mb = L->h_red[5], E0 = L->h_red[8];
  CHECK(std::isfinite(E0) && std::isfinite(nrm2), QD_ERR_NAN,
        "qd_flow_step: non-finite energy or generator norm at s = %g", f->s);
  inf->s = f->s;
  inf->E0 = E0;
  inf->nrm1 = f->nrm1;
  inf->nrm2 = nrm2;
  inf->crit = f->crit;  // the criterion before this step, as the reference's trace
  inf->terms = terms;
  ++f->rows;
  if (f->nrm1 * 1.5 < nrm2) {  // reject: back to the previous state, smaller step
    ++f->rejected;
    f->s = f->s - f->stp;
    swap_ops(f->G, f->G0);
    swap_ops(f->HS, f->HS0);
    swap_ops(f->ETA, f->ETA0);
    f->stp = f->stp / 2.0 + (double)1e-3f;
    inf->accepted = 0;
  } else {
    f->crit = std::fabs(mb);
    f->E0 = E0;
    f->iteration += 1;
    inf->accepted = 1;
  }
  inf->converged = f->crit <= kConvCriteria ? 1 : 0;
  return QD_OK;
}
}  // namespace

extern "C" {

int qd_flow_step(qd_flow* f, qd_flow_step_info* info) {
  CHECK(f, QD_ERR_ARG, "qd_flow_step: null flow");
  TRY(use_device(f->L));
  qd_flow_step_info inf;
  bool conv = false;
  TRY(flow_begin(f, &inf, &conv));
  if (!conv) {
    int terms = 0;
    TRY(qd_bch_expand(f->HS, f->G, f->HAM, f->INT1, f->INT2, f->AD, f->w1, f->w2, f->HCC, f->OCC, f->flags,
                      &terms));
    TRY(flow_end_launch(f));
    TRY(flow_end_finish(f, terms, &inf));
  }
  if (info) *info = inf;
  return QD_OK;
}

int qd_flow_omega(const qd_flow* f, qd_op** G) {
  CHECK(f && G, QD_ERR_ARG, "qd_flow_omega: null argument");
  *G = f->G;
  return QD_OK;
}

int qd_flow_state(const qd_flow* f, qd_flow_result* r) {
  CHECK(f && r, QD_ERR_ARG, "qd_flow_state: null argument");
  r->E0 = f->E0;
  r->s = f->s;
  r->iterations = f->iteration;
  r->rejected = f->rejected;
  r->commutators = f->comms;
  r->rows = f->rows;
  return QD_OK;
}

int qd_flow_destroy(qd_flow* f) {
  if (!f) return QD_OK;
  cudaSetDevice(f->L->device);
  flow_home_hs(f);
  cudaStreamSynchronize(f->L->stream);
  (void)cudaGetLastError();
  delete f;  // the workspaces stay with the layout
  return QD_OK;
}

int qd_magnus_flow(const qd_op* HAM, qd_op* HS, unsigned flags, int max_iter, double* trace,
                   qd_flow_result* result) {
  qd_flow* f = nullptr;
  TRY(qd_flow_create(HAM, HS, flags, &f));
  int rc = QD_OK, loops = 0;
  while (f->crit > kConvCriteria) {
    if (loops++ >= max_iter) {
      qd::set_error("qd_magnus_flow: not converged after %d steps (crit %.3e)", max_iter, f->crit);
      rc = QD_ERR_NOCONV;
      break;
    }
    qd_flow_step_info inf;
    if ((rc = qd_flow_step(f, &inf))) break;
    const int row = f->rows - 1;
    if (trace && row < max_iter) {
      double* t = trace + 7 * row;
      t[0] = f->iteration - inf.accepted; t[1] = inf.s; t[2] = inf.E0; t[3] = inf.nrm1; t[4] = inf.nrm2;
      t[5] = inf.crit; t[6] = inf.accepted ? inf.terms : -inf.terms;
    }
  }
  if (result) qd_flow_state(f, result);
  std::string msg = rc ? qd::last_error() : std::string();
  qd_flow_destroy(f);
  if (rc) qd::set_error("%s", msg.c_str());
  return rc;
}

}  // extern "C"

namespace {
// ---- batched flows: several instances in lockstep -------------------------
// Every instance runs on its own layout's stream with the kernels and graphs
// of a separate flow (a generator-like Omega leaves no work that a launch
// merged over the instances would share), so that the results are those of
// separate flows; the host launches a step of all of them before it waits
// for any, and the instances' kernels fill the chip together.
//
// BCH_EXPAND of several flows: a step seen before is one graph launch per
// flow; the others go term by term together.
int bch_batch(const std::vector<qd_flow*>& fl, std::vector<int>& terms) {
  const double conv = (double)1e-5f;
  std::vector<char> graph(fl.size(), 0), direct(fl.size(), 0);
  std::vector<double*> p0(fl.size());
  std::vector<int> live;
  auto pandya = [&](const qd_flow* f) { return (f->flags & QD_PANDYA) != 0; };
  for (size_t j = 0; j < fl.size(); ++j) {
    qd_flow* f = fl[j];
    TRY(build_programs(f->L));
    f->INT2->herm = 1;
    f->AD->herm = 1;
    terms[j] = 0;
    bool launched = false;
    TRY(bch_step_launch(f->L, f->HS, f->G, f->HAM, f->INT2, f->AD, f->w1, f->w2, f->HCC, f->OCC, pandya(f), &launched));
    graph[j] = launched;
    if (launched) continue;
    direct[j] = reads_h(f->HAM, f->HS, f->INT2->d, f->AD->d);
    if (!direct[j]) {
      TRY(qd_copy_arrays(f->HAM, f->HS));
      TRY(qd_copy_arrays(f->HAM, f->INT2));
    }
    f->HS->zero_mask = f->HAM->zero_mask;
    p0[j] = f->INT2->d;
    live.push_back((int)j);
  }
  for (int i = 2; i <= 12 && !live.empty(); ++i) {
    const double cof = kCof[i - 2];
    for (int j : live) {
      qd_flow* f = fl[j];
      swap_ops(f->INT2, f->AD);
      const bool first = direct[j] && i == 2;
      TRY(bch_term(f->L, f->G, first ? f->HAM : f->AD, f->INT2, first ? f->HAM : f->HS, f->HS, f->w1, f->w2, f->HCC,
                   f->OCC, pandya(f), i == 2, cof));
      f->HS->zero_mask &= f->INT2->zero_mask;
      ++terms[j];
    }
    std::vector<int> next;
    for (int j : live) {
      QD_CUDA(cudaStreamSynchronize(fl[j]->L->stream));
      const double n1 = fl[j]->L->h_red[1], n2 = fl[j]->L->h_red[2];
      if (!(n2 * cof / n1 < conv)) next.push_back(j);
    }
    live.swap(next);
  }
  for (size_t j = 0; j < fl.size(); ++j) {
    qd_flow* f = fl[j];
    if (graph[j])
      TRY(bch_step_finish(f->L, f->HS, f->G, f->HAM, f->INT2, f->AD, f->HCC, f->OCC, pandya(f), &terms[j]));
    else if (f->INT2->d != p0[j])  // the workspaces keep their buffers
      swap_ops(f->INT2, f->AD);
  }
  return QD_OK;
}

// The lockstep batch: per flow step the instances not yet converged run their
// step halves and one BCH_EXPAND, launched for all before any is waited for.  An instance that fails or exceeds max_iter leaves the
// batch with its own status.
int flow_batch_lockstep(int count, const qd_op* const* HAM, qd_op* const* HS, unsigned flags, int max_iter,
                        qd_flow_result* results, int* status, std::vector<std::string>& msg) {
  std::vector<qd_layout*> Ls(count);
  for (int i = 0; i < count; ++i) {
    Ls[i] = HAM[i]->L;
    TRY(use_device(Ls[i]));
  }
  std::vector<qd_flow*> fl(count, nullptr);
  std::vector<int> loops(count, 0);
  int rc = QD_OK;
  for (int i = 0; i < count; ++i) {
    std::memset(&results[i], 0, sizeof(qd_flow_result));
    status[i] = qd_flow_create(HAM[i], HS[i], flags, &fl[i]);
    if (status[i] != QD_OK) msg[i] = qd::last_error();
  }
  while (rc == QD_OK) {
    std::vector<qd_flow*> act;
    std::vector<int> idx;
    std::vector<qd_flow_step_info> inf(count);
    for (int i = 0; i < count; ++i) {
      if (status[i] != QD_OK || !fl[i] || fl[i]->crit <= kConvCriteria) continue;
      if (loops[i]++ >= max_iter) {
        status[i] = QD_ERR_NOCONV;
        char b[128];
        snprintf(b, sizeof(b), "not converged after %d steps (crit %.3e)", max_iter, fl[i]->crit);
        msg[i] = b;
        continue;
      }
      bool conv = false;
      status[i] = flow_begin(fl[i], &inf[i], &conv);
      if (status[i] != QD_OK) {
        msg[i] = qd::last_error();
        continue;
      }
      act.push_back(fl[i]);
      idx.push_back(i);
    }
    if (act.empty()) break;
    std::vector<int> terms(act.size(), 0);
    rc = bch_batch(act, terms);
    if (rc) break;
    for (int half = 0; half < 2; ++half)
      for (size_t k = 0; k < act.size(); ++k) {
        const int i = idx[k];
        if (status[i] != QD_OK) continue;
        status[i] = half == 0 ? flow_end_launch(act[k]) : flow_end_finish(act[k], terms[k], &inf[i]);
        if (status[i] != QD_OK) msg[i] = qd::last_error();
      }
  }
  const std::string batch_err = rc ? qd::last_error() : std::string();
  for (int i = 0; i < count; ++i) {
    if (fl[i]) {
      qd_flow_state(fl[i], &results[i]);
      qd_flow_destroy(fl[i]);
    }
    if (rc) {
      status[i] = rc;
      msg[i] = batch_err;
    }
  }
  return QD_OK;
}
}  // namespace

extern "C" {

int qd_magnus_flow_batch(int count, const qd_op* const* HAM, qd_op* const* HS, unsigned flags, int max_iter,
                         qd_flow_result* results, int* status) {
  CHECK(count >= 0, QD_ERR_ARG, "qd_magnus_flow_batch: negative count");
  if (count == 0) return QD_OK;
  CHECK(HAM && HS && results && status, QD_ERR_ARG, "qd_magnus_flow_batch: null argument");
  for (int i = 0; i < count; ++i) {
    CHECK(HAM[i] && HS[i], QD_ERR_ARG, "qd_magnus_flow_batch: null operator %d", i);
    for (int j = 0; j < i; ++j)
      CHECK(HAM[i]->L != HAM[j]->L, QD_ERR_ARG,
            "qd_magnus_flow_batch: instances %d and %d share a layout (one stream per instance)", j, i);
  }
  std::vector<std::string> msg(count);
  bool lockstep = !(flags & QD_BATCH_STREAMS);
  for (int i = 0; i < count && lockstep; ++i)
    lockstep = HAM[i]->L->device == HAM[0]->L->device && HAM[i]->L->split_slices == 0 && !HAM[i]->L->prof.on;
  if (lockstep) {
    TRY(flow_batch_lockstep(count, HAM, HS, flags & ~QD_BATCH_STREAMS, max_iter, results, status, msg));
    for (int i = 0; i < count; ++i)
      if (status[i] != QD_OK) {
        qd::set_error("qd_magnus_flow_batch: instance %d: %s", i, msg[i].c_str());
        return status[i];
      }
    return QD_OK;
  }
  // one host thread per instance; each flow runs on its own layout's stream,
  // so the instances' kernels run concurrently on the device
  flags &= ~QD_BATCH_STREAMS;
  std::vector<std::thread> th;
  th.reserve(count);
  for (int i = 0; i < count; ++i)
    th.emplace_back([&, i]() {
      std::memset(&results[i], 0, sizeof(qd_flow_result));
      status[i] = qd_magnus_flow(HAM[i], HS[i], flags, max_iter, nullptr, &results[i]);
      if (status[i] != QD_OK) msg[i] = qd::last_error();
    });
  for (auto& t : th) t.join();
  for (int i = 0; i < count; ++i)
    if (status[i] != QD_OK) {
      qd::set_error("qd_magnus_flow_batch: instance %d: %s", i, msg[i].c_str());
      return status[i];
    }
  return QD_OK;
}

}  // extern "C"

namespace qd {
void graphs_free(qd_layout* L) {
  if (auto* m = reinterpret_cast<TermGraphs*>(L->graphs)) {
    for (auto& kv : *m)
      if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    delete m;
    L->graphs = nullptr;
  }
  if (auto* m = reinterpret_cast<StepGraphs*>(L->step_graphs)) {
    for (auto& kv : *m)
      if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
    delete m;
    L->step_graphs = nullptr;
  }
}
}  // namespace qd
