// qd_internal.hpp -- host/device structures of the IM-SRG(2) commutator engine.
//
// Layout mirrors the reference's type(full_ham) / type(block) / type(cc_mat)
// (src/ME_general.f90:13-62) with everything needed on the device flattened
// into index tables:
//   * one FP64 array per operator in vectorize order (ME_general.f90:1871-1989)
//   * per (M_L,M_S) block: nhh, nph, npp and the six sub-block offsets
//   * a dense m*m pair table: ordered pair (a,b) -> (class, block, index, swap),
//     which is reindex's i_array (ME_general.f90:1028-1080) plus the ordering
//     sign of v_elem (ME_general.f90:1586-1599)
//   * cross-coupled (Pandya) blocks of build_cross_coupled (ME_general.f90:363-448)
//   * single-particle (m_l, m_s) groups: the only one-body couplings that reach
//     a block-diagonal two-body element (used to restrict the 122 sums).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <map>
#include <memory>
#include <string>
#include <memory>
#include <type_traits>
#include <vector>

#include "../../include/qd_imsrg.h"

namespace qd {

typedef long long i64;

// class ids of the nine stored parts of an operator (bit positions of
// qd_op::zero_mask)
enum Part { P_FHH = 0, P_FPP, P_FPH, P_HHHH, P_PPPP, P_PPHH, P_PHPH, P_PPPH, P_PHHH, P_COUNT };
constexpr unsigned ALL_PARTS = (1u << P_COUNT) - 1;
// Further bit of qd_op::zero_mask: no one-body entry couples states of
// different (m_l, m_s) (such entries are all known to be zero).
constexpr unsigned CONSERVES = 1u << (P_COUNT + 1);
// A holds only fph and Vpphh (the Magnus generator, the White generator).
inline bool gen_like(unsigned zmask) {
  return ((zmask | (1u << P_FPH) | (1u << P_PPHH)) & ALL_PARTS) == ALL_PARTS;
}
constexpr unsigned ONE_BODY = (1u << P_FHH) | (1u << P_FPP) | (1u << P_FPH);

// pair-table packing: idx (13 bits) | block (10 bits) | class-1 (2 bits) | swap (1 bit)
__host__ __device__ inline int pt_idx(int e) { return e & 0x1FFF; }
__host__ __device__ inline int pt_blk(int e) { return (e >> 13) & 0x3FF; }
__host__ __device__ inline int pt_cls(int e) { return (e >> 23) & 0x3; }  // 0 hh, 1 ph, 2 pp
__host__ __device__ inline int pt_swap(int e) { return (e >> 25) & 0x1; }
inline int pt_pack(int idx, int blk, int cls, int swap) {
  return idx | (blk << 13) | (cls << 23) | (swap << 25);
}

// Device view of a layout (passed by value to kernels).
struct DevLayout {
  int n, m, mp, nblock, ncc, mlmax;
  i64 o_fhh, o_fpp, o_fph, neq;
  const int4* blk;        // nhh, nph, npp, ntot
  const i64* boff;        // 6 per block: hhhh, pppp, pphh, phph, ppph, phhh
  const int2* pairs;      // per block: hh pairs, ph pairs, pp pairs (0-based, a<b)
  const int* pbase;       // start of block q's pairs
  const int* ptab;        // m*m ordered pair -> packed, -1 on the diagonal
  const int* gid;         // (ml,ms) group of each state
  const int* gstart;      // CSR of group members (increasing states)
  const int* gmem;
  const int2* ccmap;      // m*m: (cc block, row), 0-based
  const int2* ccdim;      // r, nb per cc block
  const i64* ccxoff;      // offset of X(r,nb) per cc block
  const i64* cczoff;      // offset of the r x r product per cc block q >= ncc - 1 - q
  const int2* ccab;       // concatenated (i,j) row pairs of the cc blocks
  const int* ccab_base;
  const int2* cchp;       // concatenated (hole, particle) column pairs
  const int* cchp_base;
  // all non-empty two-body sub-blocks in vectorize order: start offset and
  // (block << 3) | (part - P_HHHH)
  const i64* s2off;
  const int* s2id;
  int ns2;
  i64 o2;                 // first two-body entry of the vectorize array
  // per two-body part p (0..5 = P_HHHH..P_PHHH): start of block q's entries
  // in the part's own flat numbering (pcum[p*nblock + q]) and the total
  const i64* pcum;
  i64 pcnt[6];
  // X (cross-coupled) flat numbering: cc block of each X entry via ccxoff
};

// ---- grouped FP64 GEMM program --------------------------------------------
enum GemmMode { GM_ACC = 0, GM_ACC_PAIR = 1, GM_SET = 2, GM_SET_PAIR = 3 };

struct GSeg {       // acc += alpha * op(A) * op(B), alpha = c * hv[0]^pa * hv[1]^pb
  i64 offA, offB;
  int lda, ldb, K;
  signed char srcA, srcB, tA, tB;
  signed char pa, pb, depA, depB;  // dep: part id of the source operator (-1 none)
  double c;
};
struct GProb {
  int M, N, ldc, seg0, nseg, mode, outbuf, pad;
  i64 offC;
  double sc;                       // pair transpose coefficient sc * hv[0]^spa * hv[1]^spb
  signed char spa, spb, pad2[6];
};
struct GTask {
  int prob;
  int r0, c0;  // first row and column of the tile
  int shape;   // tile_shape(rows, columns)
};

constexpr int NBUF = 7;
struct Bufs {
  const double* p[NBUF];
};
struct GemmProgram {
  std::vector<GProb> probs;
  std::vector<GSeg> segs;
  GProb* d_probs = nullptr;
  GSeg* d_segs = nullptr;
  // task lists cached per (maskA, maskB): problems with a long K, and
  // K-short problems (every active segment together K <= 16)
  std::map<std::pair<unsigned, unsigned>, std::pair<GTask*, int>> tasks, tasks_short;
  void clear_device();
};

}  // namespace qd

namespace qd {
// stages timed by the optional per-stage CUDA-event profiler
struct OneBody;  // tables of the fused one-body stage (onebody.cu)
struct PhGen;    // tables and buffers of the particle-hole channel of a generator-like A (ph_gen.cu)
enum Stage { S_E0 = 0, S_111, S_121, S_221, S_122, S_CALC_CC, S_LADDER, S_PANDYA_GEMM, S_PANDYA_GATHER, S_GLUE,
             S_COUNT };
struct StageProf {
  bool on = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pending[S_COUNT];
  double ms[S_COUNT] = {0};
  long long count[S_COUNT] = {0};
};
}  // namespace qd

struct qd_layout {
  int device = 0;
  int children = 0;      // live operators and cross-coupled matrices on this layout
  bool closing = false;  // qd_layout_destroy was called while children were alive
  qd::StageProf prof;
  long long nlaunch = 0;  // kernels this library launched for the layout
  int n = 0, m = 0, mp = 0, emax = 0, nblock = 0, ncc = 0, mlmax = 0;
  qd::i64 neq = 0, o_fhh = 1, o_fpp = 0, o_fph = 0;
  std::vector<int> qn;      // m x 3 (n, ml, ms)
  std::vector<double> eig;  // m
  std::vector<int4> blk;
  std::vector<qd::i64> boff;
  std::vector<int2> pairs;
  std::vector<int> pbase;
  std::vector<int> ptab, gid, gstart, gmem;
  std::vector<int2> ccmap, ccdim, ccab, cchp;
  std::vector<int> ccab_base, cchp_base;
  // Rows of a cc block are ordered by the (ml,ms) group of their first state,
  // then (i, j): the rows (i in G1, j in G2) form one run; below the block of
  // no transfer, as the reversed pairs of the opposite block.  ccref maps each
  // row (indexed like ccab) to its row in the reference's (i, j) loop order.
  std::vector<int> ccref;
  std::vector<qd::i64> ccxoff, cczoff;
  qd::i64 xsize = 0, zsize = 0;
  std::vector<qd::i64> s2off, pcum;
  std::vector<int> s2id;
  // device copies
  qd::DevLayout dev{};
  std::vector<void*> dev_allocs;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  // work arena (grown on demand, freed with the layout)
  double* d_z = nullptr;          // Pandya products, zsize doubles
  double* d_red = nullptr;        // reduction partials
  double* h_red = nullptr;        // pinned scalar results
  double* d_axn = nullptr;        // partial sums of the fused BCH update (axpy + norms)
  double* d_axp = nullptr;        // the same for the update split between k_gen_pppp and the rest
  const longlong2* d_axrest = nullptr;  // {offset, entries} of the pieces outside Vpppp
  int naxrest = 0, naxp = 0;            // pieces; CTAs of k_gen_pppp
  int* d_ccflag = nullptr;        // per cross-coupled block: fph of A or B non-zero (121)
  const int4* d_cctask = nullptr;  // calc_cc: {cross-coupled block, first row, first column}
  int ncctask = 0;
  const int* d_tgt221 = nullptr;  // one-body targets whose states share (m_l, m_s) (fused 221)
  int ntgt221 = -1;
  qd::OneBody* onebody = nullptr;
  qd::PhGen* ph_gen = nullptr;
  // branches of one commutator that run beside the main stream's (api.cu)
  static constexpr int NSIDE = 3;
  cudaStream_t side[NSIDE] = {nullptr};
  cudaEvent_t ev_fork = nullptr, ev_side[NSIDE] = {nullptr};
  int serial_calls = 0;  // calls that went without them
  qd::i64 ws_bytes = 0;
  // GEMM programs
  qd::GemmProgram prog_ladder, prog_221, prog_111, prog_pandya;
  qd::GemmProgram prog_ladder_gen;  // the blocks of prog_ladder that gen_ladder_fused leaves out
  bool programs_built = false;
  // split form of the GEMM programs: slices per operand (0 = plain FP64)
  int split_slices = 0;
  void* split = nullptr;  // plans and workspaces (split_gemm.cu)
  // BCH terms replayed as CUDA graphs (api.cu)
  bool use_graphs = true;
  void* graphs = nullptr;       // per-term graphs
  void* step_graphs = nullptr;  // whole BCH steps with the truncation decided on the device
  long long graphs_captured = 0, graph_replays = 0;
  long long step_first = 0, step_per_term = 0;  // launches of the step graph in flight
};

struct qd_op {
  qd_layout* L = nullptr;
  int herm = 1;
  double* d = nullptr;
  unsigned zero_mask = 0;  // parts known to be identically zero
  bool exposed = false;    // a raw pointer to d was handed out: the caller may write between calls
};

struct qd_cc {
  qd_layout* L = nullptr;
  double herm = 1.0;
  double* d = nullptr;  // X, xsize doubles
  bool filled = false;  // calc_cc has written X (otherwise X == 0)
};

namespace qd {

// error plumbing
void set_error(const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
#define QD_CUDA(call)                                   \
  do {                                                  \
    cudaError_t e_ = (call);                            \
    if (e_ != cudaSuccess) return qd::cuda_fail(e_, #call); \
  } while (0)

// A plan's table from host memory, at its place when this returns.  A copy
// from pageable memory may return before it has arrived, and the layouts'
// streams do not wait for the legacy stream: a kernel launched next could
// read what the (recycled) memory held before.
inline cudaError_t copy_table(void* dst, const void* src, size_t bytes) {
  const cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  return e != cudaSuccess ? e : cudaStreamSynchronize(cudaStreamLegacy);
}

// Device memory of one plan, tables and scratch together in one allocation
// that belongs to the layout.  The tables lie in the order of add(), each on
// the next multiple of ALIGN bytes.  commit() brings them to the device and
// sets every pointer, or on failure none and keeps nothing.
class PlanMemory {
 public:
  static constexpr size_t ALIGN = 256;
  template <class T, class P>
  void add(std::vector<T> v, P** out) {
    static_assert(std::is_same<typename std::remove_const<P>::type, T>::value, "pointer of another type");
    auto kept = std::make_shared<std::vector<T>>(std::move(v));
    pieces_.push_back(Piece{kept->data(), kept->size() * sizeof(T), (const void**)out});
    kept_.push_back(kept);
  }
  template <class T>
  void room(i64 n, T** out) {  // not initialised
    pieces_.push_back(Piece{nullptr, (size_t)n * sizeof(T), (const void**)out});
  }
  int commit(qd_layout* L);

 private:
  struct Piece {
    const void* src;
    size_t bytes;
    const void** out;  // may be null
  };
  std::vector<Piece> pieces_;
  std::vector<std::shared_ptr<void>> kept_;
};

int layout_build(qd_layout* L, int nbody, int emax, const double* eig);
int layout_upload(qd_layout* L);
void layout_free_device(qd_layout* L);
int ensure_reduction(qd_layout* L);
int ensure_z(qd_layout* L);
int build_programs(qd_layout* L);

// part helpers
i64 part_count(const qd_layout* L, int part);  // total elements of a part over all blocks

// BCH update of one term, HS = src + cof C with |src| and |C| (src: HS itself,
// or the series' first operator), for the
// C_pppp entries where they are produced (k_gen_pppp); partial receives two
// sums of squares per CTA.  kidx: a device counter that picks the coefficient.
struct HsUpdate {
  const double* src = nullptr;
  double* HS = nullptr;
  double cof = 0.0;
  int* kidx = nullptr;
  double* partial = nullptr;
};
// BCH_EXPAND's exit test on the device, taken with a term's update
struct BchDecide {
  cudaGraphConditionalHandle hloop = 0, hnext = 0;
  int on = 0, set_next = 0;
  double conv = 0.0;
};
// kernels (kernels_*.cu)
int launch_axpy(qd_layout* L, const double* a, double sa, const double* b, double sb, double* c, i64 n);
// the same on E0, fph and Vpphh alone (every other part zero in a, b and c)
int launch_axpy_gen(qd_layout* L, const double* a, double sa, const double* b, double sb, double* c);
int launch_axpy_norms(qd_layout* L, const double* a, double sa, const double* b, double sb, double* c,
                      double* dout2, int* kidx = nullptr, const BchDecide& D = BchDecide{});
// The same for every entry outside Vpppp, with the CTAs' sums of k_gen_pppp
// (HsUpdate::partial) added; *upd is filled by hs_update_begin, which also
// makes the tables and buffers (ahead of a stream capture: prepare_hs_update).
int prepare_hs_update(qd_layout* L);
int hs_update_begin(qd_layout* L, const double* src, double* HS, double cof, int* kidx, HsUpdate* upd);
int launch_axpy_norms_rest(qd_layout* L, const double* b, const HsUpdate& upd, double* dout2,
                           const BchDecide& D = BchDecide{});
int prepare_program(qd_layout* L, GemmProgram& P, unsigned maskA, unsigned maskB);
int prepare_122(qd_layout* L, const qd_op* A, const qd_op* B);
std::string tuning_report_122(const qd_layout* L);
double* scratch_operator(qd_layout* L);
int reduce_dot_range(qd_layout* L, const double* a, const double* b, i64 o, i64 n, double scale, double add,
                     double* dout);
int reduce_dot_part(qd_layout* L, const double* a, const double* b, int part, double scale, double add, double* dout);
int reduce_mbpt2(qd_layout* L, const double* h, double* dout);
int reduce_hhtrace(qd_layout* L, const double* h, double* dout);
// zmask: parts known to be zero (fph and Vpphh alone are read if the rest is)
int reduce_norm(qd_layout* L, const double* a, unsigned zmask, double* dout);
double* red_slot(qd_layout* L, int k);
int launch_white(qd_layout* L, double* gen, const double* h, int herm);
int launch_keep_parts(qd_layout* L, double* op, unsigned keep);
int launch_121(qd_layout* L, const qd_op* A, const qd_op* B, double* C);
int launch_221_trace(qd_layout* L, const qd_op* A, const qd_op* B, const qd_op* w1, const qd_op* w2, double* C);
// One product of ph_gen: Y (r x rows, at offY) = X_B (r x nb, at offB) X'_A^T (rows x nb, at offA)
struct PhProduct {
  int r, rows, nb;
  i64 offY, offB, offA;
};
int build_ph_products(qd_layout* L, const std::vector<PhProduct>& v, GemmProgram& P);
int prepare_ph_gen(qd_layout* L);
int launch_ph_gen_products(qd_layout* L, const qd_op* A, const double* XB, double hB);
int launch_ph_gen(qd_layout* L, double hA, double hB, double* C);
void ph_gen_free(qd_layout* L);
int prepare_onebody(qd_layout* L);
int launch_onebody(qd_layout* L, const qd_op* A, const qd_op* B, double* C, bool* done);
void onebody_free(qd_layout* L);
int launch_221_fused(qd_layout* L, const qd_op* A, const qd_op* B, double* C);
// CTAs of k_gen_pppp for L (each writes two partial sums), 0 if it is not used
int gen_pppp_ctas(qd_layout* L, int* n);
// ladder: for a generator-like A also the ladders of the blocks for which
// gen_ladder_fused holds (the caller then runs prog_ladder_gen, not prog_ladder)
// st2: second stream: the parts other than C_pppp of a generator-like A,
// every other launch of the tiles otherwise (null: the layout's); upd: update
// HS with C_pppp (generator-like A only)
int launch_122(qd_layout* L, const qd_op* A, const qd_op* B, double* C, bool ladder, cudaStream_t st2 = nullptr,
               const HsUpdate* upd = nullptr);
bool gen_ladder_fused(const qd_layout* L, int q);
int launch_calc_cc(qd_layout* L, const qd_op* H, double* X);
int make_branches(qd_layout* L);  // the side streams and events of a layout (api.cu)
int use_branches(qd_layout* L, bool* use);
// Particle-hole channel (commutators.f90:716-980): C += the four re-coupled
// Z terms, over the commutator_122 tiles (kernels_122.cu).
int launch_pandya_tiles(qd_layout* L, const double* Z, double* C);
int prepare_pandya(qd_layout* L);
int run_program(qd_layout* L, GemmProgram& P, const double* const* bufs, double hv0, double hv1, unsigned maskA,
                unsigned maskB);
int run_program_f64(qd_layout* L, GemmProgram& P, const double* const* bufs, double hv0, double hv1, unsigned maskA,
                    unsigned maskB);
int build_eom_ladders(qd_layout* L, const std::vector<int>& partner, const std::vector<i64>& qoff, GemmProgram& P);
void drop_eom_plans(const qd_layout* L);
void fill_random(const qd_layout* L, int herm, uint64_t seed, double sigma, int conserve, double* out);
int run_program_split(qd_layout* L, GemmProgram& P, const double* const* bufs, double hv0, double hv1, unsigned maskA,
                      unsigned maskB);
void split_free(qd_layout* L);
void graphs_free(qd_layout* L);

}  // namespace qd
