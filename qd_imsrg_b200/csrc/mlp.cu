// mlp.cu -- the per-element network of the learned warm start:
//   16 -> 256 -> 256 -> 1, GELU (erf form) after the two hidden layers,
//   FP32 master weights, BF16 copies of the 256 x 256 layer and of the
//   activations that feed it, FP32 accumulation everywhere.
// Training: mean squared error, full backward pass, Adam.  Every kernel is
// written here: the 256-wide products run on the tensor cores
// (mma.sync.m16n8k16 bf16 -> f32, NT layout: both operands K-contiguous),
// the 16-wide first layer, the 1-wide last layer, the batch reductions of the
// gradients (fixed order, deterministic) and Adam on CUDA cores.
//
// Parameters (one FP32 vector, QD_MLP_NPARAM entries): W1 [256][16], b1 [256],
// W2 [256][256], b2 [256], w3 [256], b3 [1]; W[out][in].
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "dev_common.cuh"

typedef __nv_bfloat16 bf16;

namespace qd {
namespace {

constexpr int NI = 16, NH = 256;
constexpr i64 O_W1 = 0, O_B1 = O_W1 + NH * NI, O_W2 = O_B1 + NH, O_B2 = O_W2 + NH * NH, O_W3 = O_B2 + NH,
              O_B3 = O_W3 + NH, NPARAM = O_B3 + 1;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// ---- C[M][N] (+= over split-K slices into partial buffers) = A[M][K] B[N][K]^T
constexpr int GBM = 64, GBN = 64, GBK = 32, GLD = GBK + 8;

__device__ __forceinline__ void mma_bf16(float* d, const unsigned* a, const unsigned* b) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// 16 bytes into shared memory, zeros where !ok
__device__ __forceinline__ void cp16(void* smem, const void* g, bool ok) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(g), "r"(ok ? 16 : 0) : "memory");
}

// K and kchunk multiples of GBK; lda, ldb multiples of 8 (16-byte rows).
// Slice z = blockIdx.z covers k in [z*kchunk, min(K, (z+1)*kchunk)) and
// writes C + z * cstride.  Bound: the latency of a slab's loads; three slabs
// are in flight (one at a time: 300 us a gradient of 8,192 rows with the
// reductions below as they were; now see mlp_grad).
constexpr int GST = 3;
__global__ void __launch_bounds__(128) k_gemm_nt_bf16(const bf16* __restrict__ A, int lda, const bf16* __restrict__ B,
                                                      int ldb, float* __restrict__ C, int ldc, i64 cstride, int M,
                                                      int N, int K, int kchunk) {
  __shared__ __align__(16) bf16 As[GST][GBM][GLD];
  __shared__ __align__(16) bf16 Bs[GST][GBN][GLD];
  const int m0 = blockIdx.y * GBM, n0 = blockIdx.x * GBN;
  const int kb = blockIdx.z * kchunk, ke = min(K, kb + kchunk);
  C += (i64)blockIdx.z * cstride;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1, g = lane >> 2, t = lane & 3;
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.f;
  auto load = [&](int k0, int st) {
#pragma unroll
    for (int it = 0; it < 2; ++it) {  // 64 rows x 4 vectors of 8 per operand
      const int v = tid + it * 128, r = v >> 2, seg = (v & 3) * 8;
      const bool oa = m0 + r < M, ob = n0 + r < N;
      cp16(&As[st][r][seg], oa ? A + (i64)(m0 + r) * lda + k0 + seg : A, oa);
      cp16(&Bs[st][r][seg], ob ? B + (i64)(n0 + r) * ldb + k0 + seg : B, ob);
    }
  };
#pragma unroll
  for (int st = 0; st < GST - 1; ++st) {
    if (kb + st * GBK < ke) load(kb + st * GBK, st);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  int st = 0;
  for (int k0 = kb; k0 < ke; k0 += GBK) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GST - 2) : "memory");
    __syncthreads();  // slab st is here, slab st - 1 is read by nobody any more
    if (k0 + (GST - 1) * GBK < ke) load(k0 + (GST - 1) * GBK, (st + GST - 1) % GST);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
    for (int kk = 0; kk < GBK; kk += 16) {
      unsigned af[2][4], bfr[4][2];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        const int rb = wm * 32 + mi * 16;
        af[mi][0] = *reinterpret_cast<const unsigned*>(&As[st][rb + g][kk + 2 * t]);
        af[mi][1] = *reinterpret_cast<const unsigned*>(&As[st][rb + g + 8][kk + 2 * t]);
        af[mi][2] = *reinterpret_cast<const unsigned*>(&As[st][rb + g][kk + 2 * t + 8]);
        af[mi][3] = *reinterpret_cast<const unsigned*>(&As[st][rb + g + 8][kk + 2 * t + 8]);
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        const int cb = wn * 32 + ni * 8;
        bfr[ni][0] = *reinterpret_cast<const unsigned*>(&Bs[st][cb + g][kk + 2 * t]);
        bfr[ni][1] = *reinterpret_cast<const unsigned*>(&Bs[st][cb + g][kk + 2 * t + 8]);
      }
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) mma_bf16(acc[mi][ni], af[mi], bfr[ni]);
    }
    st = (st + 1) % GST;
  }
#pragma unroll
  for (int mi = 0; mi < 2; ++mi)
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {
      const int r0 = m0 + wm * 32 + mi * 16 + g, c = n0 + wn * 32 + ni * 8 + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + 8 * h;
        if (r >= M) continue;
        if (c < N) C[(i64)r * ldc + c] = acc[mi][ni][2 * h];
        if (c + 1 < N) C[(i64)r * ldc + c + 1] = acc[mi][ni][2 * h + 1];
      }
    }
}

// ---- layer 1: Z1 = X W1^T + b1, H1 = GELU(Z1) -> bf16 row-major (and
// transposed).  One CTA per RB rows, thread j = unit j: its weights stay in
// registers, the transposed copy goes through shared memory in 16-byte runs.
constexpr int RB = 32;
// the RB x NH tile t[row][unit] as columns of out (leading dimension ld), rows r0..
__device__ __forceinline__ void write_transposed(const bf16 (*t)[NH + 8], bf16* __restrict__ out, i64 ld, i64 r0,
                                                 int rows) {
  if (rows == RB && (ld & 7) == 0) {
    for (int e = threadIdx.x; e < NH * (RB / 8); e += blockDim.x) {
      const int j = e / (RB / 8), seg = (e % (RB / 8)) * 8;
      __align__(16) bf16 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = t[seg + k][j];
      *reinterpret_cast<uint4*>(out + (i64)j * ld + r0 + seg) = *reinterpret_cast<const uint4*>(v);
    }
  } else {
    for (int e = threadIdx.x; e < NH * rows; e += blockDim.x) out[(i64)(e / rows) * ld + r0 + e % rows] = t[e % rows][e / rows];
  }
}

__global__ void __launch_bounds__(NH) k_layer1(const float* __restrict__ X, const float* __restrict__ P,
                                               float* __restrict__ Z1, bf16* __restrict__ H1, bf16* __restrict__ H1t,
                                               i64 n) {
  __shared__ __align__(16) float x[RB * NI];
  __shared__ bf16 tt[RB][NH + 8];
  const i64 r0 = (i64)blockIdx.x * RB;
  const int rows = (int)min((i64)RB, n - r0), j = threadIdx.x;
  for (int e = j; e < rows * NI; e += NH) x[e] = X[r0 * NI + e];
  float w[NI];
#pragma unroll
  for (int c = 0; c < NI; ++c) w[c] = P[O_W1 + j * NI + c];
  const float b = P[O_B1 + j];
  __syncthreads();
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    float z = b;
#pragma unroll
    for (int c = 0; c < NI; ++c) z += x[r * NI + c] * w[c];
    const bf16 h = __float2bfloat16_rn(gelu(z));
    const i64 o = (r0 + r) * NH + j;
    if (Z1) Z1[o] = z;
    H1[o] = h;
    if (H1t) tt[r][j] = h;
  }
  if (!H1t) return;
  __syncthreads();
  write_transposed(tt, H1t, n, r0, rows);
}

// ---- layer 2 epilogue and layer 3: Z2 += b2, H2 = GELU(Z2), y = H2 w3 + b3 (warp per row)
__global__ void k_layer23(float* __restrict__ Z2, const float* __restrict__ P, float* __restrict__ y, i64 n) {
  const i64 i = (i64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  float s = 0.f;
  for (int j = lane; j < NH; j += 32) {
    const float z = Z2[i * NH + j] + P[O_B2 + j];
    Z2[i * NH + j] = z;
    s += gelu(z) * P[O_W3 + j];
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) y[i] = s + P[O_B3];
}

// ---- the same with the loss and the last layer's backward: per chunk of RB
// rows Z2 += b2, y = GELU(Z2) w3 + b3, dy = 2 (y - t) / n, the sum of
// (y - t)^2, dZ2 = dy (x) w3 * GELU'(Z2) as bf16 (row-major and transposed),
// and the chunk's db2, dw3, db3.  Z2 is read once and never written back.
__global__ void __launch_bounds__(NH) k_tail(const float* __restrict__ Z2, const float* __restrict__ P,
                                             const float* __restrict__ tg, i64 n, bf16* __restrict__ dZ2,
                                             bf16* __restrict__ dZ2t, float* __restrict__ part,
                                             float* __restrict__ lpart) {
  extern __shared__ __align__(16) float zs[];  // [RB][NH]
  __shared__ bf16 tt[RB][NH + 8];
  __shared__ float dys[RB];
  __shared__ double sq[RB];
  const i64 r0 = (i64)blockIdx.x * RB;
  const int rows = (int)min((i64)RB, n - r0), tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int r = w; r < RB; r += NH / 32) {  // a warp per row, as k_layer23
    if (r >= rows) {
      if (lane == 0) sq[r] = 0.0;
      continue;
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NH / 32; ++k) {
      const int j = lane + 32 * k;
      const float z = Z2[(r0 + r) * NH + j] + P[O_B2 + j];
      zs[r * NH + j] = z;
      s += gelu(z) * P[O_W3 + j];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const float d = s + P[O_B3] - tg[r0 + r];
      dys[r] = 2.0f * d / (float)n;
      sq[r] = (double)d * d;
    }
  }
  __syncthreads();
  const int j = tid;
  const float w3 = P[O_W3 + j];
  float db2 = 0.f, dw3 = 0.f, db3 = 0.f;
#pragma unroll 2
  for (int r = 0; r < rows; ++r) {
    const float z = zs[r * NH + j], d = dys[r], v = d * w3 * gelu_d(z);
    const bf16 q = __float2bfloat16_rn(v);
    dZ2[(r0 + r) * NH + j] = q;
    tt[r][j] = q;
    db2 += v;
    dw3 += d * gelu(z);
    db3 += d;
  }
  float* o = part + (i64)blockIdx.x * (2 * NH + 1);
  o[j] = db2;
  o[NH + j] = dw3;
  if (j == 0) {
    o[2 * NH] = db3;
    double s = 0.0;
    for (int r = 0; r < RB; ++r) s += sq[r];
    lpart[blockIdx.x] = (float)s;
  }
  __syncthreads();
  write_transposed(tt, dZ2t, n, r0, rows);
}

// per chunk of RB rows: dZ1 = dH1 * GELU'(Z1); db1[j] += dZ1_ij; dW1[j][c] += dZ1_ij X_ic
__global__ void __launch_bounds__(NH) k_red1(const float* __restrict__ dH1, const float* __restrict__ Z1,
                                             const float* __restrict__ X, i64 n, float* __restrict__ part) {
  __shared__ __align__(16) float x[RB * NI];
  const i64 r0 = (i64)blockIdx.x * RB;
  const int rows = (int)min((i64)RB, n - r0), j = threadIdx.x;
  for (int e = j; e < rows * NI; e += NH) x[e] = X[r0 * NI + e];
  float db1 = 0.f, dw[NI];
#pragma unroll
  for (int c = 0; c < NI; ++c) dw[c] = 0.f;
  __syncthreads();
#pragma unroll 4
  for (int r = 0; r < rows; ++r) {
    const float d = dH1[(r0 + r) * NH + j] * gelu_d(Z1[(r0 + r) * NH + j]);
    db1 += d;
#pragma unroll
    for (int c = 0; c < NI; ++c) dw[c] += d * x[r * NI + c];
  }
  float* o = part + (i64)blockIdx.x * (NH + NH * NI);
  o[j] = db1;
#pragma unroll
  for (int c = 0; c < NI; ++c) o[NH + j * NI + c] = dw[c];
}

// out[e] = sum over chunks z of part[z * ld + e], e < ne: CS_P threads per
// entry take every CS_P-th chunk and add up in a fixed order
constexpr int CS_E = 32, CS_P = 8;
__global__ void __launch_bounds__(CS_E * CS_P) k_sum_chunks(const float* __restrict__ part, i64 nch, int ld, int ne,
                                                            float* __restrict__ out) {
  __shared__ float sh[CS_P][CS_E];
  const int l = threadIdx.x % CS_E, p = threadIdx.x / CS_E, e = blockIdx.x * CS_E + l;
  float s = 0.f;
  if (e < ne) {
#pragma unroll 8
    for (i64 z = p; z < nch; z += CS_P) s += part[z * ld + e];
  }
  sh[p][l] = s;
  __syncthreads();
  if (p || e >= ne) return;
  s = 0.f;
#pragma unroll
  for (int k = 0; k < CS_P; ++k) s += sh[k][l];
  out[e] = s;
}

// gradient vector G from the sums of the chunk partials (s23: db2, dw3, db3;
// s1: db1, dW1) and the slices of the dW2 product, all in fixed order
__global__ void k_grad_collect(const float* __restrict__ s23, const float* __restrict__ s1,
                               const float* __restrict__ kpart, int nz, float* __restrict__ G) {
  const i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= NPARAM) return;
  float s = 0.f;
  if (e < O_B1) {  // W1[j][c]
    s = s1[NH + e];
  } else if (e < O_W2) {  // b1
    s = s1[e - O_B1];
  } else if (e < O_B2) {  // W2[j][l]
#pragma unroll 8
    for (int z = 0; z < nz; ++z) s += kpart[(i64)z * NH * NH + (e - O_W2)];
  } else {  // b2, w3, b3
    s = s23[e - O_B2];
  }
  G[e] = s;
}

__global__ void k_adam(float* __restrict__ P, const float* __restrict__ G, float* __restrict__ M,
                       float* __restrict__ V, float lr, float c1, float c2) {
  const i64 e = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= NPARAM) return;
  const float g = G[e];
  const float m = 0.9f * M[e] + 0.1f * g, v = 0.999f * V[e] + 0.001f * g * g;
  M[e] = m;
  V[e] = v;
  P[e] -= lr * (m / c1) / (sqrtf(v / c2) + 1e-8f);
}

// bf16 copies of W2 (row-major [out][in]) and its transpose
__global__ void k_w2_bf16(const float* __restrict__ P, bf16* __restrict__ W2b, bf16* __restrict__ W2tb) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= NH * NH) return;
  const int j = e / NH, l = e % NH;
  const bf16 v = __float2bfloat16_rn(P[O_W2 + e]);
  W2b[e] = v;
  W2tb[(i64)l * NH + j] = v;
}

}  // namespace
}  // namespace qd

struct qd_mlp {
  int device = 0;
  float *P = nullptr, *M = nullptr, *V = nullptr, *G = nullptr;
  bf16 *W2b = nullptr, *W2tb = nullptr;
  long long step = 0;
  // activations of up to cap rows, and what a gradient needs beside them for up to gcap
  qd::i64 cap = 0, gcap = 0;
  void *params = nullptr, *acts = nullptr, *grads = nullptr;  // all memory, one allocation each
  bf16* H1 = nullptr;
  float* Z2 = nullptr;
  float *Z1 = nullptr, *dH1 = nullptr;
  bf16 *H1t = nullptr, *dZ2 = nullptr, *dZ2t = nullptr;
  float *p23 = nullptr, *p1 = nullptr, *lpart = nullptr, *kpart = nullptr;  // partials per RB rows, dW2 slices
  float *s23 = nullptr, *s1 = nullptr;                                       // their sums
  std::vector<float> h_loss;        // host copy of lpart
  cudaStream_t loss_st = nullptr;   // brings it while the rest of the gradient runs
  cudaEvent_t loss_ev = nullptr;
  int kslices = 0;
};

using namespace qd;

namespace {
// n elements of T at the end of a memory plan of *bytes so far
template <class T>
T* mlp_place(void* base, size_t* bytes, i64 n) {
  T* p = base ? reinterpret_cast<T*>((char*)base + *bytes) : nullptr;
  *bytes += ((size_t)n * sizeof(T) + 255) / 256 * 256;
  return p;
}

i64 mlp_rows(i64 n) { return (n + 1023) / 1024 * 1024; }

// (Re)allocates *mem for what plan(base) places (called without memory first,
// for the size).  cudaMalloc takes about 0.4 ms for arrays of this size: with
// eleven of them, and 2.8 ms for pinned memory for the loss, a network's first
// gradient (8,192 rows) took 5.4 ms and its destruction 3.3; now 0.8 and 0.9.
template <class F>
int mlp_alloc(void** mem, i64* cap, i64 rows, F plan) {
  if (*mem) cudaFree(*mem);
  *mem = nullptr;
  *cap = 0;
  QD_CUDA(cudaMalloc(mem, plan(nullptr)));
  plan(*mem);
  *cap = rows;
  return QD_OK;
}

// a forward pass of n rows: 1.5 KB a row
int mlp_ensure(qd_mlp* m, i64 n) {
  if (n <= m->cap) return QD_OK;
  const i64 c = mlp_rows(n);
  return mlp_alloc(&m->acts, &m->cap, c, [&](void* b) {
    size_t o = 0;
    m->H1 = mlp_place<bf16>(b, &o, c * NH);
    m->Z2 = mlp_place<float>(b, &o, c * NH);
    return o;
  });
}

// a gradient of n rows: further 4.1 KB a row
int mlp_ensure_grad(qd_mlp* m, i64 n) {
  if (n <= m->gcap) return QD_OK;
  const i64 c = mlp_rows(n), nch = c / RB;
  m->kslices = (int)std::max<i64>(1, std::min<i64>(64, c / 512));
  return mlp_alloc(&m->grads, &m->gcap, c, [&](void* b) {
    size_t o = 0;
    m->Z1 = mlp_place<float>(b, &o, c * NH);
    m->dH1 = mlp_place<float>(b, &o, c * NH);
    m->H1t = mlp_place<bf16>(b, &o, c * NH);
    m->dZ2 = mlp_place<bf16>(b, &o, c * NH);
    m->dZ2t = mlp_place<bf16>(b, &o, c * NH);
    m->p23 = mlp_place<float>(b, &o, nch * (2 * NH + 1));
    m->p1 = mlp_place<float>(b, &o, nch * (NH + NH * NI));
    m->lpart = mlp_place<float>(b, &o, nch);
    m->kpart = mlp_place<float>(b, &o, (i64)m->kslices * NH * NH);
    return o;
  });
}

// C = A B^T, or with *slices > 1 the K slices' partial products one after
// another in C (*slices: how many)
int gemm_nt(const bf16* A, int lda, const bf16* B, int ldb, float* C, int ldc, int M, int N, int K, int* slices,
            cudaStream_t st) {
  if (K % GBK) {
    set_error("mlp: inner dimension %d is not a multiple of %d", K, GBK);
    return QD_ERR_ARG;
  }
  const int want = slices ? *slices : 1;
  const int kchunk = ((K + want - 1) / want + GBK - 1) / GBK * GBK, nz = (K + kchunk - 1) / kchunk;
  dim3 grid((N + GBN - 1) / GBN, (M + GBM - 1) / GBM, nz);
  k_gemm_nt_bf16<<<grid, 128, 0, st>>>(A, lda, B, ldb, C, ldc, (i64)M * ldc, M, N, K, kchunk);
  if (slices) *slices = nz;
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// layers 1 and 2 of rows [0, n) of X: Z2 without its bias (keeps Z1, H1, H1t when train)
int mlp_hidden(qd_mlp* m, const float* X, i64 n, bool train, cudaStream_t st) {
  int rc = mlp_ensure(m, n);
  if (rc) return rc;
  k_layer1<<<(unsigned)((n + RB - 1) / RB), NH, 0, st>>>(X, m->P, train ? m->Z1 : nullptr, m->H1,
                                                        train ? m->H1t : nullptr, n);
  return gemm_nt(m->H1, NH, m->W2b, NH, m->Z2, NH, (int)n, NH, NH, nullptr, st);
}

// forward of rows [0, n) of X into y
int mlp_forward(qd_mlp* m, const float* X, i64 n, float* y, cudaStream_t st) {
  int rc = mlp_hidden(m, X, n, false, st);
  if (rc) return rc;
  k_layer23<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(m->Z2, m->P, y, n);
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// gradient of mean((y - t)^2) into G; the chunks' sums of squares stay in
// m->lpart (with want_loss, mlp_loss brings them).
// Bound: latency of nine launches.  A batch of 8,192 rows, with the earlier
// reductions (64 CTAs for all rows, a barrier per row) and now: 302 and 104 us.
int mlp_grad(qd_mlp* m, const float* X, const float* T, i64 n, float* G, bool want_loss, cudaStream_t st) {
  if (n <= 0 || n % GBK) {
    set_error("qd_mlp: the batch (%lld rows) must be a positive multiple of %d", (long long)n, GBK);
    return QD_ERR_ARG;
  }
  int rc = mlp_ensure_grad(m, n);
  if (!rc) rc = mlp_hidden(m, X, n, true, st);
  if (rc) return rc;
  const i64 nch = (n + RB - 1) / RB;
  k_tail<<<(unsigned)nch, NH, sizeof(float) * RB * NH, st>>>(m->Z2, m->P, T, n, m->dZ2, m->dZ2t, m->p23, m->lpart);
  if (want_loss) {
    if (!m->loss_st) QD_CUDA(cudaStreamCreateWithFlags(&m->loss_st, cudaStreamNonBlocking));
    if (!m->loss_ev) QD_CUDA(cudaEventCreateWithFlags(&m->loss_ev, cudaEventDisableTiming));
    QD_CUDA(cudaEventRecord(m->loss_ev, st));
  }
  // dW2[j][l] = sum_i dZ2[i][j] H1[i][l]: A = dZ2^T (256 x n), B = H1^T (256 x n), K = n
  int nz = m->kslices;
  if ((rc = gemm_nt(m->dZ2t, (int)n, m->H1t, (int)n, m->kpart, NH, NH, NH, (int)n, &nz, st))) return rc;
  // dH1 = dZ2 W2: A = dZ2 (n x 256), B = W2^T (256 x 256)
  if ((rc = gemm_nt(m->dZ2, NH, m->W2tb, NH, m->dH1, NH, (int)n, NH, NH, nullptr, st))) return rc;
  k_red1<<<(unsigned)nch, NH, 0, st>>>(m->dH1, m->Z1, X, n, m->p1);
  k_sum_chunks<<<(2 * NH + 1 + CS_E - 1) / CS_E, CS_E * CS_P, 0, st>>>(m->p23, nch, 2 * NH + 1, 2 * NH + 1, m->s23);
  k_sum_chunks<<<(NH + NH * NI + CS_E - 1) / CS_E, CS_E * CS_P, 0, st>>>(m->p1, nch, NH + NH * NI, NH + NH * NI, m->s1);
  k_grad_collect<<<(unsigned)((NPARAM + 255) / 256), 256, 0, st>>>(m->s23, m->s1, m->kpart, nz, G);
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

// The loss of the gradient just launched on st, and the end of that gradient:
// a few KB to pageable memory, on a stream of its own, which holds up the host
// but not the kernels after k_tail.  A gradient of 8,192 rows: copied on st to
// pinned memory behind k_tail 110 us, at its end 112, this way 104.
int mlp_loss(qd_mlp* m, i64 n, cudaStream_t st, float* loss) {
  const i64 nch = (n + RB - 1) / RB;
  m->h_loss.resize((size_t)nch);
  QD_CUDA(cudaStreamWaitEvent(m->loss_st, m->loss_ev, 0));
  QD_CUDA(cudaMemcpyAsync(m->h_loss.data(), m->lpart, sizeof(float) * nch, cudaMemcpyDeviceToHost, m->loss_st));
  QD_CUDA(cudaStreamSynchronize(m->loss_st));
  QD_CUDA(cudaStreamSynchronize(st));
  double s = 0.0;
  for (float v : m->h_loss) s += v;
  *loss = (float)(s / (double)n);
  return QD_OK;
}
}  // namespace

extern "C" {

int qd_mlp_create(int device, uint64_t seed, qd_mlp** out) {
  if (!out) {
    set_error("qd_mlp_create: null output");
    return QD_ERR_ARG;
  }
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    set_error("qd_mlp_create: no CUDA device");
    return QD_ERR_NODEVICE;
  }
  qd_mlp* m = new qd_mlp();
  if (device < 0)
    cudaGetDevice(&m->device);
  else
    m->device = device;
  QD_CUDA(cudaSetDevice(m->device));
  // He-style initialisation, fixed seed
  std::vector<float> p(NPARAM, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<float> nd(0.f, 1.f);
  for (i64 e = O_W1; e < O_B1; ++e) p[e] = nd(rng) * std::sqrt(2.0f / NI);
  for (i64 e = O_W2; e < O_B2; ++e) p[e] = nd(rng) * std::sqrt(2.0f / NH);
  for (i64 e = O_W3; e < O_B3; ++e) p[e] = nd(rng) * std::sqrt(1.0f / NH);
  int rc = QD_OK;
  i64 one = 0;
  rc = mlp_alloc(&m->params, &one, 1, [&](void* b) {
    size_t o = 0;
    m->P = mlp_place<float>(b, &o, NPARAM);
    m->M = mlp_place<float>(b, &o, NPARAM);
    m->V = mlp_place<float>(b, &o, NPARAM);
    m->G = mlp_place<float>(b, &o, NPARAM);
    m->W2b = mlp_place<bf16>(b, &o, NH * NH);
    m->W2tb = mlp_place<bf16>(b, &o, NH * NH);
    m->s23 = mlp_place<float>(b, &o, 2 * NH + 1);
    m->s1 = mlp_place<float>(b, &o, NH + NH * NI);
    return o;
  });
  if (rc) {
    delete m;
    return rc;
  }
  QD_CUDA(cudaMemcpy(m->P, p.data(), sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
  QD_CUDA(cudaMemset(m->M, 0, sizeof(float) * NPARAM));
  QD_CUDA(cudaMemset(m->V, 0, sizeof(float) * NPARAM));
  QD_CUDA(cudaFuncSetAttribute(k_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(float) * RB * NH)));
  k_w2_bf16<<<NH * NH / 256, 256>>>(m->P, m->W2b, m->W2tb);
  QD_CUDA(cudaDeviceSynchronize());
  *out = m;
  return QD_OK;
}

int qd_mlp_destroy(qd_mlp* m) {
  if (!m) return QD_OK;
  cudaSetDevice(m->device);
  cudaDeviceSynchronize();
  if (m->loss_st) cudaStreamDestroy(m->loss_st);
  if (m->loss_ev) cudaEventDestroy(m->loss_ev);
  for (void* p : {m->params, m->acts, m->grads})
    if (p) cudaFree(p);
  (void)cudaGetLastError();
  delete m;
  return QD_OK;
}

int qd_mlp_get_params(const qd_mlp* m, float* host, int64_t n) {
  if (!m || !host || n != NPARAM) {
    set_error("qd_mlp_get_params: need %lld floats", (long long)NPARAM);
    return QD_ERR_ARG;
  }
  QD_CUDA(cudaSetDevice(m->device));
  QD_CUDA(cudaMemcpy(host, m->P, sizeof(float) * NPARAM, cudaMemcpyDeviceToHost));
  return QD_OK;
}

int qd_mlp_set_params(qd_mlp* m, const float* host, int64_t n) {
  if (!m || !host || n != NPARAM) {
    set_error("qd_mlp_set_params: need %lld floats", (long long)NPARAM);
    return QD_ERR_ARG;
  }
  QD_CUDA(cudaSetDevice(m->device));
  QD_CUDA(cudaMemcpy(m->P, host, sizeof(float) * NPARAM, cudaMemcpyHostToDevice));
  QD_CUDA(cudaMemset(m->M, 0, sizeof(float) * NPARAM));
  QD_CUDA(cudaMemset(m->V, 0, sizeof(float) * NPARAM));
  m->step = 0;
  k_w2_bf16<<<NH * NH / 256, 256>>>(m->P, m->W2b, m->W2tb);
  QD_CUDA(cudaDeviceSynchronize());
  return QD_OK;
}

int qd_mlp_forward(qd_mlp* m, const float* d_X, float* d_y, int64_t n, void* stream) {
  if (!m || (n > 0 && (!d_X || !d_y)) || n < 0) {
    set_error("qd_mlp_forward: bad argument");
    return QD_ERR_ARG;
  }
  QD_CUDA(cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  const i64 chunk = 1 << 18;  // bounded activation workspace
  for (i64 r = 0; r < n; r += chunk) {
    const i64 k = std::min<i64>(chunk, n - r);
    int rc = mlp_forward(m, d_X + r * NI, k, d_y + r, st);
    if (rc) return rc;
  }
  return QD_OK;
}

int qd_mlp_grad(qd_mlp* m, const float* d_X, const float* d_T, int64_t n, float* d_grad, float* loss, void* stream) {
  if (!m || !d_X || !d_T || !d_grad) {
    set_error("qd_mlp_grad: null argument");
    return QD_ERR_ARG;
  }
  QD_CUDA(cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  int rc = mlp_grad(m, d_X, d_T, n, d_grad, loss != nullptr, st);
  if (rc) return rc;
  if (loss) return mlp_loss(m, n, st, loss);
  QD_CUDA(cudaStreamSynchronize(st));
  return QD_OK;
}

int qd_mlp_train_step(qd_mlp* m, const float* d_X, const float* d_T, int64_t n, float lr, float* loss,
                      void* stream) {
  if (!m || !d_X || !d_T) {
    set_error("qd_mlp_train_step: null argument");
    return QD_ERR_ARG;
  }
  QD_CUDA(cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  int rc = mlp_grad(m, d_X, d_T, n, m->G, loss != nullptr, st);
  if (!rc && loss) rc = mlp_loss(m, n, st, loss);
  if (rc) return rc;
  m->step += 1;
  const float c1 = 1.0f - std::pow(0.9f, (float)m->step), c2 = 1.0f - std::pow(0.999f, (float)m->step);
  k_adam<<<(unsigned)((NPARAM + 255) / 256), 256, 0, st>>>(m->P, m->G, m->M, m->V, lr, c1, c2);
  k_w2_bf16<<<NH * NH / 256, 256, 0, st>>>(m->P, m->W2b, m->W2tb);
  QD_CUDA(cudaGetLastError());
  return QD_OK;
}

}  // extern "C"
