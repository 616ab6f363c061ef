// dndsg_mlp.cuh -- learned warm start for the VR coefficients (no counterpart in
// the reference): a per-cell MLP 64 -> 64 -> 64 -> 64 -> 20 (SiLU), BF16 weights
// and activations, FP32 accumulation, on the 5th-generation tensor cores
// (tcgen05.mma with the accumulators in tensor memory): inference (k_mlp_tc) and
// training (k_mlp_train_tc: forward, backward with the weight and input
// gradients, then Adam on the FP32 master parameters).
//
// The network extrapolates the Jacobi sequence: from the starting coefficients
// x0 and two plain sweeps x1 = J(x0), x2 = J(x1) it proposes the converged
// coefficients x* (for an error dominated by one slow mode of eigenvalue l,
// x* - x2 = (x2 - x1) l / (1 - l); the network learns the local, many-mode
// version of that from the solver's own iterations).
// Features of cell i (d1 = x1 - x0, d2 = x2 - x1):
//   x[4k + v]      = du_k[v] / s_v,  du_k = u_j(k) - u_i over the face slots k < 4
//                    (zero for boundary or absent slots), s_v = max_k |du_k[v]|
//   x[16 + 4q + v] = d1[q][v] / r_v,  r_v = max_q |d1[q][v]|
//   x[36 + 4q + v] = d2[q][v] / r_v
//   x[56 + 2k + d] = slot k's face centre in the cell's own polynomial frame,
//                    (xi, eta) = Pinv (x_f - c_i)
// Output y[4q + v] = (x* - x2)[q][v] / r_v.  Increments and the remaining error
// are linear in the error of x0 and the sweep acts on each variable alike, so
// this scaling makes the learned map homogeneous of degree one per variable.
// Scales are floored so that a converged or uniform region gives finite features.
#pragma once
#include <cuda_bf16.h>

#include <string>

#include "dndsg_bodies.cuh"

// what a training call reads back, in one copy (a copy of its own for the flags took 3 us per step)
struct MlpResult {
  double loss;
  unsigned flags;  // kFlagTimeout from the tensor-core kernels
};
// a network of the C interface
struct dndsg_mlp {
  int device = 0;
  float *P = nullptr, *M = nullptr, *V = nullptr, *G = nullptr;
  float* part = nullptr;  // per CTA of the training kernel: its gradients and loss [sms][kTrPart], 8.6 MB.  (From the first training
                          // call instead of the creation: that call took 1.2-2.4 ms for 0.6)
  int sms = 148, rows = 0;
  __nv_bfloat16* W = nullptr;
  double* loss = nullptr;     // of an MlpResult
  unsigned* flags = nullptr;  // of the same
  int64_t step = 0;
  bool attrFwd = false, attrTrain = false;
  int featureMode = 0;  // the feature design the network is trained for (dndsg_mlp_set_features)
  std::string err;
};

namespace dg {

constexpr int kIn = 64, kInP = 64, kHid = 64, kOut = 20, kOutP = 32;
// FP32 master parameters, contiguous: W1[64][64] b1[64] W2[64][64] b2[64] W3[64][64] b3[64] W4[32][64] b4[32]
// (W[n][k]: output unit n, input k; padded rows/columns are kept at zero)
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kHid * kInP, kOffW2 = kOffB1 + kHid, kOffB2 = kOffW2 + kHid * kHid,
              kOffW3 = kOffB2 + kHid, kOffB3 = kOffW3 + kHid * kHid, kOffW4 = kOffB3 + kHid,
              kOffB4 = kOffW4 + kOutP * kHid, kNParam = kOffB4 + kOutP;
// BF16 weight copy (the matrices only), same order without biases
constexpr int kWOff1 = 0, kWOff2 = kWOff1 + kHid * kInP, kWOff3 = kWOff2 + kHid * kHid, kWOff4 = kWOff3 + kHid * kHid,
              kNW = kWOff4 + kOutP * kHid;

DG_HD float sigm(float z) {
#if defined(__CUDA_ARCH__)
  return 1.0f / (1.0f + __expf(-z));
#else
  return 1.0f / (1.0f + expf(-z));
#endif
}
DG_HD float silu(float z) { return z * sigm(z); }
DG_HD float silu_grad(float z) {
  float s = sigm(z);
  return s * (1.0f + z * (1.0f - s));
}

// the coefficient iterates the features are taken from
template <class T>
struct MlpIters {
  const T* x0;
  const T* x1;
  const T* x2;
  const float* geom;  // [N][8] slot face centres in each cell's own frame
};

// features of one cell into x[64] and the output scales r[4]
template <class T>
DG_HD void mlp_cell_features(int64_t i, const HotView<T>& h, const MlpIters<T>& it, float x[kInP], float r[4]) {
  double du[4][4], ui[4];
  for (int v = 0; v < 4; v++) ui[v] = h.u[i * 4 + v];
  for (int k = 0; k < 4; k++)
    for (int v = 0; v < 4; v++) du[k][v] = 0.0;
  for (int k = 0; k < h.nfmax && k < 4; k++) {
    if (h.vrMode[aos(i, k, h.nfmax)] != VR_INNER) continue;
    const int64_t j = h.vrNbr[aos(i, k, h.nfmax)];
    for (int v = 0; v < 4; v++) du[k][v] = h.u[j * 4 + v] - ui[v];
  }
  double d1[20], d2[20];
  for (int e = 0; e < 20; e++) {
    const double a = it.x0[i * 20 + e], b = it.x1[i * 20 + e], c = it.x2[i * 20 + e];
    d1[e] = b - a;
    d2[e] = c - b;
  }
  auto clampf = [](double a) { return (float)(a > 1e3 ? 1e3 : (a < -1e3 ? -1e3 : a)); };
  for (int v = 0; v < 4; v++) {
    double m = 0, md = 0;
    for (int k = 0; k < 4; k++) m = dmax(m, fabs(du[k][v]));
    for (int q = 0; q < 5; q++) md = dmax(md, fabs(d1[4 * q + v]));
    const double s = dmax(m, dmax(1e-12 * fabs(ui[v]), 1e-30));
    const double rv = dmax(md, 1e-30);
    r[v] = (float)rv;
    for (int k = 0; k < 4; k++) x[4 * k + v] = clampf(du[k][v] / s);
    for (int q = 0; q < 5; q++) {
      x[16 + 4 * q + v] = clampf(d1[4 * q + v] / (double)r[v]);
      x[36 + 4 * q + v] = clampf(d2[4 * q + v] / (double)r[v]);
    }
  }
  for (int k = 0; k < 8; k++) x[56 + k] = it.geom[i * 8 + k];
}

// The second input design, the one the configuration names: the neighbour mean differences to up to 4
// neighbours and the previous-step coefficients x0 (the coefficients the reconstruction starts from:
// those the previous stage or step left), before any sweep:
//   x[4k + v]      = du_k[v] / s_v   as above
//   x[16 + 4q + v] = x0[q][v] / s_v  (coefficients are mean differences over lengths: the same scale)
//   x[36 .. 55]    = 0
//   x[56 + 2k + d] = slot k's face centre in the cell's own polynomial frame
// Output y[4q + v] = (x* - x0)[q][v] / s_v, returned scales r = s.
template <class T>
DG_HD void mlp_cell_features_prev(int64_t i, const HotView<T>& h, const T* x0, const float* geom, float x[kInP],
                                  float r[4]) {
  double du[4][4], ui[4];
  for (int v = 0; v < 4; v++) ui[v] = h.u[i * 4 + v];
  for (int k = 0; k < 4; k++)
    for (int v = 0; v < 4; v++) du[k][v] = 0.0;
  for (int k = 0; k < h.nfmax && k < 4; k++) {
    if (h.vrMode[aos(i, k, h.nfmax)] != VR_INNER) continue;
    const int64_t j = h.vrNbr[aos(i, k, h.nfmax)];
    for (int v = 0; v < 4; v++) du[k][v] = h.u[j * 4 + v] - ui[v];
  }
  auto clampf = [](double a) { return (float)(a > 1e3 ? 1e3 : (a < -1e3 ? -1e3 : a)); };
  for (int v = 0; v < 4; v++) {
    double m = 0;
    for (int k = 0; k < 4; k++) m = dmax(m, fabs(du[k][v]));
    const double sv = dmax(m, dmax(1e-12 * fabs(ui[v]), 1e-30));
    r[v] = (float)sv;
    for (int k = 0; k < 4; k++) x[4 * k + v] = clampf(du[k][v] / sv);
    for (int q = 0; q < 5; q++) x[16 + 4 * q + v] = clampf((double)x0[i * 20 + 4 * q + v] / sv);
  }
  for (int k = 36; k < 56; k++) x[k] = 0.f;
  for (int k = 0; k < 8; k++) x[56 + k] = geom[i * 8 + k];
}

}  // namespace dg

#if defined(__CUDACC__)
namespace dg {
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

struct MlpDev {
  const float* P;   // FP32 master parameters [kNParam]
  const bf16* W;    // BF16 weight matrices [kNW]
};

// ---------------------------------------------------------------- inference on the tensor cores (tcgen05)
// 128 rows (cells) per tile, one per thread of a 128-thread CTA.  Each layer is one 128 x N x 64
// product, four tcgen05.mma (kind::f16: BF16 operands in shared memory, FP32 accumulator in
// tensor memory, K = 16 each) issued by one thread and completed on an mbarrier; every thread then
// reads its own accumulator row with tcgen05.ld (warp w owns tensor-memory lanes 32w..32w+31, which
// are rows 32w..32w+31 of the 128-row accumulator), adds the bias, applies SiLU and writes the next
// layer's operand row.  Operands use the K-major, no-swizzle canonical layout: 8-row x 16-byte core
// matrices, core matrices along K 128 B apart (leading byte offset), 8-row groups 1024 B apart
// (stride byte offset), so the K step k0 of an instruction starts 32 k0 / 16 bytes further.
constexpr int kTcRows = 128;
constexpr int kTcCols = 64;  // tensor-memory columns: the widest layer (N = 64, FP32)
// The forward operands have K = 80: 64 inputs and 16 more columns, of which three carry the bias.  The
// activation rows hold ones there and the weight rows the bias as three BF16 numbers that sum to it exactly
// (24 bits), so the accumulator comes out with the bias in.  The weights and biases of the SiLU layers are
// halved (exact): the accumulator is w = z / 2 and SiLU(z) = w + w tanh(w).  Per activation the epilogue is
// then one special-function operation, one multiply-add and half a conversion, where it had three more
// operations and a shared-memory load; it is what bounds this kernel.
constexpr int kTcK = 80;
struct TcSmem {
  alignas(128) unsigned char W[3 * kHid * kTcK * 2 + kOutP * kTcK * 2];  // W1..W4, core-matrix layout
  alignas(128) unsigned char A[kTcRows * kTcK * 2];                      // the current layer's input rows, same layout
  uint64_t bar;
  uint32_t tmem;
};

// tensor memory: every resident CTA holds kTcCols of the SM's 512 columns, and an allocation that
// cannot be met waits; the launch keeps at most 4 CTAs per SM (shared memory and registers allow 4)
static_assert(sizeof(TcSmem) > 233472 / 9, "at most 8 CTAs of k_mlp_tc per SM");
static_assert(4 * (sizeof(TcSmem) + 1024) <= 233472, "4 CTAs of k_mlp_tc per SM");

// the bias of layer l, entry k, from the FP32 master parameters
__device__ __forceinline__ float tc_bias_s(const float* P, int layer, int k) {
  const int off = layer == 0 ? kOffB1 : layer == 1 ? kOffB2 : layer == 2 ? kOffB3 : kOffB4;
  return P[off + k];
}

// byte offset of element (row, k) of a K-major operand in the core-matrix layout: 64 wide (training) and
// kTcK wide (inference)
__device__ __forceinline__ uint32_t cm_off(int row, int k) {
  return (uint32_t)((row >> 3) * 1024 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}
__device__ __forceinline__ uint32_t cm_off_k(int row, int k) {
  return (uint32_t)((row >> 3) * (kTcK * 16) + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}
// shared-memory matrix descriptor: start address, leading byte offset 128, stride byte offset 1024 (kTcK
// wide: 1280), descriptor version 1, no swizzle (all addresses and offsets in 16-byte units)
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
         (1ull << 46);
}
__device__ __forceinline__ uint64_t umma_desc_k(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(kTcK * 16 >> 4) << 32) |
         (1ull << 46);
}
// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M = 128, N
__host__ __device__ constexpr uint32_t umma_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTcRows >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 16 consecutive FP32 columns of this thread's accumulator row
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
  for (int k = 0; k < 16; k++) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// SiLU(z) from w = z / 2 through sigmoid(z) = (1 + tanh(z / 2)) / 2 with the hardware tanh: one
// special-function operation per activation instead of an exponential and a reciprocal.  The relative error of
// that tanh, at most 2^-11, is an absolute one of |z| 2^-12 here.  That is below the BF16 rounding the
// activation gets next (2^-9 of it) down to z = -2; further down 1 + tanh cancels and the small negative tail loses
// relative accuracy (1% at z = -4), where the training kernel's exponential does not
__device__ __forceinline__ float silu_half(float w) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(w));
  return fmaf(w, t, w);
}
__device__ __forceinline__ uint4 pack8(const float* x) {
  __nv_bfloat162 p[4];
  for (int e = 0; e < 4; e++) p[e] = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
  return *reinterpret_cast<uint4*>(p);
}

// inputs and outputs of the tensor-core forward
// Src::kTile: the whole tile is loaded by the CTA together (coalesced), a tile ahead; else row by row
struct TcFeaturesX {  // given features X [n][64]
  static constexpr bool kTile = true;
  const float* X;
  // this thread's sixteenth of the 128 x 64 tile starting at row r0: 32 B of X per step
  __device__ void fetch_tile(int64_t r0, int64_t n, float4 v[16]) const {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int e = threadIdx.x + j * kTcRows, row = e >> 3, kc = e & 7;
      v[2 * j] = v[2 * j + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r0 + row < n) {
        const float4* q = reinterpret_cast<const float4*>(X + (r0 + row) * kIn + 8 * kc);
        v[2 * j] = q[0];
        v[2 * j + 1] = q[1];
      }
    }
  }
  __device__ void put_tile(const float4 v[16], unsigned char* A) const {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int e = threadIdx.x + j * kTcRows;
      *reinterpret_cast<uint4*>(A + cm_off_k(e >> 3, 8 * (e & 7))) = pack8(&v[2 * j].x);
    }
  }
  __device__ void load(int64_t, int64_t, float*, float*) const {}
};
struct TcOutY {  // Y [n][20] = the network output
  float* Y;
  __device__ void store(int64_t r, int64_t n, const float* y, const float*) const {
    if (r >= n) return;
    float* o = Y + r * kOut;
    if ((reinterpret_cast<uintptr_t>(Y) & 15u) == 0) {
#pragma unroll
      for (int k = 0; k < kOut; k += 4) *reinterpret_cast<float4*>(o + k) = make_float4(y[k], y[k + 1], y[k + 2], y[k + 3]);
    } else {
      for (int k = 0; k < kOut; k++) o[k] = y[k];
    }
  }
};
template <class T, int MODE>
struct TcCellFeatures {  // the warm-start features of cell r (MODE 0: Jacobi extrapolation, 1: previous coefficients)
  static constexpr bool kTile = false;
  HotView<T> h;
  MlpIters<T> it;
  __device__ void load(int64_t r, int64_t n, float x[kInP], float sc[4]) const {
    if (r < n) {
      if (MODE == 0) mlp_cell_features<T>(r, h, it, x, sc);
      else mlp_cell_features_prev<T>(r, h, it.x0, it.geom, x, sc);
    } else {
      for (int k = 0; k < kInP; k++) x[k] = 0.f;
      for (int v = 0; v < 4; v++) sc[v] = 0.f;
    }
  }
  __device__ void fetch_tile(int64_t, int64_t, float4*) const {}
  __device__ void put_tile(const float4*, unsigned char*) const {}
};
template <class T>
struct TcWarmStart {  // dst = base + y r (base: x2 for MODE 0, x0 for MODE 1)
  const T* x2;
  T* dst;
  __device__ void store(int64_t r, int64_t n, const float* y, const float* sc) const {
    if (r < n)
      for (int o = 0; o < kOut; o++) dst[r * 20 + o] = (T)((double)x2[r * 20 + o] + (double)y[o] * (double)sc[o & 3]);
  }
};

template <class Src, class Dst>
__global__ void __launch_bounds__(kTcRows, 4) k_mlp_tc(MlpDev m, Src src, Dst dst, int64_t n, unsigned* flags) {
  extern __shared__ __align__(128) unsigned char raw[];
  TcSmem& S = *reinterpret_cast<TcSmem*>(raw);
  const int tid = threadIdx.x, warp = tid >> 5;
  // the weights (row-major [N][64] BF16 in global memory) into the core-matrix layout, 16 B at a time, halved in
  // front of a SiLU; then the bias columns
  constexpr int kLayerBytes = kHid * kTcK * 2;
  for (int e = tid; e < (3 * kHid + kOutP) * 8; e += blockDim.x) {
    const int row = e >> 3, kc = e & 7;
    const int layer = row < 3 * kHid ? row / kHid : 3, rl = row - layer * kHid;
    const int woff = layer == 0 ? kWOff1 : layer == 1 ? kWOff2 : layer == 2 ? kWOff3 : kWOff4;
    uint4 q = *reinterpret_cast<const uint4*>(m.W + woff + rl * 64 + 8 * kc);
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
    if (layer < 3)
      for (int k = 0; k < 4; k++) h[k] = __hmul2(h[k], __float2bfloat162_rn(0.5f));
    *reinterpret_cast<uint4*>(S.W + layer * kLayerBytes + cm_off_k(rl, 8 * kc)) = q;
  }
  for (int row = tid; row < 3 * kHid + kOutP; row += blockDim.x) {
    const int layer = row < 3 * kHid ? row / kHid : 3, rl = row - layer * kHid;
    float bias = tc_bias_s(m.P, layer, rl) * (layer < 3 ? 0.5f : 1.0f);
    float c[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int k = 0; k < 3; k++) {
      float h = __bfloat162float(__float2bfloat16(bias));
      if (isinf(h) && !isinf(bias)) h = __bfloat162float(__float2bfloat16_rz(bias));  // above the largest BF16 number
      c[k] = h;
      bias = isinf(h) ? 0.f : bias - h;
    }
    unsigned char* w = S.W + layer * kLayerBytes;
    *reinterpret_cast<uint4*>(w + cm_off_k(rl, 64)) = pack8(c);
    *reinterpret_cast<uint4*>(w + cm_off_k(rl, 72)) = make_uint4(0, 0, 0, 0);
  }
  {
    const float ones[8] = {1.f, 1.f, 1.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    *reinterpret_cast<uint4*>(S.A + cm_off_k(tid, 64)) = pack8(ones);
    *reinterpret_cast<uint4*>(S.A + cm_off_k(tid, 72)) = make_uint4(0, 0, 0, 0);
  }
  const uint32_t bar = smem_u32(&S.bar);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                 "r"(kTcCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = S.tmem, trow = tbase + ((uint32_t)(warp * 32) << 16);
  const uint32_t aAddr = smem_u32(S.A), wAddr = smem_u32(S.W);
  uint32_t phase = 0;
  bool failed = false, stop = false;
  float4 next[16];
  if constexpr (Src::kTile) src.fetch_tile((int64_t)blockIdx.x * kTcRows, n, next);
  for (int64_t tile = blockIdx.x; tile * kTcRows < n && !stop; tile += gridDim.x) {
    const int64_t r = tile * kTcRows + tid;
    float sc[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (Src::kTile) {
      src.put_tile(next, S.A);
    } else {
      float x[kInP];
      src.load(r, n, x, sc);
      for (int kc = 0; kc < 8; kc++) *reinterpret_cast<uint4*>(S.A + cm_off_k(tid, 8 * kc)) = pack8(x + 8 * kc);
    }
#pragma unroll
    for (int layer = 0; layer < 4; layer++) {
      proxy_fence_smem();  // the operand rows written by this thread, to the tensor cores
      tc_fence_before();   // and its accumulator reads, before the next product
      stop = __syncthreads_or(failed);
      if (stop) break;
      if (tid == 0) {
        tc_fence_after();
        for (int ks = 0; ks < kTcK / 16; ks++)
          umma_bf16(tbase, umma_desc_k(aAddr + 256 * ks), umma_desc_k(wAddr + layer * kLayerBytes + 256 * ks),
                    layer < 3 ? umma_idesc(kHid) : umma_idesc(kOutP), ks > 0);
        umma_commit(bar);
      }
      if constexpr (Src::kTile)
        if (layer == 2) src.fetch_tile((tile + gridDim.x) * kTcRows, n, next);
      failed = !mbar_wait(bar, phase, kWaitLimit);
      phase ^= 1u;
      tc_fence_after();
      if (layer < 3) {
#pragma unroll
        for (int c0 = 0; c0 < kHid; c0 += 32) {
          float z[32];
          tmem_ld16(trow + c0, z);
          tmem_ld16(trow + c0 + 16, z + 16);
          tmem_wait_ld();
          for (int k = 0; k < 32; k++) z[k] = silu_half(z[k]);
          for (int kc = 0; kc < 4; kc++) *reinterpret_cast<uint4*>(S.A + cm_off_k(tid, c0 + 8 * kc)) = pack8(z + 8 * kc);
        }
      } else {
        float z[32];
        tmem_ld16(trow, z);
        tmem_ld16(trow + 16, z + 16);
        tmem_wait_ld();
        if (!failed) dst.store(r, n, z, sc);
      }
    }
  }
  if (failed) atomicOr(flags, kFlagTimeout);
  tc_fence_before();
  if (__syncthreads_or(failed)) {  // the last commit may still be in flight
    if (tid == 0) mbar_wait(bar, phase ^ 1u, kWaitLimit);
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(kTcCols) : "memory");
  }
}

// loss = mean over rows and the 20 outputs of (y - t)^2; gradients accumulate into G
// ---------------------------------------------------------------- training on the tensor cores (tcgen05)
// 128 rows per tile.  A tile is a chain of eight products with an epilogue after each, so one CTA per SM keeps
// two tiles in flight: two groups of 256 threads (row 32 (warp % 4) + lane, columns 32 (warp / 4 % 2) .. + 31)
// work on a tile each, and one thread of a 17th warp issues the products of both, in the order in which the
// groups' operands get ready (a group arrives on its `ready` barrier, the product commits to its `done`
// barrier; no barrier of the whole block inside a tile).  All 512 tensor-memory columns:
//   cols 128 g + 0-63    pre-activations z of group g's current layer (recomputed for the backward pass from the
//                        stored operand: a product more instead of 128 columns for z1..z3)
//   cols 128 g + 64-127  group g's backward product dH = dz W
//   cols 256-511         dW1 .. dW4, accumulated over all of the CTA's tiles (M = 64: output unit u in
//                        tensor-memory lane (u & 15) + 32 (u >> 4), the half-subpartition layout of M = 64)
// Every operand stays in the one layout it is written in, the K-major core-matrix layout of the forward
// products ([rows][64 units], cm_off); the products that need an operand transposed read it as an
// MN-major operand instead (the same bytes: MN-blocks of 8 units 128 B apart, K-blocks of 8 rows 1024 B
// apart), so nothing is copied transposed:
//   forward       z_l  = h_{l-1} W_l^T       A h_{l-1} K-major, B W_l K-major         M 128, N 64 | 32, K 64
//   input grad    dH   = dz_l W_l            A dz_l K-major,    B W_l MN-major         M 128, N 64, K 64 | 32
//   weight grad   dW_l += dz_l^T h_{l-1}     A dz_l MN-major,   B h_{l-1} MN-major     M 64, N 64, K 128
constexpr int kTrCols = 512, kTrGroups = 2, kTrGroup = 256;  // threads of a group
constexpr int kTrThreads = kTrGroups * kTrGroup + 32;
struct TrTcSmem {
  alignas(128) unsigned char Wf[3 * kHid * 128 + kOutP * 128];  // W_l [N][64], core-matrix layout
  struct Tile {
    alignas(128) unsigned char X[kTcRows * 128];     // the tile's features [128][64]
    alignas(128) unsigned char H[3][kTcRows * 128];  // h1, h2, h3 [128][64]
    alignas(128) unsigned char DZ[kTcRows * 128];    // dz_l [128][64] (dz4: units >= 32 zero)
  } t[kTrGroups];
  alignas(16) float b[3 * kHid + kOutP];  // biases
  float gb[3 * kHid + kOutP];             // bias gradients of the CTA
  uint64_t ready[kTrGroups], done[kTrGroups];
  uint32_t tmem;
};
static_assert(sizeof(TrTcSmem) > 233472 / 2 && sizeof(TrTcSmem) <= 227 * 1024, "one CTA per SM: it holds all 512 tensor-memory columns");

// MN-major shared-memory descriptor of the same core-matrix layout: leading byte offset (K-blocks of 8 rows)
// 1024, stride byte offset (MN-blocks of 8 units) 128, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(1024 >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
         (1ull << 46);
}
// instruction descriptor of kind::f16 with the operands' majors (a_major bit 15, b_major bit 16) and M
__host__ __device__ constexpr uint32_t umma_idesc_mk(int m, int n, bool aMN, bool bMN) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (aMN ? (1u << 15) : 0u) | (bMN ? (1u << 16) : 0u) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
// one butterfly round of a 16-column warp sum: lanes L and L ^ O trade halves of their W columns, each
// keeping the half its bit O selects, summed with the partner's copy of the same columns
template <int W, int O>
__device__ __forceinline__ void tr_bfly(float* v, int lane) {
  const bool up = (lane & O) != 0;
#pragma unroll
  for (int k = 0; k < W; k++) {
    const float send = up ? v[k] : v[k + W], keep = up ? v[k + W] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, O);
  }
}
// the sums over the warp's 32 rows of 16 column values v (destroyed): four butterfly rounds halve the
// columns a lane holds (8 + 4 + 2 + 1 shuffles, against 5 per column for 16 separate reductions), a last one
// completes the sum; the lane returns that of column tr_sum_col(lane)
__device__ __forceinline__ float tr_sum16(float* v, int lane) {
  tr_bfly<8, 16>(v, lane);
  tr_bfly<4, 8>(v, lane);
  tr_bfly<2, 4>(v, lane);
  tr_bfly<1, 2>(v, lane);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}
__device__ __forceinline__ int tr_sum_col(int lane) {
  return ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
}
// whether an mbarrier phase is complete, without waiting
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// 32 values of a row, as BF16, into columns c0 .. c0 + 31 of a 64-wide K-major operand (c0 % 8 == 0)
__device__ __forceinline__ void tc_store32(unsigned char* A, int row, int c0, const float* x) {
#pragma unroll
  for (int h = 0; h < 4; h++) *reinterpret_cast<uint4*>(A + cm_off(row, c0 + 8 * h)) = pack8(x + 8 * h);
}

// Each CTA writes its gradients and loss to a row of `part` [gridDim][kTrPart], which k_mlp_adam or
// k_mlp_reduce sums in row order (atomic adds of 148 CTAs to the same 14,560 addresses took longer).  Within a CTA
// the order is not fixed: the bias gradients of 16 warps meet in shared-memory atomics, and the weight gradients of the
// two groups' tiles accumulate in the order in which the tiles get ready.
// Measured, eight steps of 65,536 rows: 954 us with one tile in flight per SM and atomics, 790 us with two
// tiles, 579 us with the rows; a step of 1,048,576 rows 1.10 ms -> 0.65 ms.
constexpr int kTrPart = kNParam + 4;  // parameters' gradients, then the loss as a double, and padding to 16 bytes
static_assert(kNParam % 2 == 0 && kTrPart % 4 == 0, "the loss and every row are aligned");
__global__ void __launch_bounds__(kTrThreads, 1) k_mlp_train_tc(MlpDev m, const float* X, const float* Tg, int64_t n,
                                                                float invCount, float* part, unsigned* flags) {
  extern __shared__ __align__(128) unsigned char raw[];
  TrTcSmem& S = *reinterpret_cast<TrTcSmem*>(raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // the weights (row-major [N][64] BF16 in global memory) into the core-matrix layout, 16 B at a time
  for (int e = tid; e < (3 * kHid + kOutP) * 8; e += blockDim.x) {
    const int row = e >> 3, kc = e & 7;
    const int layer = row < 3 * kHid ? row / kHid : 3, rl = row - layer * kHid;
    const int woff = layer == 0 ? kWOff1 : layer == 1 ? kWOff2 : layer == 2 ? kWOff3 : kWOff4;
    *reinterpret_cast<uint4*>(S.Wf + layer * kHid * 128 + cm_off(rl, 8 * kc)) =
        *reinterpret_cast<const uint4*>(m.W + woff + rl * 64 + 8 * kc);
  }
  for (int e = tid; e < 3 * kHid + kOutP; e += blockDim.x) {
    S.gb[e] = 0.f;
    S.b[e] = tc_bias_s(m.P, e < 3 * kHid ? e / kHid : 3, e < 3 * kHid ? e % kHid : e - 3 * kHid);
  }
  if (warp == kTrGroups * kTrGroup / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                 "r"(kTrCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int g = 0; g < kTrGroups; g++) {
      mbar_init(smem_u32(&S.ready[g]), kTrGroup / 32);
      mbar_init(smem_u32(&S.done[g]), 1);
    }
    fence_mbar_init();
  }
  proxy_fence_smem();  // the weights, to the tensor cores
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tb = S.tmem;
  const int64_t tiles = (n + kTcRows - 1) / kTcRows, slots = (int64_t)kTrGroups * gridDim.x;
  bool failed = false;
  double lossLocal = 0.0;
  if (warp == kTrGroups * kTrGroup / 32) {
    // ---- the products of both groups.  Steps of a tile: 0-3 forward; 4-7 backward of layers 3..0: dW_l, dH and
    // the previous layer's z again
    if (lane == 0) {
      constexpr uint32_t idFwd64 = umma_idesc_mk(kTcRows, kHid, false, false);
      constexpr uint32_t idFwd32 = umma_idesc_mk(kTcRows, kOutP, false, false);
      constexpr uint32_t idDH = umma_idesc_mk(kTcRows, kHid, false, true);
      constexpr uint32_t idDW = umma_idesc_mk(64, kHid, true, true);
      const uint32_t aW = smem_u32(S.Wf);
      int64_t step[kTrGroups], steps[kTrGroups];
      for (int g = 0; g < kTrGroups; g++) {
        const int64_t first = blockIdx.x + (int64_t)g * gridDim.x;
        step[g] = 0;
        steps[g] = first < tiles ? 8 * ((tiles - first + slots - 1) / slots) : 0;
      }
      unsigned started = 0;  // layers whose dW holds something
      uint32_t idle = 0;
      while (step[0] < steps[0] || step[1] < steps[1]) {
        for (int g = 0; g < kTrGroups; g++) {
          if (step[g] >= steps[g] || !mbar_test(smem_u32(&S.ready[g]), (uint32_t)step[g] & 1u)) continue;
          tc_fence_after();
          const uint32_t aX = smem_u32(S.t[g].X), aH = smem_u32(S.t[g].H[0]), aDZ = smem_u32(S.t[g].DZ);
          const uint32_t z = tb + 128u * g;
          constexpr uint32_t kOp = kTcRows * 128;
          const int k = (int)(step[g] & 7);
          const int f = k < 4 ? k : 6 - k;  // the layer whose z is formed (-1: none)
          if (k >= 4) {
            const int l = 7 - k;
            const uint32_t aPrev = l > 0 ? aH + (l - 1) * kOp : aX, aWl = aW + (uint32_t)l * kHid * 128;
            const bool acc = started >> l & 1u;
            started |= 1u << l;
            for (int ks = 0; ks < kTcRows / 16; ks++)
              umma_bf16(tb + 256 + 64u * l, umma_desc_mn(aDZ + 2048 * ks), umma_desc_mn(aPrev + 2048 * ks), idDW, acc || ks > 0);
            if (l > 0) {
              const int kst = l == 3 ? kOutP / 16 : kHid / 16;  // K = the layer's output units
              for (int ks = 0; ks < kst; ks++)
                umma_bf16(z + 64, umma_desc(aDZ + 256 * ks), umma_desc_mn(aWl + 2048 * ks), idDH, ks > 0);
            }
          }
          if (f >= 0) {
            const uint32_t aIn = f > 0 ? aH + (f - 1) * kOp : aX, aWf = aW + (uint32_t)f * kHid * 128;
            for (int ks = 0; ks < 4; ks++)
              umma_bf16(z, umma_desc(aIn + 256 * ks), umma_desc(aWf + 256 * ks), f < 3 ? idFwd64 : idFwd32, ks > 0);
          }
          umma_commit(smem_u32(&S.done[g]));
          step[g]++;
          idle = 0;
        }
        if (++idle == kWaitLimit) {
          failed = true;
          break;
        }
      }
      for (int g = 0; g < kTrGroups; g++)  // nothing in flight when the block leaves
        if (step[g] > 0) mbar_wait(smem_u32(&S.done[g]), (uint32_t)(step[g] - 1) & 1u, kWaitLimit);
    }
    __syncwarp();
  } else {
    const int grp = tid / kTrGroup, gt = tid % kTrGroup, q = warp & 3, half = (gt >> 5) >> 2, row = 32 * q + lane, c0 = 32 * half;
    TrTcSmem::Tile& T = S.t[grp];
    const uint32_t ready = smem_u32(&S.ready[grp]), done = smem_u32(&S.done[grp]);
    const uint32_t tz = tb + 128u * grp + ((uint32_t)(q * 32) << 16) + c0;
    uint32_t phase = 0;
    float bsum[4][2] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};  // bias gradients of this lane's columns
    // operands written: hand over to the tensor cores and wait for the product
    auto product = [&]() {
      proxy_fence_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ready) : "memory");
    };
    auto wait = [&]() {
      if (!failed) failed = !mbar_wait(done, phase, kWaitLimit);
      phase ^= 1u;
      failed = __any_sync(0xffffffffu, failed);
      tc_fence_after();
    };
    // 32 B of X per step: chunk e = gt + 256 j of the tile (row e / 8, columns 8 (e % 8) .. + 7), loaded a tile ahead
    float4 nx[8];
    auto fetch = [&](int64_t r0) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int e = gt + j * kTrGroup, rw = e >> 3, kc = e & 7;
        nx[2 * j] = nx[2 * j + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r0 + rw < n) {
          const float4* p = reinterpret_cast<const float4*>(X + (r0 + rw) * kIn + 8 * kc);
          nx[2 * j] = p[0];
          nx[2 * j + 1] = p[1];
        }
      }
    };
    int64_t tile = blockIdx.x + (int64_t)grp * gridDim.x;
    if (tile < tiles) fetch(tile * kTcRows);
    for (; tile < tiles && !failed; tile += slots) {
      const int64_t r = tile * kTcRows + row;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int e = gt + j * kTrGroup;
        *reinterpret_cast<uint4*>(T.X + cm_off(e >> 3, 8 * (e & 7))) = pack8(&nx[2 * j].x);
      }
      product();
      float v[32];
      // ---- forward: h_l = SiLU(z_l + b_l) into H[l]
#pragma unroll
      for (int l = 0; l < 3; l++) {
        wait();
        tmem_ld16(tz, v);
        tmem_ld16(tz + 16, v + 16);
        tmem_wait_ld();
        for (int k = 0; k < 32; k += 4) {
          const float4 b = *reinterpret_cast<const float4*>(&S.b[l * kHid + c0 + k]);
          v[k] = silu(v[k] + b.x);
          v[k + 1] = silu(v[k + 1] + b.y);
          v[k + 2] = silu(v[k + 2] + b.z);
          v[k + 3] = silu(v[k + 3] + b.w);
        }
        tc_store32(T.H[l], row, c0, v);
        product();
      }
      // ---- y = z4 + b4, dz4 = 2 (y - t) / count on the 20 outputs (columns below 32)
      float tg[kOut];
      if (half == 0)
        for (int k = 0; k < kOut; k += 4) {
          float4 t4 = make_float4(0.f, 0.f, 0.f, 0.f);
          if (r < n) {
            const float* p = Tg + r * kOut + k;
            if ((reinterpret_cast<uintptr_t>(Tg) & 15u) == 0) t4 = *reinterpret_cast<const float4*>(p);
            else t4 = make_float4(p[0], p[1], p[2], p[3]);
          }
          tg[k] = t4.x; tg[k + 1] = t4.y; tg[k + 2] = t4.z; tg[k + 3] = t4.w;
        }
      wait();
      if (half == 0) {
        tmem_ld16(tz, v);
        tmem_ld16(tz + 16, v + 16);
        tmem_wait_ld();
        for (int k = 0; k < 32; k++) {
          if (k < kOut && r < n) {
            const float dd = v[k] + S.b[3 * kHid + k] - tg[k < kOut ? k : 0];
            lossLocal += (double)dd * dd;
            v[k] = 2.f * dd * invCount;
          } else {
            v[k] = 0.f;
          }
        }
      } else {
        for (int k = 0; k < 32; k++) v[k] = 0.f;  // units 32 .. 63 stay zero
      }
      tc_store32(T.DZ, row, c0, v);
      product();
      if (half == 0) {
        bsum[3][0] += tr_sum16(v, lane);
        bsum[3][1] += tr_sum16(v + 16, lane);
      }
      // ---- backward: dz_{l-1} = dH SiLU'(z_{l-1} + b_{l-1})
#pragma unroll
      for (int l = 3; l > 0; l--) {
        if (l == 1) fetch((tile + slots) * kTcRows);
        wait();
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          float z[16];
          tmem_ld16(tz + 64 + h, v + h);
          tmem_ld16(tz + h, z);
          tmem_wait_ld();
#pragma unroll
          for (int k = 0; k < 16; k += 4) {
            const float4 b = *reinterpret_cast<const float4*>(&S.b[(l - 1) * kHid + c0 + h + k]);
            v[h + k] = r < n ? v[h + k] * silu_grad(z[k] + b.x) : 0.f;
            v[h + k + 1] = r < n ? v[h + k + 1] * silu_grad(z[k + 1] + b.y) : 0.f;
            v[h + k + 2] = r < n ? v[h + k + 2] * silu_grad(z[k + 2] + b.z) : 0.f;
            v[h + k + 3] = r < n ? v[h + k + 3] * silu_grad(z[k + 3] + b.w) : 0.f;
          }
        }
        tc_store32(T.DZ, row, c0, v);
        product();
        bsum[l - 1][0] += tr_sum16(v, lane);
        bsum[l - 1][1] += tr_sum16(v + 16, lane);
      }
      wait();  // dW_1: the tile's operands are free
    }
    if ((lane & 1) == 0)
#pragma unroll
      for (int l = 0; l < 4; l++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (l < 3 || half == 0) atomicAdd(&S.gb[l * kHid + c0 + 16 * h + tr_sum_col(lane)], bsum[l][h]);
  }
  if (failed) atomicOr(flags, kFlagTimeout);
  tc_fence_before();
  const bool bad = __syncthreads_or(failed);
  tc_fence_after();
  // the CTA's weight gradients and bias gradients: dW_l unit u = 16 q + t in lane t < 16 of the warps of lane
  // quarter q, columns 16 g .. 16 g + 15
  float* row = part + (int64_t)blockIdx.x * kTrPart;
  __shared__ double lossW[kTrThreads / 32];
  lossLocal = warp_sum_d(lossLocal);
  if (lane == 0) lossW[warp] = lossLocal;
  __syncthreads();
  if (tid == 0) {
    double t = 0;
    for (int w = 0; w < kTrThreads / 32; w++) t += lossW[w];
    *reinterpret_cast<double*>(row + kNParam) = t;
  }
  if (bad)  // after a timeout: a defined row
    for (int e = tid; e < kNParam; e += kTrThreads) row[e] = 0.f;
  if (!bad && warp < 16) {
    const int q = warp & 3, col0 = 16 * (warp >> 2), u = 16 * q + lane;
    const bool mine = lane < 16;
    for (int l = 0; l < 4; l++) {
      const int N = l < 3 ? kHid : kOutP;
      const int woff = l == 0 ? kOffW1 : l == 1 ? kOffW2 : l == 2 ? kOffW3 : kOffW4;
      float gv[16];
      tmem_ld16(tb + ((uint32_t)(q * 32) << 16) + 256 + 64u * l + col0, gv);
      tmem_wait_ld();
      if (mine && u < N)
        for (int k = 0; k < 16; k += 4)
          *reinterpret_cast<float4*>(&row[woff + u * 64 + col0 + k]) = make_float4(gv[k], gv[k + 1], gv[k + 2], gv[k + 3]);
    }
    for (int e = tid; e < 3 * kHid + kOutP; e += kTrGroups * kTrGroup) {
      const int off = e < kHid ? kOffB1 + e : e < 2 * kHid ? kOffB2 + e - kHid : e < 3 * kHid ? kOffB3 + e - 2 * kHid
                                                                                            : kOffB4 + e - 3 * kHid;
      row[off] = S.gb[e];
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kTrGroups * kTrGroup / 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(kTrCols) : "memory");
  }
}

// sum over the rows of `part` of entry e: 4 threads per entry (a block of 256: 64 entries), each over a
// quarter of the rows, added in order; valid in the entry's first thread
constexpr int kRedEntries = 64;
__device__ __forceinline__ float tr_sum_rows(const float* part, int rows, int e, float (*sh)[kRedEntries]) {
  const int k = threadIdx.x / kRedEntries, x = threadIdx.x % kRedEntries;
  float a = 0.f;
  if (e < kNParam)
    for (int b = k * rows / 4; b < (k + 1) * rows / 4; b++) a += part[(int64_t)b * kTrPart + e];
  sh[k][x] = a;
  __syncthreads();
  return (sh[0][x] + sh[1][x]) + (sh[2][x] + sh[3][x]);
}
// the loss, by one warp
__device__ __forceinline__ void tr_sum_loss(const float* part, int rows, double* loss) {
  double t = 0;
  for (int b = threadIdx.x & 31; b < rows; b += 32) t += *reinterpret_cast<const double*>(&part[(int64_t)b * kTrPart + kNParam]);
  t = warp_sum_d(t);
  if ((threadIdx.x & 31) == 0) *loss = t;
}
__global__ void __launch_bounds__(256) k_mlp_reduce(const float* part, int rows, float* G, double* loss) {
  __shared__ float sh[4][kRedEntries];
  const int e = blockIdx.x * kRedEntries + threadIdx.x % kRedEntries;
  const float g = tr_sum_rows(part, rows, e, sh);
  if (threadIdx.x < kRedEntries && e < kNParam) G[e] = g;
  if (blockIdx.x == 0 && threadIdx.x / 32 == 7) tr_sum_loss(part, rows, loss);
}
// Adam (Kingma & Ba) on the FP32 master parameters, from the rows of gradients; padded entries stay zero;
// refreshes the BF16 copy.  Nothing changes once a wait of this network ran out (flags): the gradient is then not one
__global__ void __launch_bounds__(256) k_mlp_adam(float* P, float* Mo, float* V, const float* part, int rows, double* loss, bf16* W,
                                                  const unsigned* flags, float lr, float b1, float b2, float eps, float c1, float c2) {
  __shared__ float sh[4][kRedEntries];
  const int e = blockIdx.x * kRedEntries + threadIdx.x % kRedEntries;
  const float g = tr_sum_rows(part, rows, e, sh);
  if (blockIdx.x == 0 && threadIdx.x / 32 == 7) tr_sum_loss(part, rows, loss);
  if (threadIdx.x >= kRedEntries || e >= kNParam) return;
  const float m0 = Mo[e], v0 = V[e], p0 = P[e];  // and the flag, one wait for all (read before the rows it took 2 us per step)
  if (*flags) return;
  bool pad = false;
  int wi = -1;
  if (e < kOffB1) { pad = (e % kInP) >= kIn; wi = kWOff1 + e; }
  else if (e >= kOffW2 && e < kOffB2) wi = kWOff2 + (e - kOffW2);
  else if (e >= kOffW3 && e < kOffB3) wi = kWOff3 + (e - kOffW3);
  else if (e >= kOffW4 && e < kOffB4) { pad = (e - kOffW4) / kHid >= kOut; wi = kWOff4 + (e - kOffW4); }
  else if (e >= kOffB4) pad = (e - kOffB4) >= kOut;
  if (pad) { P[e] = 0.f; if (wi >= 0) W[wi] = __float2bfloat16(0.f); return; }
  const float m = b1 * m0 + (1.f - b1) * g, v = b2 * v0 + (1.f - b2) * g * g;
  Mo[e] = m;
  V[e] = v;
  const float p = p0 - lr * (m * c1) / (sqrtf(v * c2) + eps);
  P[e] = p;
  if (wi >= 0) W[wi] = __float2bfloat16(p);
}
__global__ void k_mlp_to_bf16(const float* P, bf16* W) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= kNParam) return;
  int wi = -1;
  if (e < kOffB1) wi = kWOff1 + e;
  else if (e >= kOffW2 && e < kOffB2) wi = kWOff2 + (e - kOffW2);
  else if (e >= kOffW3 && e < kOffB3) wi = kWOff3 + (e - kOffW3);
  else if (e >= kOffW4 && e < kOffB4) wi = kWOff4 + (e - kOffW4);
  if (wi >= 0) W[wi] = __float2bfloat16(P[e]);
}

}  // namespace dg
#endif
