// Training and inference kernels of the learned Steiner placement network
// (no counterpart in the reference), and their C ABI.
//
// One block carries 32 rows through the network, forward and back, with bf16
// operands on the tensor cores and fp32 accumulation.  The weight gradients of
// 32 rows go to their own slice of a partial-gradient buffer (no atomics, so
// the sum is deterministic); the slices are summed in order, and Adam updates
// the fp32 master parameters and their bf16 copies.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <random>
#include <vector>

#include "../../include/gqm_refine.h"
#include "learned.cuh"
#include "team.cuh"

namespace gqm {
namespace {

// One block carries 32 rows (a group) forward and back: kGroupWarps warps share
// the tiles of every product.
constexpr int kGroupWarps = 8, kGroupThreads = 32 * kGroupWarps;
// rows padded by 8 bf16, so that the fragment loads of a warp hit 32 distinct banks
constexpr int kHStride = kHid + 8;
struct GroupSmem {
  MlpWSmem w;
  uint16_t x[32 * kXStride];
  uint16_t a1[32 * kHStride], a2[32 * kHStride], dz2[32 * kHStride], dz1[32 * kHStride];
  float dy[32];
  int row[32];
};

// One 16 x 8 tile of C = A B by a warp: A(i,k) = a[i*ai + k*ak], B(k,j) =
// b[k*bk + j*bj], K a multiple of 16; the accumulator fragment in d (lane =
// 4 g + q holds (g, 2q), (g, 2q+1), (g+8, 2q), (g+8, 2q+1)).
__device__ __forceinline__ void tile_gemm(int K, const uint16_t *a, int ai, int ak, const uint16_t *b, int bk, int bj,
                                          float *d) {
  const int lane = (int)(threadIdx.x & 31u), g = lane >> 2, q = lane & 3;
  d[0] = d[1] = d[2] = d[3] = 0.0f;
  for (int k0 = 0; k0 < K; k0 += 16) {
    const uint16_t *A = a + k0 * ak;
    const uint16_t *B = b + k0 * bk;
    uint32_t ra[4], rb[2];
    ra[0] = pack2(A[g * ai + (2 * q) * ak], A[g * ai + (2 * q + 1) * ak]);
    ra[1] = pack2(A[(g + 8) * ai + (2 * q) * ak], A[(g + 8) * ai + (2 * q + 1) * ak]);
    ra[2] = pack2(A[g * ai + (2 * q + 8) * ak], A[g * ai + (2 * q + 9) * ak]);
    ra[3] = pack2(A[(g + 8) * ai + (2 * q + 8) * ak], A[(g + 8) * ai + (2 * q + 9) * ak]);
    rb[0] = pack2(B[(2 * q) * bk + g * bj], B[(2 * q + 1) * bk + g * bj]);
    rb[1] = pack2(B[(2 * q + 8) * bk + g * bj], B[(2 * q + 9) * bk + g * bj]);
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(ra[0]), "r"(ra[1]), "r"(ra[2]), "r"(ra[3]), "r"(rb[0]), "r"(rb[1]));
  }
}
// f(i, j, value) for the lane's four entries of the tile at (i0, j0)
template <class F>
__device__ __forceinline__ void tile_each(int i0, int j0, const float *d, F f) {
  const int lane = (int)(threadIdx.x & 31u), g = lane >> 2, q = lane & 3;
  f(i0 + g, j0 + 2 * q, d[0]);
  f(i0 + g, j0 + 2 * q + 1, d[1]);
  f(i0 + g + 8, j0 + 2 * q, d[2]);
  f(i0 + g + 8, j0 + 2 * q + 1, d[3]);
}

// Forward and backward of one group: positions base .. base + 31 of a sequence
// of `end` rows; position p is row idx[off + p] (or off + p without idx).
// Positions past the end are padding: zero features, no loss, no gradient.  The
// loss is sum (y - t)^2 / denom; the group's weight gradients go to g and its
// loss to *lossp.  The weights lie in s.w, the fp32 biases and w3 in P.
//
// A group is a chain of seven dependent stages, 5.5 us with eight warps; one
// warp alone took most of a batch's 87 us with it (its products one tile after
// another, every operand gathered from global or unpadded shared memory).
// Every sum keeps its order:
// a tile's products accumulate over k as before, a row's output over the 64
// hidden units in order, a column's bias gradient over the 32 rows in order.
__device__ void group_fwd_bwd(GroupSmem &s, const MlpDev &P, const float *X, const float *T, const int *idx,
                              long long off, long long base, long long end, float denom, float *g, float *lossp) {
  const int tid = (int)threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 32) {
    const long long p = base + tid;
    s.row[tid] = p < end ? (idx ? idx[off + p] : (int)(off + p)) : -1;
  }
  __syncthreads();
  {
    const int r = tid >> 3, c = (tid & 7) * 4, row = s.row[r];
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (row >= 0) {
      const float *x = X + (long long)row * kFeat + c;
      v = make_float4(x[0], x[1], x[2], x[3]);
    }
    uint16_t *o = s.x + r * kXStride + c;
    o[0] = f2bf(v.x);
    o[1] = f2bf(v.y);
    o[2] = f2bf(v.z);
    o[3] = f2bf(v.w);
  }
  __syncthreads();
  float d[4];
  // a1 = relu(x W1^T + b1)
  for (int i0 = 0; i0 < 32; i0 += 16) {
    tile_gemm(kFeat, s.x + i0 * kXStride, kXStride, 1, s.w.w1 + warp * 8 * kW1Stride, 1, kW1Stride, d);
    tile_each(i0, warp * 8, d, [&](int i, int j, float h) {
      const float v = h + P.b1[j];
      s.a1[i * kHStride + j] = f2bf(v > 0.0f ? v : 0.0f);
    });
  }
  __syncthreads();
  // a2 = relu(a1 W2^T + b2)
  for (int i0 = 0; i0 < 32; i0 += 16) {
    tile_gemm(kHid, s.a1 + i0 * kHStride, kHStride, 1, s.w.w2 + warp * 8 * kW2Stride, 1, kW2Stride, d);
    tile_each(i0, warp * 8, d, [&](int i, int j, float h) {
      const float v = h + P.b2[j];
      s.a2[i * kHStride + j] = f2bf(v > 0.0f ? v : 0.0f);
    });
  }
  __syncthreads();
  if (warp == 0) {  // a lane per row
    const int row = s.row[lane];
    const float t = row >= 0 ? T[row] : 0.0f;
    float y = P.b3[0];
    for (int j = 0; j < kHid; ++j) y += bf2f(s.a2[lane * kHStride + j]) * bf2f(P.w3[j]);
    const float err = row >= 0 ? y - t : 0.0f;
    float l = err * err;
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (lane == 0) *lossp = l / denom;
    const float dy = 2.0f * err / denom;
    s.dy[lane] = dy;
    float db3 = dy;
    for (int o = 16; o; o >>= 1) db3 += __shfl_xor_sync(0xffffffffu, db3, o);
    if (lane == 0) g[kOffB3] = db3;
  }
  __syncthreads();
  // dz2 = dy w3 [a2 > 0]  (bf16)
  for (int k = tid; k < 32 * kHid; k += kGroupThreads) {
    const int r = k >> 6, j = k & 63;
    s.dz2[r * kHStride + j] = f2bf(s.a2[r * kHStride + j] != 0 ? s.dy[r] * bf2f(P.w3[j]) : 0.0f);
  }
  if (tid >= 128 && tid < 128 + kHid) {  // output layer's weights
    const int j = tid - 128;
    float acc = 0.0f;
    for (int r = 0; r < 32; ++r) acc += s.dy[r] * bf2f(s.a2[r * kHStride + j]);
    g[kOffW3 + j] = acc;
  }
  __syncthreads();
  // dz1 = (dz2 W2) [a1 > 0]  (bf16)
  for (int i0 = 0; i0 < 32; i0 += 16) {
    tile_gemm(kHid, s.dz2 + i0 * kHStride, kHStride, 1, s.w.w2 + warp * 8, kW2Stride, 1, d);
    tile_each(i0, warp * 8, d, [&](int i, int j, float h) {
      s.dz1[i * kHStride + j] = f2bf(s.a1[i * kHStride + j] != 0 ? h : 0.0f);
    });
  }
  // gW2[j][i] = sum_r dz2[r][j] a1[r][i]
  for (int j0 = 0; j0 < kHid; j0 += 16) {
    tile_gemm(32, s.dz2 + j0, 1, kHStride, s.a1 + warp * 8, kHStride, 1, d);
    tile_each(j0, warp * 8, d, [&](int j, int i, float v) { g[kOffW2 + j * kHid + i] = v; });
  }
  if (tid < kHid) {
    float acc = 0.0f;
    for (int r = 0; r < 32; ++r) acc += bf2f(s.dz2[r * kHStride + tid]);
    g[kOffB2 + tid] = acc;
  }
  __syncthreads();
  // gW1[j][i] = sum_r dz1[r][j] x[r][i]: 4 x 4 tiles
  for (int k = warp; k < 16; k += kGroupWarps) {
    const int j0 = (k >> 2) * 16, i0 = (k & 3) * 8;
    tile_gemm(32, s.dz1 + j0, 1, kHStride, s.x + i0, kXStride, 1, d);
    tile_each(j0, i0, d, [&](int j, int i, float v) { g[kOffW1 + j * kFeat + i] = v; });
  }
  if (tid >= 192 && tid < 192 + kHid) {
    const int j = tid - 192;
    float acc = 0.0f;
    for (int r = 0; r < 32; ++r) acc += bf2f(s.dz1[r * kHStride + j]);
    g[kOffB1 + j] = acc;
  }
  __syncthreads();
}

// inference as the placement step runs it (weights staged per block,
// activations in registers), kInferWarpsMax warps per block
__global__ void k_mlp_infer(MlpDev P, const float *X, long long n, float *out) {
  __shared__ MlpInferTiles sm;
  mlp_stage(P, sm.w);
  __syncthreads();
  const int warp = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u);
  uint16_t *x = sm.x[warp];
  const long long nw = (n + 31) / 32;
  for (long long gw = (long long)blockIdx.x * kInferWarpsMax + warp; gw < nw;
       gw += (long long)gridDim.x * kInferWarpsMax) {
    const long long row = gw * 32 + lane;
    float f[kFeat];
    if (row < n) {
      const float4 *xr = reinterpret_cast<const float4 *>(X + row * kFeat);
      for (int j = 0; j < kFeat / 4; ++j) {
        const float4 v = xr[j];
        f[4 * j] = v.x;
        f[4 * j + 1] = v.y;
        f[4 * j + 2] = v.z;
        f[4 * j + 3] = v.w;
      }
    } else {
      for (int j = 0; j < kFeat; ++j) f[j] = 0.0f;
    }
    mlp_put_row(x, lane, f);
    __syncwarp();
    const float y = mlp_forward_regs(sm.w, x);
    __syncwarp();
    if (row < n) out[row] = y;
  }
}
static int infer_blocks(long long n) {
  const long long nw = (n + 31) / 32;
  return (int)std::max<long long>(1, std::min<long long>((nw + kInferWarpsMax - 1) / kInferWarpsMax, 148 * 8));
}

// Forward and backward of rows [row0, row0 + nrows) (through idx when not null)
// with the loss  sum (y - t)^2 / denom.  Group w writes its weight gradients to
// part[w][.] and its loss to lossp[w].
__global__ void __launch_bounds__(kGroupThreads) k_mlp_fwd_bwd(MlpDev P, const float *X, const float *T, const int *idx,
                                                               long long row0, long long nrows, float denom, float *part,
                                                               float *lossp) {
  __shared__ GroupSmem s;
  mlp_stage(P, s.w);
  __syncthreads();
  const long long gw = blockIdx.x;
  group_fwd_bwd(s, P, X, T, idx, row0, gw * 32, nrows, denom, part + (size_t)gw * kParamCount, lossp + gw);
}

// grad[p] = sum over groups of part[w][p]; loss = sum of lossp
__global__ void k_mlp_reduce(const float *part, const float *lossp, int nw, float *grad, float *loss) {
  for (int p = (int)(blockIdx.x * blockDim.x + threadIdx.x); p < kParamCount; p += (int)(gridDim.x * blockDim.x)) {
    float acc = 0.0f;
    for (int w = 0; w < nw; ++w) acc += part[(size_t)w * kParamCount + p];
    grad[p] = acc;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    float acc = 0.0f;
    for (int w = 0; w < nw; ++w) acc += lossp[w];
    *loss = acc;
  }
}

// Adam on one fp32 master parameter; refreshes its bf16 copy.
struct AdamState {
  float *params, *m, *v;
  uint16_t *w1, *w2, *w3;
  float *bias;
};
__device__ __forceinline__ void adam_step(const AdamState &A, int p, float gp, float lr, float b1, float b2, float eps,
                                          float c1, float c2) {
  const float mp = b1 * A.m[p] + (1.0f - b1) * gp, vp = b2 * A.v[p] + (1.0f - b2) * gp * gp;
  A.m[p] = mp;
  A.v[p] = vp;
  const float x = A.params[p] - lr * (mp / c1) / (sqrtf(vp / c2) + eps);
  A.params[p] = x;
  if (p < kOffB1)
    A.w1[p - kOffW1] = f2bf(x);
  else if (p < kOffW2)
    A.bias[p - kOffB1] = x;
  else if (p < kOffB2)
    A.w2[p - kOffW2] = f2bf(x);
  else if (p < kOffW3)
    A.bias[kHid + p - kOffB2] = x;
  else if (p < kOffB3)
    A.w3[p - kOffW3] = f2bf(x);
  else
    A.bias[2 * kHid] = x;
}

// One epoch by one cooperative launch: for every batch the groups' forward and
// backward passes, a barrier, the gradients' sums (over the groups in order)
// with Adam, a barrier.  loss[step] gets the batch's loss; c[step] = (1 - b1^t,
// 1 - b2^t) comes from the host.  A batch of 1,024 rows takes 12.5 us (the
// chain of a group 5.5 us, the sums and Adam 2.2 us, the barriers 3.3 us, the
// weights 1.6 us); as three launches, a download and a synchronisation it took
// 87 us.
__global__ void __launch_bounds__(kGroupThreads, 1)
    k_mlp_epoch(MlpDev P, const float *X, const float *T, const int *idx, long long n, int batch, float *part,
                float *lossp, float *loss, const float2 *c, AdamState A, float lr, float b1, float b2, float eps,
                GridBar *bar, int *err) {
  __shared__ GroupSmem s;
  GridTeam team{bar, (int)gridDim.x, (int)blockIdx.x, 0ull, err, GQM_ERR_CUDA};
  int step = 0;
  for (long long r0 = 0; r0 < n; r0 += batch, ++step) {
    const long long rows = n - r0 < batch ? n - r0 : batch;
    const int groups = (int)((rows + 31) / 32);
    if (team.rank < groups) mlp_stage(P, s.w);
    __syncthreads();
    for (int w = team.rank; w < groups; w += team.nb)
      group_fwd_bwd(s, P, X, T, idx, r0, (long long)w * 32, rows, (float)rows, part + (size_t)w * kParamCount,
                    lossp + w);
    if (!team.sync()) return;
    const float2 cs = c[step];
    for (int p = team.tid(); p < kParamCount; p += team.size()) {
      float acc = 0.0f;
#pragma unroll 8
      for (int w = 0; w < groups; ++w) acc += part[(size_t)w * kParamCount + p];
      adam_step(A, p, acc, lr, b1, b2, eps, cs.x, cs.y);
    }
    if (team.rank == team.nb - 1 && threadIdx.x == 0) {
      float acc = 0.0f;
#pragma unroll 8
      for (int w = 0; w < groups; ++w) acc += lossp[w];
      loss[step] = acc;
    }
    if (!team.sync()) return;
  }
}

// Device copy of a network: bf16 weights and fp32 biases (b1, b2, b3).
struct MlpBuf {
  uint16_t *w = nullptr;  // w1 | w2 | w3
  float *b = nullptr;     // b1 | b2 | b3
  MlpDev dev() const { return mlp_dev(w, b); }
  int upload(const float *params, cudaStream_t st) {
    if (!w && (cudaMalloc((void **)&w, sizeof(uint16_t) * kMlpW) != cudaSuccess ||
               cudaMalloc((void **)&b, sizeof(float) * kMlpB) != cudaSuccess))
      return GQM_ERR_MEMORY;
    std::vector<uint16_t> hw(kMlpW);
    std::vector<float> hb(kMlpB);
    mlp_pack(params, hw.data(), hb.data());
    if (cudaMemcpyAsync(w, hw.data(), sizeof(uint16_t) * hw.size(), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(b, hb.data(), sizeof(float) * hb.size(), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return GQM_ERR_CUDA;
    return GQM_OK;
  }
  void release() {
    if (w) cudaFree(w);
    if (b) cudaFree(b);
    w = nullptr;
    b = nullptr;
  }
};

template <class T>
int dmalloc(T **p, size_t n) {
  return cudaMalloc((void **)p, sizeof(T) * (n ? n : 1)) == cudaSuccess ? GQM_OK : GQM_ERR_MEMORY;
}

// Arrays of one call carved from one allocation (a dozen cudaMalloc and cudaFree
// calls cost more than a millisecond).  With a null base it only measures.
struct Carve {
  char *base;
  size_t off = 0;
  template <class T>
  T *take(size_t n) {
    off = (off + 255) & ~(size_t)255;
    T *p = reinterpret_cast<T *>(base + off);
    off += sizeof(T) * (n ? n : 1);
    return p;
  }
};

// forward + backward + reduction over rows [row0, row0+nrows) of (X, T, idx)
int grad_pass(const MlpBuf &B, const float *dX, const float *dT, const int *didx, long long row0, long long nrows,
              float denom, float *dpart, float *dlossp, float *dgrad, float *dloss, cudaStream_t st) {
  const int nw = (int)((nrows + 31) / 32);
  k_mlp_fwd_bwd<<<nw, kGroupThreads, 0, st>>>(B.dev(), dX, dT, didx, row0, nrows, denom, dpart, dlossp);
  k_mlp_reduce<<<(kParamCount + 255) / 256, 256, 0, st>>>(dpart, dlossp, nw, dgrad, dloss);
  return cudaGetLastError() == cudaSuccess ? GQM_OK : GQM_ERR_CUDA;
}

}  // namespace
}  // namespace gqm

extern "C" {

int gqm_mlp_infer(int device, const float *params, const float *features, long long n, float *out) {
  using namespace gqm;
  if (!params || n < 0 || (n > 0 && (!features || !out))) return GQM_ERR_ARGUMENT;
  if (n == 0) return GQM_OK;
  if (cudaSetDevice(device) != cudaSuccess) return GQM_ERR_NO_DEVICE;
  cudaStream_t st;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return GQM_ERR_CUDA;
  MlpBuf B;
  float *dX = nullptr, *dY = nullptr;
  int rc = B.upload(params, st);
  if (!rc) rc = dmalloc(&dX, (size_t)n * kFeat);
  if (!rc) rc = dmalloc(&dY, (size_t)n);
  if (!rc) {
    cudaMemcpyAsync(dX, features, sizeof(float) * kFeat * n, cudaMemcpyHostToDevice, st);
    k_mlp_infer<<<infer_blocks(n), 32 * kInferWarpsMax, 0, st>>>(B.dev(), dX, n, dY);
    cudaMemcpyAsync(out, dY, sizeof(float) * n, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) rc = GQM_ERR_CUDA;
  }
  if (dX) cudaFree(dX);
  if (dY) cudaFree(dY);
  B.release();
  cudaStreamDestroy(st);
  return rc;
}

int gqm_mlp_time(int device, const float *params, long long n, int iters, float *ms) {
  using namespace gqm;
  if (!params || !ms || n <= 0 || n > (1LL << 28) || iters <= 0) return GQM_ERR_ARGUMENT;
  if (cudaSetDevice(device) != cudaSuccess) return GQM_ERR_NO_DEVICE;
  cudaStream_t st;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return GQM_ERR_CUDA;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  MlpBuf B;
  float *dX = nullptr, *dY = nullptr;
  int rc = B.upload(params, st);
  if (!rc) rc = dmalloc(&dX, (size_t)n * kFeat);
  if (!rc) rc = dmalloc(&dY, (size_t)n);
  if (!rc && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) rc = GQM_ERR_CUDA;
  if (!rc) {
    cudaMemsetAsync(dX, 0, sizeof(float) * kFeat * n, st);
    const int blocks = infer_blocks(n);
    k_mlp_infer<<<blocks, 32 * kInferWarpsMax, 0, st>>>(B.dev(), dX, n, dY);
    cudaEventRecord(e0, st);
    for (int i = 0; i < iters; ++i) k_mlp_infer<<<blocks, 32 * kInferWarpsMax, 0, st>>>(B.dev(), dX, n, dY);
    cudaEventRecord(e1, st);
    float t = 0.0f;
    if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess ||
        cudaEventElapsedTime(&t, e0, e1) != cudaSuccess)
      rc = GQM_ERR_CUDA;
    else
      *ms = t / (float)iters;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (dX) cudaFree(dX);
  if (dY) cudaFree(dY);
  B.release();
  cudaStreamDestroy(st);
  return rc;
}

int gqm_mlp_grad(int device, const float *params, const float *features, const float *targets, long long n,
                 float *loss, float *grad) {
  using namespace gqm;
  if (!params || !features || !targets || !loss || !grad || n <= 0 || n > (1LL << 24)) return GQM_ERR_ARGUMENT;
  if (cudaSetDevice(device) != cudaSuccess) return GQM_ERR_NO_DEVICE;
  cudaStream_t st;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return GQM_ERR_CUDA;
  MlpBuf B;
  float *dX = nullptr, *dT = nullptr, *dpart = nullptr, *dlp = nullptr, *dg = nullptr, *dl = nullptr;
  const int nw = (int)((n + 31) / 32);
  int rc = B.upload(params, st);
  if (!rc) rc = dmalloc(&dX, (size_t)n * kFeat) | dmalloc(&dT, (size_t)n) | dmalloc(&dpart, (size_t)nw * kParamCount) |
                dmalloc(&dlp, (size_t)nw) | dmalloc(&dg, (size_t)kParamCount) | dmalloc(&dl, 1);
  if (!rc) {
    cudaMemcpyAsync(dX, features, sizeof(float) * kFeat * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dT, targets, sizeof(float) * n, cudaMemcpyHostToDevice, st);
    rc = grad_pass(B, dX, dT, nullptr, 0, n, (float)n, dpart, dlp, dg, dl, st);
    cudaMemcpyAsync(grad, dg, sizeof(float) * kParamCount, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(loss, dl, sizeof(float), cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) rc = GQM_ERR_CUDA;
  }
  for (float *p : {dX, dT, dpart, dlp, dg, dl})
    if (p) cudaFree(p);
  B.release();
  cudaStreamDestroy(st);
  return rc;
}

int gqm_mlp_train(int device, float *params, const float *features, const float *targets, long long n, int epochs,
                  int batch, float lr, unsigned seed, float *loss) {
  using namespace gqm;
  if (!params || !features || !targets || n <= 0 || epochs < 0 || batch <= 0 || batch % 64 != 0 || !(lr > 0.0f))
    return GQM_ERR_ARGUMENT;
  if (cudaSetDevice(device) != cudaSuccess) return GQM_ERR_NO_DEVICE;
  cudaStream_t st;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return GQM_ERR_CUDA;
  MlpBuf B;
  float *dX = nullptr, *dT = nullptr, *dpart = nullptr, *dlp = nullptr, *dl = nullptr;
  float *dp = nullptr, *dm = nullptr, *dv = nullptr;
  float2 *dc = nullptr;
  GridBar *dbar = nullptr;
  int *didx = nullptr, *derr = nullptr;
  char *mem = nullptr;
  const int nw = (int)std::min<long long>(batch / 32, (n + 31) / 32);
  const long long steps = (n + batch - 1) / batch;
  int sms = 0, per = 0;
  int rc = B.upload(params, st);
  if (!rc && (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
              cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mlp_epoch, kGroupThreads, 0) != cudaSuccess ||
              sms < 1 || per < 1))
    rc = GQM_ERR_CUDA;
  for (int pass = 0; pass < 2 && !rc; ++pass) {  // measure, then carve
    Carve c{mem};
    dX = c.take<float>((size_t)n * kFeat);
    dT = c.take<float>((size_t)n);
    dpart = c.take<float>((size_t)nw * kParamCount);
    dlp = c.take<float>((size_t)nw);
    dl = c.take<float>((size_t)steps);
    dp = c.take<float>(kParamCount);
    dm = c.take<float>(kParamCount);
    dv = c.take<float>(kParamCount);
    didx = c.take<int>((size_t)n);
    dc = c.take<float2>((size_t)steps);
    dbar = c.take<GridBar>(1);
    derr = c.take<int>(1);
    if (pass == 0) rc = dmalloc(&mem, c.off);
  }
  float last = 0.0f;
  if (!rc) {
    cudaMemcpyAsync(dX, features, sizeof(float) * kFeat * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dT, targets, sizeof(float) * n, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(dp, params, sizeof(float) * kParamCount, cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(dm, 0, sizeof(float) * kParamCount, st);
    cudaMemsetAsync(dv, 0, sizeof(float) * kParamCount, st);
    cudaMemsetAsync(derr, 0, sizeof(int), st);
    std::vector<int> perm(n);
    std::iota(perm.begin(), perm.end(), 0);
    std::mt19937 rng(seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    long long step = 0;
    std::vector<float> lsum(steps);
    std::vector<float2> cs(steps);
    const AdamState A{dp, dm, dv, B.w, B.w + kHid * kFeat, B.w + kHid * kFeat + kHid * kHid, B.b};
    for (int e = 0; e < epochs && !rc; ++e) {
      std::shuffle(perm.begin(), perm.end(), rng);
      for (long long k = 0; k < steps; ++k) {
        ++step;
        cs[k] = make_float2(1.0f - powf(b1, (float)step), 1.0f - powf(b2, (float)step));
      }
      cudaMemcpyAsync(didx, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, st);
      cudaMemcpyAsync(dc, cs.data(), sizeof(float2) * steps, cudaMemcpyHostToDevice, st);
      cudaMemsetAsync(dbar, 0, sizeof(GridBar), st);
      // a block per group (and 16 for the sums over the parameters), all resident
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeCooperative;
      at[0].val.cooperative = 1;
      cfg.gridDim = dim3((unsigned)std::min(std::max(nw, 16), sms));
      cfg.blockDim = dim3(kGroupThreads);
      cfg.stream = st;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      if (cudaLaunchKernelEx(&cfg, k_mlp_epoch, B.dev(), (const float *)dX, (const float *)dT, (const int *)didx, n,
                             batch, dpart, dlp, dl, (const float2 *)dc, A, lr, b1, b2, eps, dbar, derr) != cudaSuccess)
        rc = GQM_ERR_CUDA;
      int herr = 0;
      cudaMemcpyAsync(lsum.data(), dl, sizeof(float) * steps, cudaMemcpyDeviceToHost, st);
      cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, st);
      if (cudaStreamSynchronize(st) != cudaSuccess) rc = GQM_ERR_CUDA;
      if (!rc && herr) rc = herr;
      double esum = 0.0;
      for (float l : lsum) esum += l;
      last = (float)(esum / (double)steps);
    }
    if (!rc) {
      cudaMemcpyAsync(params, dp, sizeof(float) * kParamCount, cudaMemcpyDeviceToHost, st);
      if (cudaStreamSynchronize(st) != cudaSuccess) rc = GQM_ERR_CUDA;
    }
  }
  if (loss) *loss = last;
  if (mem) cudaFree(mem);
  B.release();
  cudaStreamDestroy(st);
  return rc;
}

}  // extern "C"
