// Tensor-core and elementwise kernels of the learned warm start (a small convolutional network),
// with a C ABI that takes device pointers (the caller owns every buffer). The convolutions are
// expressed as BF16 GEMMs on tcgen05 (vl_gemm.cuh) around gather kernels (im2col / col2im).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <string>

#include "../../include/vortexlab.h"
#include "vl_conv.cuh"
#include "vl_gemm.cuh"
#include "vl_groups.hpp"
#include "vl_launch.hpp"

using bf16 = __nv_bfloat16;

namespace {

int fail(int code, const std::string& m) { return vl::set_error(code, m.c_str()); }

PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_encode_mutex;

int encoder(PFN_cuTensorMapEncodeTiled_v12000* out) {
  std::lock_guard<std::mutex> g(g_encode_mutex);
  if (!g_encode) {
    cudaDriverEntryPointQueryResult q;
    void* fn = nullptr;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn)
      return fail(VL_ECUDA, "cuTensorMapEncodeTiled is not available");
    g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  *out = g_encode;
  return VL_OK;
}

// 2-D tensor map of a row-major BF16 matrix [rows][cols] with leading dimension ld (elements),
// box = 64 columns x box_rows rows, 128-byte swizzle. Out-of-range boxes read zeros.
int make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
             int box_cols = vl::gemm::BK) {
  PFN_cuTensorMapEncodeTiled_v12000 enc;
  int rc = encoder(&enc);
  if (rc) return rc;
  if (((uintptr_t)base & 15) || (ld * 2) % 16) return fail(VL_EINVAL, "GEMM operands need 16-byte aligned rows");
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(VL_EINVAL, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return VL_OK;
}

// 4-D map (C, W, H, B) of NHWC BF16 activations; a box is kc channels x bw x bh pixels spaced `stride`
// apart, rows of kc channels swizzled over their 128 or 64 bytes. Pixels outside the image read zero.
int make_map_nhwc(CUtensorMap* map, const void* x, int B, int H, int W, int C, int stride, int kc, int bw, int bh) {
  PFN_cuTensorMapEncodeTiled_v12000 enc;
  int rc = encoder(&enc);
  if (rc) return rc;
  if (((uintptr_t)x & 15) || (C * 2) % 16) return fail(VL_EINVAL, "convolution operands need 16-byte aligned pixels");
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
  cuuint32_t box[4] = {(cuuint32_t)kc, (cuuint32_t)(bw * stride), (cuuint32_t)(bh * stride), 1};
  cuuint32_t estr[4] = {1, (cuuint32_t)stride, (cuuint32_t)stride, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(x), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, kc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(VL_EINVAL, "cuTensorMapEncodeTiled (NHWC) failed (" + std::to_string((int)r) + ")");
  return VL_OK;
}

int sm_count(int dev) {
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  return n;
}

// Device workspace for split-K partial tiles, one per device, grown on demand. Split-K GEMMs of
// one device are therefore serialised on the caller's stream discipline: the library's own users
// issue them on a single stream.
std::mutex g_ws_mutex;
void* g_ws[64] = {};
size_t g_ws_bytes[64] = {};

int workspace(int dev, size_t bytes, void** out) {
  std::lock_guard<std::mutex> g(g_ws_mutex);
  if (dev < 0 || dev >= 64) return fail(VL_EINVAL, "device index out of range");
  if (g_ws_bytes[dev] < bytes) {
    if (g_ws[dev]) {
      cudaDeviceSynchronize();
      cudaFree(g_ws[dev]);
      g_ws[dev] = nullptr;
      g_ws_bytes[dev] = 0;
    }
    const size_t want = bytes + bytes / 2;
    cudaError_t e = cudaMalloc(&g_ws[dev], want);
    if (e != cudaSuccess) return fail(VL_ENOMEM, std::string("gemm workspace: ") + cudaGetErrorString(e));
    g_ws_bytes[dev] = want;
  }
  *out = g_ws[dev];
  return VL_OK;
}

// out[m, n] (leading dimension ldc) = (accumulate ? out : 0) + sum over z of ws[z][m][n], z in order.
// A thread's chain of loads is the time where the outputs are few, as they are where the splits are many: the values of
// AHEAD splits are in flight, the next ones requested before these are added (2,048 outputs of 296 splits 23 us with a
// wait for each 16, 17 with AHEAD 32, 10 with 64; 9,216 of about 150 10.6, 8.9, 5.9). Where the splits are few, 16 and
// fewer registers (303,104 outputs and more: 10 us, 13 with 32), and below 16 as few as there are, in larger blocks (GEMM
// and reduction, us: 4608 x 512 of 4 splits 47.2 with 16 ahead, 42.7 with 4; 1024 x 1024 of 10 88.1, 84.2 with 8).
template <int AHEAD>
__global__ void k_split_reduce(const float* __restrict__ ws, int splits, int M, int N, float* __restrict__ out,
                               int ldc, int accumulate) {
  constexpr int H = AHEAD / 2;
  const long long total = (long long)M * N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const float* q = ws + i;
    float s = 0.0f, v[H], u[H];
    int z = 0;
    if (splits >= AHEAD) {
#pragma unroll
      for (int k = 0; k < H; ++k) v[k] = __ldcs(q + (long long)k * total);
      for (; z + AHEAD + H <= splits; z += AHEAD) {
#pragma unroll
        for (int k = 0; k < H; ++k) u[k] = __ldcs(q + (long long)(z + H + k) * total);
#pragma unroll
        for (int k = 0; k < H; ++k) s += v[k];
#pragma unroll
        for (int k = 0; k < H; ++k) v[k] = __ldcs(q + (long long)(z + AHEAD + k) * total);
#pragma unroll
        for (int k = 0; k < H; ++k) s += u[k];
      }
#pragma unroll
      for (int k = 0; k < H; ++k) s += v[k];
      z += H;
    }
    for (; z < splits; z += H) {   // (at most AHEAD values)
#pragma unroll
      for (int k = 0; k < H; ++k) u[k] = z + k < splits ? __ldcs(q + (long long)(z + k) * total) : 0.0f;
#pragma unroll
      for (int k = 0; k < H; ++k)
        if (z + k < splits) s += u[k];
    }
    float* o = out + (i / N) * ldc + (i % N);
    *o = accumulate ? *o + s : s;
  }
}

int split_reduce(const float* ws, int splits, int M, int N, float* out, int ldc, int accumulate, cudaStream_t s) {
  const long long total = (long long)M * N;
  const int blocks = (int)std::min<long long>((total + 63) / 64, 148 * 32);
  const int wide = (int)std::min<long long>((total + 255) / 256, 148 * 8);
  if (splits >= 64)
    k_split_reduce<64><<<blocks, 64, 0, s>>>(ws, splits, M, N, out, ldc, accumulate);
  else if (splits >= 16)
    k_split_reduce<16><<<blocks, 64, 0, s>>>(ws, splits, M, N, out, ldc, accumulate);
  else if (splits >= 8)
    k_split_reduce<8><<<wide, 256, 0, s>>>(ws, splits, M, N, out, ldc, accumulate);
  else
    k_split_reduce<4><<<wide, 256, 0, s>>>(ws, splits, M, N, out, ldc, accumulate);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VL_OK : fail(VL_ECUDA, std::string("gemm split reduce: ") + cudaGetErrorString(e));
}

template <int BN>
int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, int op,
                const vl::gemm::EpiParams& ep, cudaStream_t s) {
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  constexpr int smem = vl::gemm::smem_bytes<BN>();
  if (dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(vl::gemm::k_gemm_bf16<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(VL_ECUDA, std::string("gemm smem attribute: ") + cudaGetErrorString(e));
    configured[dev] = true;
  }
  const int gx = (M + vl::gemm::BM - 1) / vl::gemm::BM, gy = (N + BN - 1) / BN;
  const int kblocks = (K + vl::gemm::BK - 1) / vl::gemm::BK;
  // Too few output tiles to fill the 148 SMs and a long K (weight gradients): split K so that about
  // two CTAs per SM run, each over at least 8 K-blocks; FP32 results without bias/activation only.
  int splits = 1;
  const int tiles = gx * gy;
  if (tiles < 148 && kblocks >= 16 && !(ep.flags & (vl::gemm::EPI_BIAS | vl::gemm::EPI_RELU | vl::gemm::EPI_BF16))) {
    splits = std::min(kblocks / 8, (296 + tiles - 1) / tiles);
    if (splits < 1) splits = 1;
  }
  const int kb_per = (kblocks + splits - 1) / splits;
  splits = (kblocks + kb_per - 1) / kb_per;
  vl::gemm::EpiParams p = ep;
  float* ws = nullptr;
  if (splits > 1) {
    void* w = nullptr;
    int rc = workspace(dev, (size_t)splits * M * N * sizeof(float), &w);
    if (rc) return rc;
    ws = (float*)w;
    p.out = ws;
    p.ldc = N;
    p.flags = 0;
    p.split_stride = (long long)M * N;
  } else {
    p.split_stride = 0;
  }
  // A short K per CTA (the im2col GEMMs of the narrow layers: 1-8 K-blocks) gains nothing from a
  // deep ring; two stages let 2 (BN 256) to 5 (BN 32) CTAs share an SM instead, so one CTA's
  // epilogue overlaps the next one's loads. TMEM stays within its 512 columns in both cases.
  const int stages = kb_per <= 8 ? 2 : vl::gemm::STAGES;
  dim3 grid(gx, gy, splits);
  vl::gemm::k_gemm_bf16<BN><<<grid, 128, vl::gemm::smem_bytes<BN>(stages), s>>>(ta, tb, kblocks, kb_per, stages, op, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string("gemm launch: ") + cudaGetErrorString(e));
  if (splits > 1) return split_reduce(ws, splits, M, N, (float*)ep.out, ep.ldc, ep.flags & vl::gemm::EPI_ACCUM, s);
  return VL_OK;
}

}  // namespace

extern "C" {

int vl_nn_gemm_bf16(const void* a, int lda, const void* b, int ldb, int M, int N, int K, void* out, int ldc,
                    const float* bias, int flags, int bn, int* err, void* stream) {
  if (!a || !b || !out || M <= 0 || N <= 0 || K <= 0) return fail(VL_EINVAL, "gemm: bad arguments");
  if (bn != 32 && bn != 64 && bn != 128 && bn != 256) return fail(VL_EINVAL, "gemm: tile N must be 32, 64, 128 or 256");
  if ((flags & vl::gemm::EPI_BIAS) && !bias) return fail(VL_EINVAL, "gemm: bias requested without a bias");
  const int op = ((flags & VL_GEMM_A_MN) ? vl::gemm::OP_A_MN : 0) | ((flags & VL_GEMM_B_MN) ? vl::gemm::OP_B_MN : 0);
  if ((op & vl::gemm::OP_B_MN) && bn < 64) return fail(VL_EINVAL, "gemm: an MN-major B needs a tile N of 64 or more");
  CUtensorMap ta, tb;
  const bool amn = op & vl::gemm::OP_A_MN, bmn = op & vl::gemm::OP_B_MN;
  int rc = make_map(&ta, a, (uint64_t)(amn ? K : M), (uint64_t)(amn ? M : K), (uint64_t)lda, amn ? 64u : vl::gemm::BM);
  if (rc) return rc;
  rc = make_map(&tb, b, (uint64_t)(bmn ? K : N), (uint64_t)(bmn ? N : K), (uint64_t)ldb, bmn ? 64u : (uint32_t)bn);
  if (rc) return rc;
  vl::gemm::EpiParams ep;
  ep.out = out;
  ep.ldc = ldc;
  ep.bias = bias;
  ep.m_valid = M;
  ep.n_valid = N;
  ep.flags = flags & (vl::gemm::EPI_ACCUM | vl::gemm::EPI_BIAS | vl::gemm::EPI_RELU | vl::gemm::EPI_BF16);
  ep.err = err;
  ep.drop_load = (flags & VL_GEMM_TEST_TIMEOUT) ? 1 : 0;
  ep.spin_limit = ep.drop_load ? (1u << 12) : vl::gemm::kSpinLimit;
  cudaStream_t s = (cudaStream_t)stream;
  switch (bn) {
    case 32: return launch_gemm<32>(ta, tb, M, N, K, op, ep, s);
    case 64: return launch_gemm<64>(ta, tb, M, N, K, op, ep, s);
    case 128: return launch_gemm<128>(ta, tb, M, N, K, op, ep, s);
    default: return launch_gemm<256>(ta, tb, M, N, K, op, ep, s);
  }
}

}  // extern "C"

// ------------------------------------------------------------------ implicit convolutions
namespace {

// The shared-memory limit of a kernel, set once a device (`configured`: the kernel's own).
int smem_limit(const void* fn, int dev, int bytes, bool (&configured)[64], const char* what) {
  static std::mutex m;
  std::lock_guard<std::mutex> g(m);
  if (dev < 64 && configured[dev]) return VL_OK;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string(what) + " smem attribute: " + cudaGetErrorString(e));
  if (dev < 64) configured[dev] = true;
  return VL_OK;
}

template <int KC>
int launch_conv(const CUtensorMap& ta, const CUtensorMap& tb, vl::gemm::ConvParams& p, int N, cudaStream_t s) {
  using namespace vl::gemm;
  int dev = 0;
  cudaGetDevice(&dev);
  const int stage = conv_stage_bytes<KC>(p.bn);
  // Two blocks share an SM where their accumulators (2 x tmem_cols columns each) fit the 512 of its tensor
  // memory: one's prologue and tail run beside the other's MMAs.
  const int per_sm = 4 * p.tmem_cols <= 512 ? 2 : 1;
  p.stages = std::min(kConvMaxStages, (per_sm == 2 ? 104 * 1024 : 208 * 1024) / stage);
  const int smem = p.stages * stage + 1024;
  static bool configured[64] = {};
  if (int rc = smem_limit((const void*)k_conv<KC>, dev, 210 * 1024, configured, "convolution")) return rc;
  const int gy = (N + p.bn - 1) / p.bn;
  const int gx = std::max(1, std::min(p.tiles, per_sm * sm_count(dev) / gy));
  k_conv<KC><<<dim3((unsigned)gx, (unsigned)gy), kConvThreads, smem, s>>>(ta, tb, p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VL_OK : fail(VL_ECUDA, std::string("convolution launch: ") + cudaGetErrorString(e));
}

// k_conv_rows for a stride-1 3x3 convolution, where it applies: `done` false otherwise.
template <int KC>
int launch_rows(const void* x, int B, int H, int W, int C, const void* w, int kp, int N, const vl::gemm::EpiParams& ep,
                bool& done, cudaStream_t s) {
  using namespace vl::gemm;
  done = false;
  RowsParams p;
  p.chunks = C / KC;
  p.box_bytes = rows_box_bytes<KC>();
  // All output channels in one block, their 9 C x bn weights and a ring of five rows in its shared memory;
  // two blocks an SM where both fit. (In two or three parts, 192 -> 64 channels took 53 us as in k_conv, 64 -> 192
  // 47 against 41.)
  constexpr int kMost = 220 * 1024;
  if (N > 256) return VL_OK;
  p.bn = N <= 32 ? 32 : (N + 63) / 64 * 64;
  if ((9LL * C * p.bn * 2 + 1023) / 1024 * 1024 + 5LL * p.chunks * p.box_bytes + 1024 > kMost) return VL_OK;
  const int row_bytes = p.chunks * p.box_bytes, wb = (9 * C * p.bn * 2 + 1023) / 1024 * 1024;
  p.tmem_cols = p.bn <= 32 ? 32 : (p.bn <= 64 ? 64 : (p.bn <= 128 ? 128 : 256));
  const int per_sm = 4 * p.tmem_cols <= 512 && wb + 5 * row_bytes + 1024 <= kMost / 2 ? 2 : 1;
  p.ring = std::min(kRowsMaxRing, (kMost / per_sm - 1024 - wb) / row_bytes);
  p.Ho = H;
  p.Wo = W;
  p.tx = (W + BM - 1) / BM;
  p.ep = ep;
  int dev = 0;
  cudaGetDevice(&dev);
  const int blocks = per_sm * sm_count(dev);
  // the segment length with the shortest longest block (a segment loads two rows more than it has tiles)
  long long best = 0;
  for (int rows = 4; rows <= 64; ++rows) {
    const long long units = (long long)B * p.tx * ((H + rows - 1) / rows);
    const long long cost = ((units + blocks - 1) / blocks) * (rows + 1);
    if (rows == 4 || cost < best) {
      best = cost;
      p.seg_rows = rows;
    }
  }
  p.segs = (H + p.seg_rows - 1) / p.seg_rows;
  const long long units = (long long)B * p.tx * p.segs;
  if (units > 0x7fffffffLL) return VL_OK;
  p.units = (int)units;
  CUtensorMap ta, tb;
  int rc = make_map_nhwc(&ta, x, B, H, W, C, 1, KC, kRowPixels, 1);
  if (rc) return rc;
  rc = make_map(&tb, w, (uint64_t)N, (uint64_t)kp, (uint64_t)kp, (uint32_t)p.bn, KC);
  if (rc) return rc;
  using Fn = void (*)(const CUtensorMap, const CUtensorMap, const RowsParams);
  const Fn fns[4] = {k_conv_rows<KC, 0>, k_conv_rows<KC, 1>, k_conv_rows<KC, 2>, k_conv_rows<KC, 3>};
  const int ch = p.chunks <= 3 ? p.chunks : 0;
  static std::mutex m;
  static bool configured[64][4] = {};
  {
    std::lock_guard<std::mutex> g(m);
    if (dev >= 64 || !configured[dev][ch]) {
      cudaError_t e = cudaFuncSetAttribute((const void*)fns[ch], cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
      if (e != cudaSuccess) return fail(VL_ECUDA, std::string("convolution smem attribute: ") + cudaGetErrorString(e));
      if (dev < 64) configured[dev][ch] = true;
    }
  }
  const int smem = wb + p.ring * row_bytes + 1024;
  fns[ch]<<<dim3((unsigned)std::min<long long>(units, blocks)), kConvThreads, smem, s>>>(ta, tb, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string("convolution launch: ") + cudaGetErrorString(e));
  done = true;
  return VL_OK;
}

// The K split of launch_gemm for a weight gradient [kp, N] over `kblocks` 64-pixel blocks, so that the partial sums
// are the same, and where the partial results go.
int wgrad_split(int dev, int kp, int N, int bn, int kblocks, int* kb_per, int* splits, vl::gemm::EpiParams* ep, float* out) {
  const int tiles = ((kp + vl::gemm::BM - 1) / vl::gemm::BM) * ((N + bn - 1) / bn);
  int n = 1;
  if (tiles < 148 && kblocks >= 16) n = std::max(1, std::min(kblocks / 8, (296 + tiles - 1) / tiles));
  *kb_per = (kblocks + n - 1) / n;
  *splits = (kblocks + *kb_per - 1) / *kb_per;
  ep->out = out;
  ep->ldc = N;
  ep->split_stride = 0;
  if (*splits > 1) {
    void* w = nullptr;
    int rc = workspace(dev, (size_t)*splits * kp * N * sizeof(float), &w);
    if (rc) return rc;
    ep->out = w;
    ep->split_stride = (long long)kp * N;
  }
  return VL_OK;
}

template <int KC>
int launch_wgrad_rows(const void* x, int B, int H, int W, int C, const void* dz, int N, int kp, float* out,
                      const vl::gemm::EpiParams& ep, cudaStream_t s) {
  using namespace vl::gemm;
  int dev = 0;
  cudaGetDevice(&dev);
  WgradRowsParams p;
  p.Ho = H;
  p.Wo = W;
  p.C = C;
  p.chunks = C / KC;
  p.kp = kp;
  p.kblocks = (int)((long long)B * H * W / 64);
  p.bn = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256));
  p.ep = ep;
  int splits = 1;
  int rc = wgrad_split(dev, kp, N, std::max(p.bn, 64), p.kblocks, &p.kb_per, &splits, &p.ep, out);
  if (rc) return rc;
  p.a_bytes = (kWgradPixels * KC * 2 + 1023) / 1024 * 1024;
  p.stage_bytes = p.a_bytes + p.bn * 128;
  p.stages = std::min(kConvMaxStages, 100 * 1024 / p.stage_bytes);
  CUtensorMap ta, tb;
  rc = make_map_nhwc(&ta, x, B, H, W, C, 1, KC, kWgradPixels, 1);
  if (rc) return rc;
  rc = make_map(&tb, dz, (uint64_t)B * H * W, (uint64_t)N, (uint64_t)N, 64u, p.bn == 32 ? 32 : 64);
  if (rc) return rc;
  static bool configured[64] = {};
  if (int rc = smem_limit((const void*)k_wgrad_rows<KC>, dev, 104 * 1024, configured, "weight gradient")) return rc;
  const int gy = (N + p.bn - 1) / p.bn;
  k_wgrad_rows<KC><<<dim3((unsigned)(3 * p.chunks), (unsigned)gy, (unsigned)splits), 128, p.stages * p.stage_bytes + 1024, s>>>(ta, tb, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string("weight gradient launch: ") + cudaGetErrorString(e));
  return splits > 1 ? split_reduce((const float*)p.ep.out, splits, kp, N, out, N, 0, s) : VL_OK;
}

template <int KC>
int launch_wgrad(const CUtensorMap& ta, const CUtensorMap& tb, vl::gemm::WgradParams& p, int kp, int N, float* out,
                 cudaStream_t s) {
  using namespace vl::gemm;
  int dev = 0;
  cudaGetDevice(&dev);
  const int gx = (kp + BM - 1) / BM, gy = (N + p.bn - 1) / p.bn;
  int splits = 1;
  int rc = wgrad_split(dev, kp, N, p.bn, p.kblocks, &p.kb_per, &splits, &p.ep, out);
  if (rc) return rc;
  const int stage = wgrad_stage_bytes<KC>(p.bn);
  p.stages = std::min(kConvMaxStages, 100 * 1024 / stage);
  static bool configured[64] = {};
  if (int rc = smem_limit((const void*)k_wgrad<KC>, dev, 104 * 1024, configured, "weight gradient")) return rc;
  k_wgrad<KC><<<dim3((unsigned)gx, (unsigned)gy, (unsigned)splits), 128, p.stages * stage + 1024, s>>>(ta, tb, p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string("weight gradient launch: ") + cudaGetErrorString(e));
  return splits > 1 ? split_reduce((const float*)p.ep.out, splits, kp, N, out, N, 0, s) : VL_OK;
}

template <int KC, int BN>
int launch_dgrad2(const CUtensorMap& ta, const CUtensorMap& tb, vl::gemm::Dgrad2Params& p, cudaStream_t s) {
  using namespace vl::gemm;
  int dev = 0;
  cudaGetDevice(&dev);
  constexpr int kStage = conv_stage_bytes<KC>(BN), kStages = std::min(kConvMaxStages, 104 * 1024 / kStage);
  p.stages = kStages;
  static bool configured[64] = {};
  if (int rc = smem_limit((const void*)k_dgrad2<KC, BN>, dev, kStages * kStage + 1024, configured, "input gradient")) return rc;
  const int gy = (p.n_valid + BN - 1) / BN;
  const int gx = std::max(1, std::min(p.units, 2 * sm_count(dev) / gy));
  k_dgrad2<KC, BN><<<dim3((unsigned)gx, (unsigned)gy), kConvThreads, kStages * kStage + 1024, s>>>(ta, tb, p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VL_OK : fail(VL_ECUDA, std::string("input gradient launch: ") + cudaGetErrorString(e));
}

// How long a kernel's waits last, and whether a load that they wait for is left out (VL_GEMM_TEST_TIMEOUT).
constexpr unsigned kTestSpins = 1u << 12;
void test_timeout(vl::gemm::EpiParams& ep, int flags) {
  ep.drop_load = (flags & VL_GEMM_TEST_TIMEOUT) ? 1 : 0;
  ep.spin_limit = ep.drop_load ? kTestSpins : vl::gemm::kSpinLimit;
}

// The 4-channel layer (x: [B, H, W, 4], 3x3, stride 1).
int launch_conv_first(const void* x, int B, int H, int W, const void* w, int kp, int N, const vl::gemm::EpiParams& ep,
                      cudaStream_t s) {
  using namespace vl::gemm;
  int dev = 0;
  cudaGetDevice(&dev);
  FirstParams p{};
  p.B = B;
  p.H = H;
  p.W = W;
  p.x = (const __nv_bfloat16*)x;
  p.pixels = (long long)B * H * W;
  p.tiles = (int)((p.pixels + BM - 1) / BM);
  p.bn = N <= 32 ? 32 : (N + 63) / 64 * 64;
  p.kp = kp;
  p.ep = ep;
  CUtensorMap tb;
  int rc = make_map(&tb, w, (uint64_t)N, (uint64_t)kp, (uint64_t)kp, (uint32_t)p.bn);
  if (rc) return rc;
  const int smem = kFirstStages * 16384 + p.bn * 128 + 1024, most = kFirstStages * 16384 + 256 * 128 + 1024;
  static bool configured[64] = {};
  if (int rc = smem_limit((const void*)k_conv_first, dev, most, configured, "convolution")) return rc;
  const int per_sm = p.bn <= 128 ? 2 : 1;
  k_conv_first<<<(unsigned)std::min(p.tiles, per_sm * sm_count(dev)), 288, smem, s>>>(tb, p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VL_OK : fail(VL_ECUDA, std::string("convolution launch: ") + cudaGetErrorString(e));
}

int launch_wgrad_first(const void* x, int B, int H, int W, const void* dz, int N, int kp, float* out,
                       const vl::gemm::EpiParams& ep, cudaStream_t s) {
  using namespace vl::gemm;
  int dev = 0;
  cudaGetDevice(&dev);
  FirstParams p{};
  p.B = B;
  p.H = H;
  p.W = W;
  p.x = (const __nv_bfloat16*)x;
  p.pixels = (long long)B * H * W;
  p.kblocks = (int)((p.pixels + 63) / 64);
  p.bn = N <= 64 ? 64 : (N <= 128 ? 128 : 256);
  p.kp = kp;
  p.ep = ep;
  int splits = 1;
  int rc = wgrad_split(dev, kp, N, p.bn, p.kblocks, &p.kb_per, &splits, &p.ep, out);
  if (rc) return rc;
  CUtensorMap tb;
  rc = make_map(&tb, dz, (uint64_t)p.pixels, (uint64_t)N, (uint64_t)N, 64u);
  if (rc) return rc;
  const int smem = kFirstStages * (8192 + p.bn * 128) + 1024, most = kFirstStages * (8192 + 256 * 128) + 1024;
  static bool configured[64] = {};
  if (int rc = smem_limit((const void*)k_wgrad_first, dev, most, configured, "weight gradient")) return rc;
  k_wgrad_first<<<(unsigned)splits, 160, smem, s>>>(tb, p);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string("weight gradient launch: ") + cudaGetErrorString(e));
  return splits > 1 ? split_reduce((const float*)p.ep.out, splits, kp, N, out, N, 0, s) : VL_OK;
}

}  // namespace

extern "C" {

int vl_nn_conv_bf16(const void* x, int B, int H, int W, int C, int stride, int taps, const void* w, int kp, int N,
                    void* out, int ldc, const float* bias, int flags, int* err, void* stream) {
  using namespace vl::gemm;
  if (!x || !w || !out || B < 1 || H < 1 || W < 1 || N < 1 || (stride != 1 && stride != 2) || (taps != 1 && taps != 9))
    return fail(VL_EINVAL, "convolution: bad arguments");
  const bool first = C == 4 && taps == 9 && stride == 1 && kp == 64 && N <= 256 && !(flags & EPI_ACCUM) &&
                     (long long)B * H * W < 0x7fffff80LL && !((uintptr_t)x & 7);
  if ((!first && (C < 32 || C % 32)) || kp % 8 || kp < taps * C || N % 8 || ldc % 8 || ((uintptr_t)out & 31) || ((uintptr_t)bias & 15))
    return fail(VL_EINVAL, "convolution: channels in 32s (or the 4-channel 3x3 layer), output channels in 8s, 32-byte aligned rows");
  if ((flags & EPI_BIAS) && !bias) return fail(VL_EINVAL, "convolution: bias requested without a bias");
  if (first) {
    EpiParams ep{};
    ep.out = out;
    ep.ldc = ldc;
    ep.bias = bias;
    ep.n_valid = N;
    ep.flags = flags & (EPI_BIAS | EPI_RELU | EPI_BF16);
    ep.err = err;
    test_timeout(ep, flags);
    return launch_conv_first(x, B, H, W, w, kp, N, ep, (cudaStream_t)stream);
  }
  const int kc = C % 64 == 0 ? 64 : 32;
  ConvParams p;
  p.Ho = (H + stride - 1) / stride;
  p.Wo = (W + stride - 1) / stride;
  p.stride = stride;
  p.taps = taps;
  p.chunks = C / kc;
  p.pad = taps == 9 ? 1 : 0;
  // the tile shape with the fewest tiles (the widest of those)
  long long best = 0;
  for (int lw = 7; lw >= 3; --lw) {
    const int bw = 1 << lw, bh = BM >> lw;
    const long long n = (long long)((p.Wo + bw - 1) / bw) * ((p.Ho + bh - 1) / bh);
    if (lw == 7 || n < best) {
      best = n;
      p.bw = bw;
      p.bh = bh;
      p.log2_bw = lw;
    }
  }
  p.tiles_x = (p.Wo + p.bw - 1) / p.bw;
  p.tiles_y = (p.Ho + p.bh - 1) / p.bh;
  if (best * B > 0x7fffffffLL) return fail(VL_EINVAL, "convolution: too many pixels");
  p.tiles = (int)(best * B);
  // channels of a block: all of them up to 256, else equal parts in 32s; halves while the tiles are too few
  // to give every SM one
  int parts = (N + 255) / 256;
  while (p.tiles * parts < 148 && N >= 64 * 2 * parts) parts *= 2;
  p.bn = (N + parts - 1) / parts;
  p.bn = p.bn <= 32 ? 32 : (p.bn + 63) / 64 * 64;
  // FP32 results of few tiles: the K split of launch_gemm for the same product (there for more blocks),
  // so that the sums are the same; with accumulation they are formed in the workspace and added as there
  p.kb_split = taps * p.chunks;
  const long long rows = (long long)B * p.Ho * p.Wo;
  float* sums = nullptr;
  {
    const int gbn = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256)), kb64 = (kp + BK - 1) / BK;
    const long long gt = ((rows + BM - 1) / BM) * ((N + gbn - 1) / gbn);
    if (gt < 148 && kb64 >= 16 && !(flags & (EPI_BIAS | EPI_RELU | EPI_BF16))) {
      const int splits = std::max(1, std::min(kb64 / 8, (int)((296 + gt - 1) / gt)));
      p.kb_split = std::min(p.kb_split, (kb64 + splits - 1) / splits * (BK / kc));
      if ((flags & EPI_ACCUM) && p.kb_split < taps * p.chunks) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (int rc = workspace(dev, (size_t)rows * N * sizeof(float), (void**)&sums)) return rc;
      }
    }
  }
  p.tmem_cols = p.bn <= 32 ? 32 : (p.bn <= 64 ? 64 : (p.bn <= 128 ? 128 : 256));
  p.ep = EpiParams{};
  p.ep.out = sums ? sums : out;
  p.ep.ldc = sums ? N : ldc;
  p.ep.bias = bias;
  p.ep.n_valid = N;
  p.ep.flags = sums ? 0 : flags & (EPI_ACCUM | EPI_BIAS | EPI_RELU | EPI_BF16);
  p.ep.err = err;
  test_timeout(p.ep, flags);
  // Rows of whole 128-pixel tiles (or nearly: at most a quarter more tiles than the best shape) without a K split
  if (stride == 1 && taps == 9 && p.kb_split == taps * p.chunks && 4LL * ((W + BM - 1) / BM) * H <= 5 * best) {
    bool done = false;
    int rc = kc == 64 ? launch_rows<64>(x, B, H, W, C, w, kp, N, p.ep, done, (cudaStream_t)stream)
                      : launch_rows<32>(x, B, H, W, C, w, kp, N, p.ep, done, (cudaStream_t)stream);
    if (rc || done) return rc;
  }
  CUtensorMap ta, tb;
  int rc = make_map_nhwc(&ta, x, B, H, W, C, stride, kc, p.bw, p.bh);
  if (rc) return rc;
  rc = make_map(&tb, w, (uint64_t)N, (uint64_t)kp, (uint64_t)kp, (uint32_t)p.bn, kc);
  if (rc) return rc;
  rc = kc == 64 ? launch_conv<64>(ta, tb, p, N, (cudaStream_t)stream) : launch_conv<32>(ta, tb, p, N, (cudaStream_t)stream);
  return rc || !sums ? rc : split_reduce(sums, 1, (int)rows, N, (float*)out, ldc, 1, (cudaStream_t)stream);
}

static int dgrad2(const void* dz, int B, int H, int W, int C, int N, const void* wt, float* dx, int accumulate, int* err,
                  void* stream, int flags) {
  using namespace vl::gemm;
  if (!dz || !wt || !dx || B < 1 || H < 1 || W < 1 || C < 8 || C % 8 || N < 32 || N % 32 || ((uintptr_t)dx & 31))
    return fail(VL_EINVAL, "stride-2 input gradient: C in 8s, N in 32s, 32-byte aligned result");
  const int kc = N % 64 == 0 ? 64 : 32;
  Dgrad2Params p;
  p.H = H;
  p.W = W;
  p.C = C;
  p.n_valid = C;
  p.chunks = N / kc;
  p.accumulate = accumulate;
  p.drop_load = (flags & VL_GEMM_TEST_TIMEOUT) ? 1 : 0;
  p.dx = dx;
  p.err = err;
  p.spin_limit = p.drop_load ? kTestSpins : kSpinLimit;
  const int hh = (H + 1) / 2, hw = (W + 1) / 2;                 // dz's grid, and that of the pixels of a class
  long long best = 0;
  for (int lw = 7; lw >= 3; --lw) {
    const long long n = (long long)((hw + (1 << lw) - 1) >> lw) * ((hh + (BM >> lw) - 1) / (BM >> lw));
    if (lw == 7 || n < best) {
      best = n;
      p.bw = 1 << lw;
      p.bh = BM >> lw;
      p.log2_bw = lw;
    }
  }
  if (best * 4 * B > 0x7fffffffLL) return fail(VL_EINVAL, "stride-2 input gradient: too many pixels");
  p.tiles_x = (hw + p.bw - 1) / p.bw;
  p.tiles_y = (hh + p.bh - 1) / p.bh;
  p.tiles = (int)best;
  p.units = (int)best * 4 * B;
  const int bn = C <= 32 ? 32 : 64;   // (128: 22 us against 20 at 32 x 64 pixels, 128 <- 256)
  CUtensorMap ta, tb;
  int rc = make_map_nhwc(&ta, dz, B, hh, hw, N, 1, kc, p.bw, p.bh);
  if (rc) return rc;
  rc = make_map(&tb, wt, (uint64_t)9 * C, (uint64_t)N, (uint64_t)N, (uint32_t)bn, kc);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  if (kc == 64) return bn == 32 ? launch_dgrad2<64, 32>(ta, tb, p, s) : launch_dgrad2<64, 64>(ta, tb, p, s);
  return bn == 32 ? launch_dgrad2<32, 32>(ta, tb, p, s) : launch_dgrad2<32, 64>(ta, tb, p, s);
}

static int wgrad(const void* x, int B, int H, int W, int C, int stride, const void* dz, int N, float* gwt, int kp, int* err,
                 void* stream, int flags) {
  using namespace vl::gemm;
  if (!x || !dz || !gwt || B < 1 || H < 1 || W < 1 || N < 1 || (stride != 1 && stride != 2))
    return fail(VL_EINVAL, "weight gradient: bad arguments");
  const int Ho = (H + stride - 1) / stride, Wo = (W + stride - 1) / stride;
  const int bw = Wo % 64 == 0 ? 64 : Wo;
  if (C == 4 && stride == 1 && kp == 64 && N <= 256 && N % 8 == 0 && (long long)B * H * W < 0x7fffff80LL &&
      !((uintptr_t)x & 7) && !((uintptr_t)gwt & 31)) {
    EpiParams ep{};
    ep.n_valid = N;
    ep.err = err;
    test_timeout(ep, flags);
    return launch_wgrad_first(x, B, H, W, dz, N, kp, gwt, ep, (cudaStream_t)stream);
  }
  if (C < 32 || C % 32 || kp < 9 * C || N % 8 || ((uintptr_t)gwt & 31) || bw > 64 || 64 % bw || Ho % (64 / bw))
    return fail(VL_EINVAL, "weight gradient: channels in 32s, output rows that 64-pixel blocks divide");
  const int kc = C % 64 == 0 ? 64 : 32;
  WgradParams p;
  p.Ho = Ho;
  p.Wo = Wo;
  p.stride = stride;
  p.pad = 1;
  p.taps = 9;
  p.C = C;
  p.kblocks = (int)((long long)B * Ho * Wo / 64);
  p.bn = N <= 64 ? 64 : (N <= 128 ? 128 : 256);
  p.ep = EpiParams{};
  p.ep.m_valid = kp;
  p.ep.n_valid = N;
  p.ep.err = err;
  test_timeout(p.ep, flags);
  // The three taps of a row as one operand: for chunks of 32 channels (batch 16, 128 x 256 pixels: 32 x 32
  // 67 -> 43 us, 96 x 32 165 -> 79) and many chunks (64 x 128 192 x 64 77 -> 57, 32 x 64 384 x 128 57 -> 49); one or two
  // 64-channel chunks leave it too few blocks (64 x 64 27 -> 30, 128 x 128 23 -> 27), wide N too many dropped products
  // (64 x 192 51 -> 77).
  if (stride == 1 && Wo % 64 == 0 && (kc == 32 || (C >= 192 && N <= 128)))
    return kc == 64 ? launch_wgrad_rows<64>(x, B, H, W, C, dz, N, kp, gwt, p.ep, (cudaStream_t)stream)
                    : launch_wgrad_rows<32>(x, B, H, W, C, dz, N, kp, gwt, p.ep, (cudaStream_t)stream);
  CUtensorMap ta, tb;
  int rc = make_map_nhwc(&ta, x, B, H, W, C, stride, kc, bw, 64 / bw);
  if (rc) return rc;
  rc = make_map(&tb, dz, (uint64_t)B * Ho * Wo, (uint64_t)N, (uint64_t)N, 64u);
  if (rc) return rc;
  return kc == 64 ? launch_wgrad<64>(ta, tb, p, kp, N, gwt, (cudaStream_t)stream)
                  : launch_wgrad<32>(ta, tb, p, kp, N, gwt, (cudaStream_t)stream);
}

int vl_nn_dgrad2_bf16(const void* dz, int B, int H, int W, int C, int N, const void* wt, float* dx, int accumulate, int* err,
                      void* stream) {
  return dgrad2(dz, B, H, W, C, N, wt, dx, accumulate, err, stream, 0);
}
int vl_nn_dgrad2_test_timeout(const void* dz, int B, int H, int W, int C, int N, const void* wt, float* dx, int accumulate,
                              int* err, void* stream) {
  return dgrad2(dz, B, H, W, C, N, wt, dx, accumulate, err, stream, VL_GEMM_TEST_TIMEOUT);
}
int vl_nn_wgrad_bf16(const void* x, int B, int H, int W, int C, int stride, const void* dz, int N, float* gwt, int kp,
                     int* err, void* stream) {
  return wgrad(x, B, H, W, C, stride, dz, N, gwt, kp, err, stream, 0);
}
int vl_nn_wgrad_test_timeout(const void* x, int B, int H, int W, int C, int stride, const void* dz, int N, float* gwt, int kp,
                             int* err, void* stream) {
  return wgrad(x, B, H, W, C, stride, dz, N, gwt, kp, err, stream, VL_GEMM_TEST_TIMEOUT);
}

}  // extern "C"

// ------------------------------------------------------------------ convolution gathers
// Activations are NHWC (row r = (b * H + y) * W + x, channels contiguous). A 3x3 convolution with
// padding 1 and stride s reads, for output pixel (b, oy, ox), the input pixels
// (s*oy + ky - 1, s*ox + kx - 1); its im2col row holds them in (ky, kx, c) order, zero-padded to
// kp columns (a multiple of 64, the GEMM's K block).
namespace {

__global__ void k_im2col(const bf16* __restrict__ x, int B, int H, int W, int C, int stride, int Ho, int Wo, int kp,
                         bf16* __restrict__ cols) {
  // one thread per 8 consecutive columns of a row: a single 16-byte load and store when C % 8 == 0
  const int G = kp >> 3;
  const long long total = (long long)B * Ho * Wo * G;
  const bool vec = (C & 7) == 0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int g = (int)(i % G);
    const long long r = i / G;
    const int ox = (int)(r % Wo);
    const long long q = r / Wo;
    const int oy = (int)(q % Ho), b = (int)(q / Ho);
    const int k0 = g * 8;
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    if (vec) {
      if (k0 < 9 * C) {
        const int tap = k0 / C, c = k0 - tap * C;
        const int iy = stride * oy + tap / 3 - 1, ix = stride * ox + tap % 3 - 1;
        if (iy >= 0 && iy < H && ix >= 0 && ix < W)
          out = *reinterpret_cast<const uint4*>(x + (((long long)b * H + iy) * W + ix) * C + c);
      }
    } else {
      __align__(16) bf16 v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = k0 + j;
        v[j] = __float2bfloat16_rn(0.0f);
        if (k < 9 * C) {
          const int tap = k / C, c = k - tap * C;
          const int iy = stride * oy + tap / 3 - 1, ix = stride * ox + tap % 3 - 1;
          if (iy >= 0 && iy < H && ix >= 0 && ix < W) v[j] = x[(((long long)b * H + iy) * W + ix) * C + c];
        }
      }
      out = *reinterpret_cast<const uint4*>(v);
    }
    *reinterpret_cast<uint4*>(cols + r * kp + k0) = out;
  }
}

// dX[b, iy, ix, c] = sum over the (oy, ox, ky, kx) that read it of dcols[(b, oy, ox), (ky, kx, c)].
// One thread per 4 consecutive channels (float4 loads) when C % 4 == 0, else per channel.
__global__ void k_col2im(const float* __restrict__ dcols, int B, int H, int W, int C, int stride, int Ho, int Wo,
                         int kp, float* __restrict__ dx, int accumulate) {
  const int V = (C & 3) == 0 ? 4 : 1;
  const int G = C / V;
  const long long total = (long long)B * H * W * G;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % G) * V;
    const long long p = i / G;
    const int ix = (int)(p % W);
    const long long q = p / W;
    const int iy = (int)(q % H), b = (int)(q / H);
    float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int ky = 0; ky < 3; ++ky) {
      const int ty = iy + 1 - ky;
      if (ty < 0 || ty % stride) continue;
      const int oy = ty / stride;
      if (oy >= Ho) continue;
      for (int kx = 0; kx < 3; ++kx) {
        const int tx = ix + 1 - kx;
        if (tx < 0 || tx % stride) continue;
        const int ox = tx / stride;
        if (ox >= Wo) continue;
        const float* src = dcols + (((long long)b * Ho + oy) * Wo + ox) * kp + (ky * 3 + kx) * C + c;
        if (V == 4) {
          const float4 v = *reinterpret_cast<const float4*>(src);
          s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w;
        } else {
          s[0] += *src;
        }
      }
    }
    float* o = dx + p * C + c;
    for (int j = 0; j < V; ++j) o[j] = accumulate ? o[j] + s[j] : s[j];
  }
}

// dz = dy * (y > 0) (ReLU; y is the layer output) or dz = dy (no activation); BF16 copies of dz
// row-major [R, C] and transposed [C, R] for the two backward GEMMs, and colsum[c, t] = the sum of
// dz over the 32 rows of row tile t (fixed order), from which the bias gradient is reduced.
__global__ void k_act_bwd(const float* __restrict__ dy, const bf16* __restrict__ y, int R, int C, int relu,
                          bf16* __restrict__ dz, bf16* __restrict__ dzt, float* __restrict__ colsum, int ntiles) {
  __shared__ float tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int r = r0 + j, c = c0 + threadIdx.x;
    float v = 0.0f;
    if (r < R && c < C) {
      v = dy[(long long)r * C + c];
      if (relu && !(__bfloat162float(y[(long long)r * C + c]) > 0.0f)) v = 0.0f;
      const bf16 h = __float2bfloat16_rn(v);
      dz[(long long)r * C + c] = h;
      v = __bfloat162float(h);
    }
    tile[j][threadIdx.x] = v;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += blockDim.y) {
    const int c = c0 + j, r = r0 + threadIdx.x;
    const float v = tile[threadIdx.x][j];
    if (dzt && c < C && r < R) dzt[(long long)c * R + r] = __float2bfloat16_rn(v);
    float sum = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (colsum && threadIdx.x == 0 && c < C) colsum[(long long)c * ntiles + blockIdx.y] = sum;
  }
}

// k_act_bwd for rows of whole 16-byte groups (C % 4 == 0, no transposed copy): a block takes 256 rows x 32
// columns, four columns a load, and sums each of its 32-row tiles by the tree of k_act_bwd's shuffles.
// Bound by its HBM traffic (10 bytes an element); the kernel above moved 4 bytes a load through one
// 32 x 32 tile a block: 524,288 x 32 69 -> 33 us.
__global__ void __launch_bounds__(256) k_act_bwd4(const float* __restrict__ dy, const bf16* __restrict__ y, int R, int C,
                                                  int relu, bf16* __restrict__ dz, float* __restrict__ colsum, int ntiles) {
  __shared__ float tile[256][33];
  const int c0 = blockIdx.x * 32;
  const long long r0 = (long long)blockIdx.y * 256;
  const int q = threadIdx.x & 7, c = c0 + 4 * q;
  float4 g[8];
  uint2 a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const long long r = r0 + (threadIdx.x >> 3) + 32 * i;
    if (r < R && c < C) {
      g[i] = __ldcs(reinterpret_cast<const float4*>(dy + r * C + c));
      if (relu) a[i] = __ldcs(reinterpret_cast<const uint2*>(y + r * C + c));
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int j = (threadIdx.x >> 3) + 32 * i;
    const long long r = r0 + j;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (r < R && c < C) {
      v[0] = g[i].x; v[1] = g[i].y; v[2] = g[i].z; v[3] = g[i].w;
      if (relu) {
        const bf16* h = reinterpret_cast<const bf16*>(&a[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (!(__bfloat162float(h[k]) > 0.0f)) v[k] = 0.0f;
      }
      bf16 o[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        o[k] = __float2bfloat16_rn(v[k]);
        v[k] = __bfloat162float(o[k]);
      }
      *reinterpret_cast<uint2*>(dz + r * C + c) = *reinterpret_cast<const uint2*>(o);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) tile[j][4 * q + k] = v[k];
  }
  if (!colsum) return;
  __syncthreads();
  const int t = threadIdx.x >> 5, col = threadIdx.x & 31;
  float v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = tile[32 * t + k][col];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < o; ++k) v[k] += v[k + o];
  }
  const long long nt = (long long)blockIdx.y * 8 + t;
  if (nt < ntiles && c0 + col < C) colsum[(long long)(c0 + col) * ntiles + nt] = v[0];
}

// db[c] = sum over the row tiles t of colsum[c, t] (one block per channel, fixed tree). Eight loads of a
// thread are in flight ahead of its additions: one at a time, the 64 of 524,288 rows took 15 us (now 6).
__global__ void k_bias_grad(const float* __restrict__ colsum, int ntiles, float* __restrict__ db) {
  __shared__ float red[256];
  const int c = blockIdx.x;
  float s = 0.0f;
  const float* src = colsum + (long long)c * ntiles;
  int t = threadIdx.x;
  for (; t + 7 * 256 < ntiles; t += 8 * 256) {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = src[t + k * 256];
#pragma unroll
    for (int k = 0; k < 8; ++k) s += v[k];
  }
  for (; t < ntiles; t += 256) s += src[t];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) db[c] = red[0];
}

// BF16 transpose [R, C] -> [C, R] (R and C even): 64 x 64 tiles moved as pairs of elements.
__global__ void k_transpose_bf16(const bf16* __restrict__ a, int R, int C, bf16* __restrict__ at) {
  __shared__ bf16 tile[64][66];
  const int c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
  for (int j = threadIdx.y; j < 64; j += blockDim.y) {
    const int r = r0 + j, c = c0 + 2 * threadIdx.x;
    __nv_bfloat162 v = __floats2bfloat162_rn(0.0f, 0.0f);
    if (r < R && c < C) v = *reinterpret_cast<const __nv_bfloat162*>(a + (long long)r * C + c);
    tile[j][2 * threadIdx.x] = v.x;
    tile[j][2 * threadIdx.x + 1] = v.y;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 64; j += blockDim.y) {
    const int c = c0 + j, r = r0 + 2 * threadIdx.x;
    if (c < C && r < R) {
      __nv_bfloat162 v;
      v.x = tile[2 * threadIdx.x][j];
      v.y = tile[2 * threadIdx.x + 1][j];
      *reinterpret_cast<__nv_bfloat162*>(at + (long long)c * R + r) = v;
    }
  }
}

// Weights of the input-gradient convolution of a stride-1 3x3 layer: wf[c, (ky, kx, co)] =
// w[co, (2 - ky, 2 - kx, c)] (taps mirrored, input and output channels swapped), zero-padded to
// kpf columns. With it dX = conv3x3(dZ, wf), an im2col of dZ and one GEMM, with no col2im.
__global__ void k_flip_weights(const bf16* __restrict__ w, int cout, int cin, int kp, int kpf, bf16* __restrict__ wf) {
  const long long total = (long long)cin * kpf;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i % kpf), c = (int)(i / kpf);
    bf16 v = __float2bfloat16_rn(0.0f);
    if (k < 9 * cout) {
      const int tap = k / cout, co = k - tap * cout;
      v = w[(long long)co * kp + (8 - tap) * cin + c];
    }
    wf[i] = v;
  }
}

// Nearest 2x upsampling of NHWC BF16 [B, H, W, C] -> [B, 2H, 2W, C] into channels [coff, coff + C)
// of an output with ctot channels; backward sums the four children into FP32.
__global__ void k_up2(const bf16* __restrict__ x, int B, int H, int W, int C, bf16* __restrict__ y, int ctot, int coff) {
  const long long total = (long long)B * 2 * H * 2 * W * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const long long p = i / C;
    const int X = (int)(p % (2 * W)), Y = (int)((p / (2 * W)) % (2 * H)), b = (int)(p / (4LL * W * H));
    y[p * ctot + coff + c] = x[(((long long)b * H + Y / 2) * W + X / 2) * C + c];
  }
}

__global__ void k_up2_bwd(const float* __restrict__ dy, int B, int H, int W, int C, int ctot, int coff,
                          float* __restrict__ dx, int accumulate) {
  const long long total = (long long)B * H * W * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const long long p = i / C;
    const int x = (int)(p % W), yy = (int)((p / W) % H), b = (int)(p / ((long long)W * H));
    float s = 0.0f;
    for (int dy2 = 0; dy2 < 2; ++dy2)
      for (int dx2 = 0; dx2 < 2; ++dx2)
        s += dy[((((long long)b * 2 * H + 2 * yy + dy2) * 2 * W) + 2 * x + dx2) * ctot + coff + c];
    dx[i] = accumulate ? dx[i] + s : s;
  }
}

// The same moves for channel counts and offsets of whole 16-byte groups (V = 8 BF16 or 4 FP32 values) and fewer
// than 2^31 groups (vl_groups.hpp): one group a thread, 32-bit index arithmetic. (The kernels of one value a thread spend their
// time on 64-bit divisions: 524,288 pixels x 64 of 96 channels, us: up2 208 -> 26, copy 43 -> 16, slice 46 -> 27,
// up2_bwd 59 -> 33.) `gc`: groups of C; `gt`, `go`: of ctot and coff.
__global__ void k_up2_v(const uint4* __restrict__ x, unsigned total, unsigned H, unsigned W, unsigned gc, uint4* __restrict__ y,
                        unsigned gt, unsigned go) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    // one source group to its four places
    const unsigned c = i % gc, p = i / gc, xx = p % W, q = p / W;       // q = b * H + row
    const uint4 v = __ldg(x + i);
    uint4* o = y + ((size_t)(2 * q) * (2 * W) + 2 * xx) * gt + go + c;
    o[0] = v;
    o[gt] = v;
    o[(size_t)2 * W * gt] = v;
    o[(size_t)(2 * W + 1) * gt] = v;
  }
}

__global__ void k_up2_bwd_v(const float4* __restrict__ dy, unsigned total, unsigned W, unsigned gc, unsigned gt, unsigned go,
                            float4* __restrict__ dx, int accumulate) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned c = i % gc, p = i / gc, xx = p % W, q = p / W;
    const float4* s = dy + ((size_t)(2 * q) * (2 * W) + 2 * xx) * gt + go + c;
    const float4 a = __ldcs(s), b = __ldcs(s + gt), d = __ldcs(s + (size_t)2 * W * gt), e = __ldcs(s + (size_t)(2 * W + 1) * gt);
    float4 v = make_float4(0.0f + a.x, 0.0f + a.y, 0.0f + a.z, 0.0f + a.w);
    v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
    v = make_float4(v.x + d.x, v.y + d.y, v.z + d.z, v.w + d.w);
    v = make_float4(v.x + e.x, v.y + e.y, v.z + e.z, v.w + e.w);
    if (accumulate) {
      const float4 o = dx[i];
      v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
    }
    dx[i] = v;
  }
}

__global__ void k_copy_channels_v(const uint4* __restrict__ x, unsigned total, unsigned gc, uint4* __restrict__ y, unsigned gt,
                                  unsigned go) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x)
    y[(size_t)(i / gc) * gt + go + i % gc] = __ldg(x + i);
}

__global__ void k_slice_channels_v(const float4* __restrict__ y, unsigned total, unsigned gc, unsigned gt, unsigned go,
                                   float4* __restrict__ x, int accumulate) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    float4 v = __ldcs(y + (size_t)(i / gc) * gt + go + i % gc);
    if (accumulate) {
      const float4 o = x[i];
      v = make_float4(o.x + v.x, o.y + v.y, o.z + v.z, o.w + v.w);
    }
    x[i] = v;
  }
}

// Copies channels [0, C) of x ([R, C]) into channels [coff, coff + C) of y ([R, ctot]) and back.
__global__ void k_copy_channels(const bf16* __restrict__ x, long long R, int C, bf16* __restrict__ y, int ctot, int coff) {
  const long long total = R * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x)
    y[(i / C) * ctot + coff + (i % C)] = x[i];
}

__global__ void k_slice_channels_f32(const float* __restrict__ y, long long R, int ctot, int coff, int C,
                                     float* __restrict__ x, int accumulate) {
  const long long total = R * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const float v = y[(i / C) * ctot + coff + (i % C)];
    x[i] = accumulate ? x[i] + v : v;
  }
}

// Masked mean-squared error over R pixels x the first `cuse` of C output channels (the target is
// [R, cuse]): loss partial sums per block (FP64) and the gradient dOut = 2 w (out - target) / count
// (zero on the other channels).
__global__ void k_mse(const float* __restrict__ out, const float* __restrict__ tgt, const float* __restrict__ w,
                      long long R, int C, int cuse, double inv_count, float* __restrict__ dout,
                      double* __restrict__ partial) {
  __shared__ double red[256];
  double s = 0.0;
  const long long total = R * C;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    // (32-bit division where the index fits: the 64-bit one was half the kernel's time)
    const long long r = i <= 0xffffffffLL ? (long long)((unsigned)i / (unsigned)C) : i / C;
    const int c = (int)(i - r * C);
    const float wi = c < cuse ? w[r] : 0.0f;
    const float d = c < cuse ? out[i] - tgt[r * cuse + c] : 0.0f;
    s += (double)wi * d * d;
    dout[i] = (float)(2.0 * inv_count) * wi * d;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) red[threadIdx.x] += red[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0] * inv_count;
}

// Adam (FP32 master weights); writes the BF16 copy the GEMMs read, padded layout kept by the
// caller (n values).
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       long long n, float lr, float b1, float b2, float eps, float c1, float c2,
                       bf16* __restrict__ wb) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16_rn(wi);
  }
}

__global__ void k_f32_to_bf16(const float* __restrict__ a, long long n, bf16* __restrict__ b) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = __float2bfloat16_rn(a[i]);
}

int grid_for(long long n) {
  constexpr long long most = vl::kMoveThreads / 256;
  long long g = (n + 255) / 256;
  return (int)(g < most ? (g < 1 ? 1 : g) : most);
}

bool grouped(const void* a, const void* b, long long values, int C, int ctot, int coff, int v) {
  return vl::move_grouped((uintptr_t)a, (uintptr_t)b, values, C, ctot, coff, v);
}

int launch_check(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VL_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return VL_OK;
}

}  // namespace

extern "C" {

int vl_nn_im2col(const void* x, int B, int H, int W, int C, int stride, int kp, void* cols, void* stream) {
  if (!x || !cols || (stride != 1 && stride != 2) || kp < 9 * C || kp % 64) return fail(VL_EINVAL, "im2col: bad arguments");
  if (((uintptr_t)x & 15) || ((uintptr_t)cols & 15)) return fail(VL_EINVAL, "im2col: buffers must be 16-byte aligned");
  const int Ho = (H + stride - 1) / stride, Wo = (W + stride - 1) / stride;
  k_im2col<<<grid_for((long long)B * Ho * Wo * (kp / 8)), 256, 0, (cudaStream_t)stream>>>(
      (const bf16*)x, B, H, W, C, stride, Ho, Wo, kp, (bf16*)cols);
  return launch_check("im2col");
}

int vl_nn_col2im(const float* dcols, int B, int H, int W, int C, int stride, int kp, float* dx, int accumulate,
                 void* stream) {
  if (!dcols || !dx || (stride != 1 && stride != 2) || kp < 9 * C || kp % 4) return fail(VL_EINVAL, "col2im: bad arguments");
  if (((uintptr_t)dcols & 15) || ((uintptr_t)dx & 15)) return fail(VL_EINVAL, "col2im: buffers must be 16-byte aligned");
  const int Ho = (H + stride - 1) / stride, Wo = (W + stride - 1) / stride;
  const long long work = (long long)B * H * W * ((C & 3) == 0 ? C / 4 : C);
  k_col2im<<<grid_for(work), 256, 0, (cudaStream_t)stream>>>(dcols, B, H, W, C, stride, Ho, Wo, kp, dx, accumulate);
  return launch_check("col2im");
}

int vl_nn_act_bwd(const float* dy, const void* y, int R, int C, int relu, void* dz, void* dzt, float* colsum,
                  void* stream) {
  if (!dy || !dz || (relu && !y)) return fail(VL_EINVAL, "act_bwd: bad arguments");
  if (!dzt && C % 4 == 0 && !(((uintptr_t)dy | (uintptr_t)dz) & 15) && !((uintptr_t)y & 7) && (R + 255) / 256 <= 65535) {
    k_act_bwd4<<<dim3((unsigned)((C + 31) / 32), (unsigned)((R + 255) / 256)), 256, 0, (cudaStream_t)stream>>>(
        dy, (const bf16*)y, R, C, relu, (bf16*)dz, colsum, (R + 31) / 32);
    return launch_check("act_bwd");
  }
  dim3 grid((C + 31) / 32, (R + 31) / 32), block(32, 8);
  k_act_bwd<<<grid, block, 0, (cudaStream_t)stream>>>(dy, (const bf16*)y, R, C, relu, (bf16*)dz, (bf16*)dzt, colsum,
                                                      (R + 31) / 32);
  return launch_check("act_bwd");
}

int vl_nn_bias_grad(const float* colsum, int R, int C, float* db, void* stream) {
  if (!colsum || !db) return fail(VL_EINVAL, "bias_grad: bad arguments");
  k_bias_grad<<<C, 256, 0, (cudaStream_t)stream>>>(colsum, (R + 31) / 32, db);
  return launch_check("bias_grad");
}

int vl_nn_transpose_bf16(const void* a, int R, int C, void* at, void* stream) {
  if (!a || !at || (R & 1) || (C & 1)) return fail(VL_EINVAL, "transpose: bad arguments (R and C must be even)");
  if (((uintptr_t)a & 3) || ((uintptr_t)at & 3)) return fail(VL_EINVAL, "transpose: buffers must be 4-byte aligned");
  dim3 grid((C + 63) / 64, (R + 63) / 64), block(32, 8);
  k_transpose_bf16<<<grid, block, 0, (cudaStream_t)stream>>>((const bf16*)a, R, C, (bf16*)at);
  return launch_check("transpose");
}

int vl_nn_flip_weights(const void* w, int cout, int cin, int kp, int kpf, void* wf, void* stream) {
  if (!w || !wf || kp < 9 * cin || kpf < 9 * cout) return fail(VL_EINVAL, "flip_weights: bad arguments");
  k_flip_weights<<<grid_for((long long)cin * kpf), 256, 0, (cudaStream_t)stream>>>((const bf16*)w, cout, cin, kp, kpf,
                                                                                  (bf16*)wf);
  return launch_check("flip_weights");
}

int vl_nn_up2(const void* x, int B, int H, int W, int C, void* y, int ctot, int coff, void* stream) {
  if (!x || !y || coff + C > ctot) return fail(VL_EINVAL, "up2: bad arguments");
  if (grouped(x, y, 4LL * B * H * W * C, C, ctot, coff, 8)) {
    const unsigned n = (unsigned)((long long)B * H * W * C / 8);
    k_up2_v<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const uint4*)x, n, (unsigned)H, (unsigned)W, (unsigned)(C / 8),
                                                           (uint4*)y, (unsigned)(ctot / 8), (unsigned)(coff / 8));
    return launch_check("up2");
  }
  k_up2<<<grid_for(4LL * B * H * W * C), 256, 0, (cudaStream_t)stream>>>((const bf16*)x, B, H, W, C, (bf16*)y, ctot, coff);
  return launch_check("up2");
}

int vl_nn_up2_bwd(const float* dy, int B, int H, int W, int C, int ctot, int coff, float* dx, int accumulate,
                  void* stream) {
  if (!dy || !dx || coff + C > ctot) return fail(VL_EINVAL, "up2_bwd: bad arguments");
  if (grouped(dy, dx, (long long)B * H * W * C, C, ctot, coff, 4)) {
    const unsigned n = (unsigned)((long long)B * H * W * C / 4);
    k_up2_bwd_v<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const float4*)dy, n, (unsigned)W, (unsigned)(C / 4),
                                                               (unsigned)(ctot / 4), (unsigned)(coff / 4), (float4*)dx, accumulate);
    return launch_check("up2_bwd");
  }
  k_up2_bwd<<<grid_for((long long)B * H * W * C), 256, 0, (cudaStream_t)stream>>>(dy, B, H, W, C, ctot, coff, dx,
                                                                                  accumulate);
  return launch_check("up2_bwd");
}

int vl_nn_copy_channels(const void* x, long long R, int C, void* y, int ctot, int coff, void* stream) {
  if (!x || !y || coff + C > ctot) return fail(VL_EINVAL, "copy_channels: bad arguments");
  if (grouped(x, y, R * C, C, ctot, coff, 8)) {
    const unsigned n = (unsigned)(R * C / 8);
    k_copy_channels_v<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const uint4*)x, n, (unsigned)(C / 8), (uint4*)y,
                                                                     (unsigned)(ctot / 8), (unsigned)(coff / 8));
    return launch_check("copy_channels");
  }
  k_copy_channels<<<grid_for(R * C), 256, 0, (cudaStream_t)stream>>>((const bf16*)x, R, C, (bf16*)y, ctot, coff);
  return launch_check("copy_channels");
}

int vl_nn_slice_channels(const float* y, long long R, int ctot, int coff, int C, float* x, int accumulate,
                         void* stream) {
  if (!x || !y || coff + C > ctot) return fail(VL_EINVAL, "slice_channels: bad arguments");
  if (grouped(y, x, R * C, C, ctot, coff, 4)) {
    const unsigned n = (unsigned)(R * C / 4);
    k_slice_channels_v<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>((const float4*)y, n, (unsigned)(C / 4),
                                                                      (unsigned)(ctot / 4), (unsigned)(coff / 4), (float4*)x,
                                                                      accumulate);
    return launch_check("slice_channels");
  }
  k_slice_channels_f32<<<grid_for(R * C), 256, 0, (cudaStream_t)stream>>>(y, R, ctot, coff, C, x, accumulate);
  return launch_check("slice_channels");
}

int vl_nn_mse(const float* out, const float* tgt, const float* w, long long R, int C, int cuse, double inv_count,
              float* dout, double* partial, int blocks, void* stream) {
  if (!out || !tgt || !w || !dout || !partial || blocks < 1 || cuse < 1 || cuse > C)
    return fail(VL_EINVAL, "mse: bad arguments");
  k_mse<<<blocks, 256, 0, (cudaStream_t)stream>>>(out, tgt, w, R, C, cuse, inv_count, dout, partial);
  return launch_check("mse");
}

int vl_nn_adam(float* w, const float* g, float* m, float* v, long long n, float lr, float b1, float b2, float eps,
               int step, void* wb, void* stream) {
  if (!w || !g || !m || !v || step < 1) return fail(VL_EINVAL, "adam: bad arguments");
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(w, g, m, v, n, lr, b1, b2, eps, c1, c2, (bf16*)wb);
  return launch_check("adam");
}

int vl_nn_f32_to_bf16(const float* a, long long n, void* b, void* stream) {
  if (!a || !b) return fail(VL_EINVAL, "f32_to_bf16: bad arguments");
  k_f32_to_bf16<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(a, n, (bf16*)b);
  return launch_check("f32_to_bf16");
}

}  // extern "C"
