// Convolutions of the warm-start network as implicit GEMMs on tcgen05 (3x3, padding 1, stride 1 or 2,
// or 1x1; NHWC BF16 activations, FP32 accumulation): the operand that im2col would write out is loaded
// tap by tap with TMA boxes of the activation tensor itself (4-D map C, W, H, B; the box of a tile is
// shifted by the tap, and what lies outside the image reads as zero, which is the padding).
//
// The K order is that of the im2col matrix, (tap, channel), in tensor-core steps of 16: every product
// is accumulated in the order in which the GEMM over the materialised matrix accumulates it, so the
// results are the same bit for bit.
//
//   k_conv    y[pixel, n] = epilogue(sum over (tap, c) of x[pixel + tap, c] w[n, (tap, c)]): the forward
//             pass, and the input gradient of a stride-1 layer (dz with mirrored weights). Persistent:
//             a block takes tiles of 128 pixels (bw x bh of one image) x bn channels in turn; warp 0
//             loads, warp 1 issues the MMAs, warps 2-5 read the accumulator of one tile while the next
//             is computed in the other (two accumulators in TMEM).
//   k_wgrad   gw[(tap, c), n] = sum over pixels of x[pixel + tap, c] dz[pixel, n]: both operands MN-major,
//             64 pixels of K at a time in row order, split over K as the plain GEMM splits it.
//
// Bound: the tile loads (x nine times through the L2, one box a tap) instead of the HBM round trip of the
// nine-fold matrix. B200, batch 16, us of im2col + GEMM -> k_conv: 128 x 256 pixels 32 -> 32 channels 129 +
// 76 -> 56, 96 -> 32 340 + 185 -> 144 (k_conv_rows below: 24 and 61); 64 x 128 64 -> 64 63 + 55 -> 23, 192 -> 64
// 170 + 103 -> 44; 32 x 64 128 -> 128 35 + 41 -> 17; 16 x 32 256 -> 256 21 + 39 -> 21. Weight gradients, GEMM over the matrix -> k_wgrad:
// 32 x 32 87 -> 67, 96 x 32 215 -> 164 (k_wgrad_rows: 43 and 79), 64 x 64 42 -> 27, 128 x 128 45 -> 23.
// Every wait on an mbarrier is bounded, as in vl_gemm.cuh.
#pragma once

#include "vl_gemm.cuh"

namespace vl {
namespace gemm {

constexpr int kConvThreads = 192;
constexpr int kConvMaxStages = 8;

struct ConvParams {
  int tiles, tiles_x, tiles_y;   // 128-pixel tiles: all, per row of tiles, per image
  int bw, bh, log2_bw;           // pixels of a tile (bw * bh = 128)
  int Ho, Wo, stride;
  int taps, chunks;              // 9 or 1; KC-channel chunks of C
  int pad;
  int stages, bn, tmem_cols;     // tmem_cols: columns of one accumulator (a power of two)
  int kb_split;                  // K blocks accumulated before the partial sum is added to `out` (all: kblocks)
  EpiParams ep;
};

__device__ __forceinline__ void tma_load_4d(const CUtensorMap* map, uint64_t* bar, void* dst, int c, int x, int y, int b) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c), "r"(x), "r"(y), "r"(b)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// K-major tile of 32-channel rows with 64-byte swizzle: rows of 64 bytes, 8-row (512-byte) atoms.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)1u << 16;
  d |= (uint64_t)(512u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)4u << 61;   // SWIZZLE_64B
  return d;
}

// MN-major tile of 32-wide column blocks with 64-byte swizzle: 8 K rows of 64 bytes form a 512-byte atom;
// the next 8 K rows follow it, the next 32 columns are 64 K rows = 4096 bytes on.
__device__ __forceinline__ uint64_t smem_desc_sw64_mn(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)(4096u >> 4) << 16;
  d |= (uint64_t)(512u >> 4) << 32;
  d |= (uint64_t)1u << 46;
  d |= (uint64_t)4u << 61;
  return d;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

// Bytes to expect of loads of `bytes`: with the test hook on, more than come, so that the waits for them run out.
__device__ __forceinline__ uint32_t expected(uint32_t bytes, int drop_load) { return bytes + (drop_load ? 16u : 0u); }

// One lane of the (converged) warp. The issuing loops run on the whole warp, so that descriptors and
// counters are warp-uniform values (the MMA takes them from uniform registers), and this lane issues.
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)));
}

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The epilogue of one accumulator: this lane's row of it (TMEM address `acc`, bn columns from column n0 of the
// output) to row `row` of `out`, if valid; `add`: onto the FP32 values there. By whole warps.
__device__ __forceinline__ void store_tile(const EpiParams& ep, uint32_t acc, int bn, int n0, bool valid, size_t row, bool add,
                                           void* out) {
  for (int c0 = 0; c0 < bn; c0 += 32) {
    uint32_t v[32];
    tmem_ld32(acc + (uint32_t)c0, v);
    if (valid) {
      const int cols = min(32, ep.n_valid - (n0 + c0));
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        float4 bv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if ((ep.flags & EPI_BIAS) && j < cols) bv = __ldg(reinterpret_cast<const float4*>(ep.bias + n0 + c0 + j));
        const float bj[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float f = __uint_as_float(v[j + i]) + bj[i];
          if (ep.flags & EPI_RELU) f = fmaxf(f, 0.0f);
          v[j + i] = __float_as_uint(f);
        }
      }
      // 32 bytes a store: whole sectors, though a lane's row lies apart from its neighbours'
      if (ep.flags & EPI_BF16) {
        __nv_bfloat16* o = (__nv_bfloat16*)out + row * ep.ldc + n0 + c0;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          if (j < cols) {                   // (the column count is a multiple of 8)
            uint32_t u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[j + 2 * i]), __uint_as_float(v[j + 2 * i + 1]));
              u[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(o + j) = make_uint4(u[0], u[1], u[2], u[3]);
          }
        }
      } else {
        float* o = (float*)out + row * ep.ldc + n0 + c0;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          if (j < cols) {
            if (add) {
              const float4 e0 = *reinterpret_cast<const float4*>(o + j), e1 = *reinterpret_cast<const float4*>(o + j + 4);
              const float e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
#pragma unroll
              for (int i = 0; i < 8; ++i) v[j + i] = __float_as_uint(e[i] + __uint_as_float(v[j + i]));
            }
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + j), "r"(v[j]), "r"(v[j + 1]),
                         "r"(v[j + 2]), "r"(v[j + 3]), "r"(v[j + 4]), "r"(v[j + 5]), "r"(v[j + 6]), "r"(v[j + 7])
                         : "memory");
          }
        }
      }
    }
    __syncwarp();
  }
}

template <int KC>
__host__ __device__ constexpr int conv_stage_bytes(int bn) {
  return (BM + bn) * KC * 2;
}

template <int KC>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv(const __grid_constant__ CUtensorMap tmA,
                                                          const __grid_constant__ CUtensorMap tmB,
                                                          const __grid_constant__ ConvParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kConvMaxStages], empty[kConvMaxStages], tfull[2], tempty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int failed, issued_loads;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n0 = (int)blockIdx.y * p.bn;
  const int kblocks = p.taps * p.chunks;
  const int stage_bytes = conv_stage_bytes<KC>(p.bn);
  const EpiParams& ep = p.ep;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    failed = 0;
    issued_loads = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"((uint32_t)(2 * p.tmem_cols)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;

  if (threadIdx.x == 0) {
    // loads: the stages of the ring in turn, in tile and K order (the counters are kept, not divided: a
    // division in this loop costs as much as the load it issues)
    const uint32_t bytes = expected((uint32_t)stage_bytes, ep.drop_load);
    int s = 0, issued = 0;
    uint32_t phase = 1;                         // of the empty barriers: the first round passes at once
    bool ok = true;
    for (int t = (int)blockIdx.x; t < p.tiles && ok; t += (int)gridDim.x) {
      const int per = p.tiles_x * p.tiles_y;
      const int b = t / per, q = t - b * per, ty = q / p.tiles_x, tx = q - ty * p.tiles_x;
      const int x0 = tx * p.bw * p.stride - p.pad, y0 = ty * p.bh * p.stride - p.pad;
      int ky = 0, kx = 0, c0 = 0;
      for (int kb = 0; kb < kblocks; ++kb) {
        if (!mbar_wait(&empty[s], phase, ep.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        uint8_t* sa = smem + s * stage_bytes;
        mbar_expect_tx(&full[s], bytes);
        tma_load_4d(&tmA, &full[s], sa, c0, x0 + kx, y0 + ky, b);
        tma_load_2d(&tmB, &full[s], sa + BM * KC * 2, kb * KC, n0);
        ++issued;
        if (++s == p.stages) {
          s = 0;
          phase ^= 1;
        }
        c0 += KC;
        if (c0 == p.chunks * KC) {
          c0 = 0;
          if (++kx == 3) {
            kx = 0;
            ++ky;
          }
        }
      }
    }
    issued_loads = issued;
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(p.bn);
    int s = 0, n = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < p.tiles && ok; t += (int)gridDim.x) {
      int left = 0, buf = 0;
      uint32_t acc = 0;
      for (int kb = 0; kb < kblocks; ++kb) {
        const bool fresh = left == 0;
        if (fresh) {                            // the next accumulator, once it has been read
          buf = n & 1;
          if (!mbar_wait(&tempty[buf], ((uint32_t)(n >> 1) & 1u) ^ 1u, ep.spin_limit)) {
            atomicExch(&failed, 1);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          acc = tmem + (uint32_t)(buf * p.tmem_cols);
          left = min(p.kb_split, kblocks - kb);
          ++n;
        }
        if (!mbar_wait(&full[s], phase, ep.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t a_addr = smem_u32(smem + s * stage_bytes), b_addr = a_addr + BM * KC * 2;
        const uint64_t da = KC == 64 ? smem_desc_sw128(a_addr) : smem_desc_sw64(a_addr);
        const uint64_t db = KC == 64 ? smem_desc_sw128(b_addr) : smem_desc_sw64(b_addr);
        --left;
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < KC / 16; ++k) mma_bf16(acc, da + 2u * k, db + 2u * k, idesc, (!fresh || k > 0) ? 1u : 0u);
          mma_commit(&empty[s]);
          if (left == 0) mma_commit(&tfull[buf]);
        }
        __syncwarp();
        if (++s == p.stages) {
          s = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp >= 2) {
    // epilogue: a warp reads the 32 rows of its TMEM lanes (its number modulo 4), a row per lane
    const int rows = (warp & 3) * 32;
    const int parts = (kblocks + p.kb_split - 1) / p.kb_split;
    int n = 0;
    bool ok = true;
    for (int t = (int)blockIdx.x; t < p.tiles && ok; t += (int)gridDim.x)
    for (int z = 0; z < parts; ++z, ++n) {
      const int buf = n & 1;
      const bool add = z > 0 || (ep.flags & EPI_ACCUM);
      if (!mbar_wait(&tfull[buf], (uint32_t)(n >> 1) & 1u, ep.spin_limit)) {
        atomicExch(&failed, 1);
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int per = p.tiles_x * p.tiles_y;
      const int b = t / per, q = t - b * per, ty = q / p.tiles_x, tx = q - ty * p.tiles_x;
      const int m = rows + lane;
      const int x = tx * p.bw + (m & (p.bw - 1)), y = ty * p.bh + (m >> p.log2_bw);
      const bool valid = x < p.Wo && y < p.Ho;
      const size_t row = ((size_t)b * p.Ho + y) * p.Wo + x;
      store_tile(ep, tmem + (uint32_t)(buf * p.tmem_cols) + ((uint32_t)rows << 16), p.bn, n0, valid, row, add, ep.out);
      // the accumulator is read: the MMAs of the tile after the next may overwrite it
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (failed && threadIdx.x == 0) {
    // drain (bounded): the copies that may still be landing in this block's shared memory
    const int issued = issued_loads;
    for (int it = issued > p.stages ? issued - p.stages : 0; it < issued; ++it)
      mbar_wait(&full[it % p.stages], (uint32_t)(it / p.stages) & 1u, ep.spin_limit);
    if (ep.err) atomicExch(ep.err, 1);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * p.tmem_cols)));
}

// ------------------------------------------------------------------ 3x3, stride 1, rows of 128 pixels
// k_conv loads every activation nine times (once a tap) and the weights once a tile. Here a block walks down a
// strip of 128-pixel rows: a ring of input rows (130 pixels, all channels) stays in shared memory, each
// tile of one output row adds one row to it, and the three taps of a row are the same shared-memory
// tile read 0, 1 or 2 pixels on (the swizzle is a function of the shared-memory address, so a descriptor
// that starts at a later row of the swizzled tile is valid). The weights of the block's channels stay in
// shared memory for all its tiles. K order and results as k_conv. Bound now by the issue and latency of its
// narrow MMAs (about 80 cycles each). B200, batch 16, k_conv -> here: 128 x 256 pixels 32 -> 32 channels 56 -> 24 us,
// 96 -> 32 144 -> 61, 32 -> 96 (FP32 result) 102 -> 59; 64 x 128 64 -> 64 23 -> 19.
struct RowsParams {
  int units, segs, tx, seg_rows;   // work units (image, column of tiles, segment of rows); rows of a segment
  int Ho, Wo;
  int chunks, bn, tmem_cols;       // KC-channel chunks of C
  int ring;                        // rows of the ring
  int box_bytes;                   // shared memory of one chunk of one row (130 pixels, 1024-byte aligned)
  EpiParams ep;
};
constexpr int kRowsMaxRing = 16;
constexpr int kRowPixels = BM + 2;

template <int KC>
__host__ __device__ constexpr int rows_box_bytes() {
  return (kRowPixels * KC * 2 + 1023) / 1024 * 1024;
}

// CH: KC-channel chunks of C, known to the compiler where that is 1, 2 or 3: the issuing thread's loop is then
// straight-line code of a few instructions an MMA (with a run-time loop over them it took 126 cycles an MMA of
// 32 channels, and was the kernel's time).
template <int KC, int CH>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv_rows(const __grid_constant__ CUtensorMap tmA,
                                                               const __grid_constant__ CUtensorMap tmB,
                                                               const __grid_constant__ RowsParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kRowsMaxRing], empty[kRowsMaxRing], wfull, tfull[2], tempty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int failed, issued_loads;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n0 = (int)blockIdx.y * p.bn;
  const int row_bytes = p.chunks * p.box_bytes, wtap_bytes = p.bn * KC * 2;
  uint8_t* weights = smem;                                  // [tap][chunk] tiles of bn rows
  uint8_t* rows = smem + (9 * p.chunks * wtap_bytes + 1023) / 1024 * 1024;
  const EpiParams& ep = p.ep;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.ring; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    mbar_init(&wfull, 1);
    failed = 0;
    issued_loads = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"((uint32_t)(2 * p.tmem_cols)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;

  if (threadIdx.x == 0) {
    const uint32_t bytes = expected((uint32_t)(p.chunks * kRowPixels * KC * 2), ep.drop_load);
    mbar_expect_tx(&wfull, (uint32_t)(9 * p.chunks * wtap_bytes));
    for (int k = 0; k < 9 * p.chunks; ++k) tma_load_2d(&tmB, &wfull, weights + k * wtap_bytes, k * KC, n0);
    int s = 0, issued = 0;
    uint32_t phase = 1;
    bool ok = true;
    for (int u = (int)blockIdx.x; u < p.units && ok; u += (int)gridDim.x) {
      const int q = u / p.segs, seg = u - q * p.segs, b = q / p.tx, tx = q - b * p.tx;
      const int y0 = seg * p.seg_rows, y1 = min(y0 + p.seg_rows, p.Ho);
      for (int y = y0 - 1; y <= y1; ++y) {                  // (rows -1 and Ho read zero)
        if (!mbar_wait(&empty[s], phase, ep.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], bytes);
        for (int c = 0; c < p.chunks; ++c) tma_load_4d(&tmA, &full[s], rows + s * row_bytes + c * p.box_bytes, c * KC, tx * BM - 1, y, b);
        ++issued;
        if (++s == p.ring) {
          s = 0;
          phase ^= 1;
        }
      }
    }
    issued_loads = issued;
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(p.bn);
    bool ok = mbar_wait(&wfull, 0, ep.spin_limit);
    if (!ok) atomicExch(&failed, 1);
    int s = 0, n = 0;                                       // s: ring slot of the row above the tile
    uint32_t phase = 0;                                     // of that slot
    for (int u = (int)blockIdx.x; u < p.units && ok; u += (int)gridDim.x) {
      const int seg = u % p.segs;
      const int y0 = seg * p.seg_rows, y1 = min(y0 + p.seg_rows, p.Ho);
      for (int y = y0; y < y1 && ok; ++y, ++n) {
        const int buf = n & 1;
        if (!mbar_wait(&tempty[buf], ((uint32_t)(n >> 1) & 1u) ^ 1u, ep.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t acc = tmem + (uint32_t)(buf * p.tmem_cols);
        const uint64_t wd = KC == 64 ? smem_desc_sw128(smem_u32(weights)) : smem_desc_sw64(smem_u32(weights));
        const uint64_t rd = KC == 64 ? smem_desc_sw128(smem_u32(rows)) : smem_desc_sw64(smem_u32(rows));
        const uint32_t wstep = (uint32_t)wtap_bytes >> 4, cstep = (uint32_t)p.box_bytes >> 4;   // in descriptor units
        int slot = s;
        uint32_t ph = phase;
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          if (ok && !mbar_wait(&full[slot], ph, ep.spin_limit)) {
            atomicExch(&failed, 1);
            ok = false;
          }
          if (!ok) continue;
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint64_t ra = rd + (uint64_t)((uint32_t)(slot * row_bytes) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int kx = 0; kx < 3; ++kx) {
              const int chunks = CH > 0 ? CH : p.chunks;
#pragma unroll
              for (int c = 0; c < (CH > 0 ? CH : chunks); ++c) {
                const uint64_t da = ra + (uint64_t)((uint32_t)(kx * KC / 8) + (uint32_t)c * cstep);
                const uint64_t db = wd + (uint64_t)((uint32_t)((ky * 3 + kx) * chunks + c) * wstep);
#pragma unroll
                for (int k = 0; k < KC / 16; ++k)
                  mma_bf16(acc, da + 2u * k, db + 2u * k, idesc, (ky | kx | c | k) != 0 ? 1u : 0u);
              }
            }
          }
          __syncwarp();
          if (++slot == p.ring) {
            slot = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        if (elect_one()) {
          mma_commit(&empty[s]);                            // the row above is done with
          mma_commit(&tfull[buf]);
        }
        __syncwarp();
        if (++s == p.ring) {
          s = 0;
          phase ^= 1;
        }
      }
      // the last two rows of the segment
      for (int i = 0; i < 2 && ok; ++i) {
        if (elect_one()) mma_commit(&empty[s]);
        __syncwarp();
        if (++s == p.ring) {
          s = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp >= 2) {
    const int prow = (warp & 3) * 32;
    int n = 0;
    bool ok = true;
    for (int u = (int)blockIdx.x; u < p.units && ok; u += (int)gridDim.x) {
      const int q = u / p.segs, seg = u - q * p.segs, b = q / p.tx, tx = q - b * p.tx;
      const int y0 = seg * p.seg_rows, y1 = min(y0 + p.seg_rows, p.Ho);
      const int x = tx * BM + prow + lane;
      for (int y = y0; y < y1; ++y, ++n) {
        const int buf = n & 1;
        if (!mbar_wait(&tfull[buf], (uint32_t)(n >> 1) & 1u, ep.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        store_tile(ep, tmem + (uint32_t)(buf * p.tmem_cols) + ((uint32_t)prow << 16), p.bn, n0, x < p.Wo,
                   ((size_t)b * p.Ho + y) * p.Wo + x, (ep.flags & EPI_ACCUM) != 0, ep.out);
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[buf]);
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (failed && threadIdx.x == 0) {
    mbar_wait(&wfull, 0, ep.spin_limit);
    const int issued = issued_loads;
    for (int it = issued > p.ring ? issued - p.ring : 0; it < issued; ++it)
      mbar_wait(&full[it % p.ring], (uint32_t)(it / p.ring) & 1u, ep.spin_limit);
    if (ep.err) atomicExch(ep.err, 1);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)(2 * p.tmem_cols)));
}

// ------------------------------------------------------------------ weight gradient
struct WgradParams {
  int Ho, Wo, stride, pad, taps;
  int C;                         // channels; a K block is 64 pixels, of a row's part or of whole rows
  int kblocks, kb_per, stages, bn;
  EpiParams ep;                  // FP32 rows (tap, c) of `out`, split-K partial results split_stride apart
};

template <int KC>
__host__ __device__ constexpr int wgrad_stage_bytes(int bn) {
  return BM * 64 * 2 + bn * 64 * 2;
}

template <int KC>
__global__ void __launch_bounds__(128, 1) k_wgrad(const __grid_constant__ CUtensorMap tmA,
                                                  const __grid_constant__ CUtensorMap tmB,
                                                  const __grid_constant__ WgradParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kConvMaxStages], empty[kConvMaxStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed, issued_loads;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int m0 = (int)blockIdx.x * BM, n0 = (int)blockIdx.y * p.bn;
  const int kb_first = (int)blockIdx.z * p.kb_per;
  const int kblocks = min(p.kblocks - kb_first, p.kb_per);
  const int stage_bytes = wgrad_stage_bytes<KC>(p.bn);
  const uint32_t tmem_cols = p.bn <= 32 ? 32u : (p.bn <= 64 ? 64u : (p.bn <= 128 ? 128u : 256u));
  const EpiParams& ep = p.ep;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    failed = 0;
    issued_loads = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  if (threadIdx.x == 0) {
    const uint32_t bytes = expected((uint32_t)stage_bytes, ep.drop_load);
    // the KC-wide column blocks of this tile: their tap and first channel (past the last: all zero)
    constexpr int NB = BM / KC;
    int kx[NB], ky[NB], c0[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const int row = m0 + i * KC, tap = row / p.C;
      c0[i] = row - tap * p.C;
      ky[i] = tap < p.taps ? (p.taps == 9 ? tap / 3 : 0) : -(1 << 24);
      kx[i] = p.taps == 9 ? tap % 3 : 0;
    }
    int issued = 0, s = 0;
    uint32_t phase = 1;
    int r0 = kb_first * 64;
    int x = r0 % p.Wo, y = r0 / p.Wo, b = y / p.Ho;
    y -= b * p.Ho;
    for (int kb = 0; kb < kblocks; ++kb) {
      if (!mbar_wait(&empty[s], phase, ep.spin_limit)) { atomicExch(&failed, 1); break; }
      uint8_t* sa = smem + s * stage_bytes;
      mbar_expect_tx(&full[s], bytes);
#pragma unroll
      for (int i = 0; i < NB; ++i)
        tma_load_4d(&tmA, &full[s], sa + i * (64 * KC * 2), c0[i], x * p.stride - p.pad + kx[i], y * p.stride - p.pad + ky[i], b);
      for (int c = 0; c < p.bn / 64; ++c) tma_load_2d(&tmB, &full[s], sa + BM * 64 * 2 + 8192 * c, n0 + 64 * c, r0);
      issued = kb + 1;
      if (++s == p.stages) {
        s = 0;
        phase ^= 1;
      }
      r0 += 64;
      if (p.Wo >= 64) {
        x += 64;
        if (x == p.Wo) {
          x = 0;
          ++y;
        }
      } else {
        y += 64 / p.Wo;
      }
      if (y == p.Ho) {
        y = 0;
        ++b;
      }
    }
    issued_loads = issued;
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(p.bn, OP_A_MN | OP_B_MN);
    int s = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < kblocks; ++kb) {
      if (!mbar_wait(&full[s], phase, ep.spin_limit)) { atomicExch(&failed, 1); break; }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t a_addr = smem_u32(smem + s * stage_bytes), b_addr = a_addr + BM * 64 * 2;
      const uint64_t da = KC == 64 ? smem_desc_sw128_mn(a_addr) : smem_desc_sw64_mn(a_addr), db = smem_desc_sw128_mn(b_addr);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k)                         // 16 K rows further: two 8-row atoms
          mma_bf16(tmem, da + (uint64_t)((KC == 64 ? 128u : 64u) * k), db + 128u * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        mma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == p.stages) {
        s = 0;
        phase ^= 1;
      }
    }
    if (elect_one()) mma_commit(&done);
  }
  __syncwarp();
  const bool have = mbar_wait(&done, 0, ep.spin_limit);
  if (!have) atomicExch(&failed, 1);
  asm volatile("tcgen05.fence::after_thread_sync;");
  __syncthreads();
  const bool good = !failed;
  if (!good && threadIdx.x == 0) {
    const int issued = issued_loads;
    for (int kb = issued > p.stages ? issued - p.stages : 0; kb < issued; ++kb)
      mbar_wait(&full[kb % p.stages], (uint32_t)(kb / p.stages) & 1u, ep.spin_limit);
    if (ep.err) atomicExch(ep.err, 1);
  }
  if (good) {
    const int row = m0 + warp * 32 + lane;
    for (int c0 = 0; c0 < p.bn; c0 += 32) {
      uint32_t v[32];
      tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
      const int cols = min(32, ep.n_valid - (n0 + c0));
      if (row < ep.m_valid) {
        float* o = (float*)ep.out + (size_t)blockIdx.z * ep.split_stride + (size_t)row * ep.ldc + n0 + c0;
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          if (j < cols)
            *reinterpret_cast<float4*>(o + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                            __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols));
}

// Weight gradient of a stride-1 3x3 layer whose output rows are whole 64-pixel blocks. k_wgrad loads the
// pixels of a K block once per tap; here a block of the grid takes one kernel row ky and one KC-channel chunk, and
// the three taps of the row are one operand: column block kx of the MN-major tile is the same shared memory
// read kx pixels on (leading offset = one pixel's row), 128 / KC of them to an MMA; what lies past kx = 2 is
// computed and dropped. K order, split and results as k_wgrad.
struct WgradRowsParams {
  int Ho, Wo, C, chunks;         // chunks: of KC channels
  int kblocks, kb_per, stages, bn, stage_bytes, a_bytes;
  int kp;
  EpiParams ep;
};
constexpr int kWgradPixels = 64 + 4;

template <int KC>
__global__ void __launch_bounds__(128, 1) k_wgrad_rows(const __grid_constant__ CUtensorMap tmA,
                                                       const __grid_constant__ CUtensorMap tmB,
                                                       const __grid_constant__ WgradRowsParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kConvMaxStages], empty[kConvMaxStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed, issued_loads;
  constexpr int ACCS = KC == 64 ? 2 : 1;                    // taps 0-1 and 2, or all three
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int ky = (int)blockIdx.x % 3, c0 = (int)blockIdx.x / 3 * KC, n0 = (int)blockIdx.y * p.bn;
  const int kb_first = (int)blockIdx.z * p.kb_per;
  const int kblocks = min(p.kblocks - kb_first, p.kb_per);
  const uint32_t acc_cols = p.bn <= 32 ? 32u : (p.bn <= 64 ? 64u : (p.bn <= 128 ? 128u : 256u));
  const uint32_t tmem_cols = acc_cols * ACCS;
  const EpiParams& ep = p.ep;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    failed = 0;
    issued_loads = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  if (threadIdx.x == 0) {
    int issued = 0, s = 0;
    uint32_t phase = 1;
    int r0 = kb_first * 64;
    int x = r0 % p.Wo, y = r0 / p.Wo, b = y / p.Ho;
    y -= b * p.Ho;
    const int boxes = (p.bn + 63) / 64;
    const uint32_t bytes = expected((uint32_t)(kWgradPixels * KC * 2 + p.bn * 128), ep.drop_load);
    for (int kb = 0; kb < kblocks; ++kb) {
      if (!mbar_wait(&empty[s], phase, ep.spin_limit)) { atomicExch(&failed, 1); break; }
      uint8_t* sa = smem + s * p.stage_bytes;
      mbar_expect_tx(&full[s], bytes);
      tma_load_4d(&tmA, &full[s], sa, c0, x - 1, y + ky - 1, b);
      for (int c = 0; c < boxes; ++c) tma_load_2d(&tmB, &full[s], sa + p.a_bytes + 8192 * c, n0 + 64 * c, r0);
      issued = kb + 1;
      if (++s == p.stages) {
        s = 0;
        phase ^= 1;
      }
      r0 += 64;
      x += 64;
      if (x == p.Wo) {
        x = 0;
        if (++y == p.Ho) {
          y = 0;
          ++b;
        }
      }
    }
    issued_loads = issued;
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(p.bn, OP_A_MN | OP_B_MN);
    const bool narrow = p.bn == 32;
    int s = 0;
    uint32_t phase = 0;
    for (int kb = 0; kb < kblocks; ++kb) {
      if (!mbar_wait(&full[s], phase, ep.spin_limit)) { atomicExch(&failed, 1); break; }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t a_addr = smem_u32(smem + s * p.stage_bytes), b_addr = a_addr + (uint32_t)p.a_bytes;
      // the swizzled-tile descriptors with the leading offset of one pixel
      uint64_t da = KC == 64 ? smem_desc_sw128_mn(a_addr) : smem_desc_sw64_mn(a_addr);
      da = (da & ~((uint64_t)0x3FFFu << 16)) | ((uint64_t)(KC * 2 >> 4) << 16);
      const uint64_t db = narrow ? smem_desc_sw64_mn(b_addr) : smem_desc_sw128_mn(b_addr);
      const uint32_t bstep = narrow ? 64u : 128u;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {                       // 16 pixels further
#pragma unroll
          for (int q = 0; q < ACCS; ++q)
            mma_bf16(tmem + acc_cols * q, da + (uint64_t)((KC == 64 ? 128u : 64u) * k + q * 2u * (KC * 2u >> 4)),
                     db + (uint64_t)(bstep * k), idesc, (kb > 0 || k > 0) ? 1u : 0u);
        }
        mma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == p.stages) {
        s = 0;
        phase ^= 1;
      }
    }
    if (elect_one()) mma_commit(&done);
  }
  __syncwarp();
  const bool have = mbar_wait(&done, 0, ep.spin_limit);
  if (!have) atomicExch(&failed, 1);
  asm volatile("tcgen05.fence::after_thread_sync;");
  __syncthreads();
  const bool good = !failed;
  if (!good && threadIdx.x == 0) {
    const int issued = issued_loads;
    for (int kb = issued > p.stages ? issued - p.stages : 0; kb < issued; ++kb)
      mbar_wait(&full[kb % p.stages], (uint32_t)(kb / p.stages) & 1u, ep.spin_limit);
    if (ep.err) atomicExch(ep.err, 1);
  }
  if (good) {
    float* out = (float*)ep.out + (size_t)blockIdx.z * ep.split_stride;
    const int m = warp * 32 + lane;
#pragma unroll
    for (int q = 0; q < ACCS; ++q) {
      const int kx = 2 * q + m / KC, row = (ky * 3 + kx) * p.C + c0 + m % KC;
      store_tile(ep, tmem + acc_cols * q + ((uint32_t)(warp * 32) << 16), p.bn, n0, kx < 3, (size_t)row, false, out);
    }
    // the rows past 9 C are zero
    if (blockIdx.x == 0)
      for (int i = (int)threadIdx.x; i < (p.kp - 9 * p.C) * p.bn; i += 128) {
        const int n = n0 + i % p.bn;
        if (n < ep.n_valid) out[(size_t)(9 * p.C + i / p.bn) * ep.ldc + n] = 0.0f;
      }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols));
}

// ------------------------------------------------------------------ the 4-channel input layer
// A pixel has 8 bytes: less than a TMA box row. Four warps gather the 9 x 4 patch of a pixel a thread and write it as
// the row (taps in order, zeros to 64) of a 128-byte swizzled tile, which serves the forward product as the K-major
// operand (128 pixels) and the weight gradient as the MN-major one (64 pixels of K). Products as over the
// im2col matrix, bit for bit (steps of 16 that are zero throughout are left out of the forward pass). B200, 16 x 128 x
// 256 pixels, 4 -> 32 channels: im2col 93 + GEMM 39 us -> 23, weight gradient over the matrix 37 -> 31.
struct FirstParams {
  int B, H, W;
  const __nv_bfloat16* x;        // [B][H][W][4]
  long long pixels;              // B H W
  int tiles;                     // forward: 128-pixel tiles
  int kblocks, kb_per;           // weight gradient: 64-pixel K blocks
  int bn, kp;
  EpiParams ep;
};
constexpr int kFirstStages = 4;

// Row `row` of a swizzled tile: the patch of pixel r (zero past the last pixel). Chunks of 16 bytes [0, CHUNKS).
template <int CHUNKS>
__device__ __forceinline__ void patch_row(const FirstParams& p, long long r, uint8_t* tile, int row) {
  uint2 t[9];
  const bool in = r < p.pixels;
  const unsigned q = (unsigned)(in ? r : 0);
  const int x = (int)(q % (unsigned)p.W), yb = (int)(q / (unsigned)p.W), y = yb % p.H;
  const uint2* src = reinterpret_cast<const uint2*>(p.x) + q;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int dy = k / 3 - 1, dx = k % 3 - 1;
    const bool ok = in && y + dy >= 0 && y + dy < p.H && x + dx >= 0 && x + dx < p.W;
    t[k] = ok ? __ldg(src + dy * p.W + dx) : make_uint2(0u, 0u);
  }
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) {
    const uint2 a = 2 * c < 9 ? t[2 * c < 9 ? 2 * c : 0] : make_uint2(0u, 0u);
    const uint2 b = 2 * c + 1 < 9 ? t[2 * c + 1 < 9 ? 2 * c + 1 : 0] : make_uint2(0u, 0u);
    *reinterpret_cast<uint4*>(tile + row * 128 + ((c ^ (row & 7)) << 4)) = make_uint4(a.x, a.y, b.x, b.y);
  }
}

// Warps 0-3 gather, warp 4 issues, warps 5-8 store.
__global__ void __launch_bounds__(288, 1) k_conv_first(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ FirstParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kFirstStages], empty[kFirstStages], wfull, tfull[2], tempty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  uint8_t* weights = smem + kFirstStages * 16384;
  const EpiParams& ep = p.ep;
  const uint32_t cols = p.bn <= 32 ? 32u : (p.bn <= 64 ? 64u : (p.bn <= 128 ? 128u : 256u));
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFirstStages; ++s) {
      mbar_init(&full[s], 128);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    mbar_init(&wfull, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(2 * cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  bool ok = true;
  if (warp < 4) {
    int s = 0;
    uint32_t phase = 1;
    for (int t = (int)blockIdx.x; t < p.tiles; t += (int)gridDim.x) {
      if (!mbar_wait(&empty[s], phase, ep.spin_limit)) {
        atomicExch(&failed, 1);
        break;
      }
      patch_row<6>(p, (long long)t * BM + threadIdx.x, smem + s * 16384, (int)threadIdx.x);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tensor cores read it
      mbar_arrive(&full[s]);
      if (++s == kFirstStages) {
        s = 0;
        phase ^= 1;
      }
    }
  } else if (warp == 4) {
    const uint32_t idesc = instr_desc_bf16(p.bn);
    if (elect_one()) {
      mbar_expect_tx(&wfull, expected((uint32_t)(p.bn * 128), ep.drop_load));
      tma_load_2d(&tmB, &wfull, weights, 0, 0);
    }
    __syncwarp();
    if (!mbar_wait(&wfull, 0, ep.spin_limit)) {
      atomicExch(&failed, 1);
      ok = false;
    }
    const uint64_t db = smem_desc_sw128(smem_u32(weights));
    int s = 0, n = 0;
    uint32_t phase = 0;
    for (int t = (int)blockIdx.x; t < p.tiles && ok; t += (int)gridDim.x, ++n) {
      const int buf = n & 1;
      if (!mbar_wait(&tempty[buf], ((uint32_t)(n >> 1) & 1u) ^ 1u, ep.spin_limit) || !mbar_wait(&full[s], phase, ep.spin_limit)) {
        atomicExch(&failed, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint64_t da = smem_desc_sw128(smem_u32(smem + s * 16384));
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 3; ++k) mma_bf16(tmem + (uint32_t)buf * cols, da + 2u * k, db + 2u * k, idesc, k > 0 ? 1u : 0u);
        mma_commit(&empty[s]);
        mma_commit(&tfull[buf]);
      }
      __syncwarp();
      if (++s == kFirstStages) {
        s = 0;
        phase ^= 1;
      }
    }
  } else {
    const int prow = (warp & 3) * 32;
    int n = 0;
    for (int t = (int)blockIdx.x; t < p.tiles; t += (int)gridDim.x, ++n) {
      const int buf = n & 1;
      if (!mbar_wait(&tfull[buf], (uint32_t)(n >> 1) & 1u, ep.spin_limit)) {
        atomicExch(&failed, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const long long r = (long long)t * BM + prow + lane;
      store_tile(ep, tmem + (uint32_t)buf * cols + ((uint32_t)prow << 16), p.bn, 0, r < p.pixels, (size_t)r, false, ep.out);
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[buf]);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (failed && threadIdx.x == 0) {
    mbar_wait(&wfull, 0, ep.spin_limit);        // the weights' copy may still be landing
    if (ep.err) atomicExch(ep.err, 1);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 4) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * cols));
}

// gwt[k, n] over the K blocks of this split: warps 0-3 gather (two threads a pixel), warp 4 loads dz and issues.
__global__ void __launch_bounds__(160, 1) k_wgrad_first(const __grid_constant__ CUtensorMap tmB, const __grid_constant__ FirstParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kFirstStages], empty[kFirstStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed, issued_loads;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int kb_first = (int)blockIdx.x * p.kb_per, kblocks = min(p.kblocks - kb_first, p.kb_per);
  const int stage_bytes = 8192 + p.bn * 128;
  const uint32_t cols = p.bn <= 64 ? 64u : (p.bn <= 128 ? 128u : 256u);
  const EpiParams& ep = p.ep;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kFirstStages; ++s) {
      mbar_init(&full[s], 65);                  // 64 gathering threads and the expected bytes of dz
      mbar_init(&empty[s], 1);
    }
    mbar_init(&done, 1);
    failed = 0;
    issued_loads = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  if (warp < 4) {
    // warps 0-1 take the even K blocks, warps 2-3 the odd ones
    for (int kb = warp >> 1; kb < kblocks; kb += 2) {
      const int s = kb % kFirstStages;
      if (!mbar_wait(&empty[s], ((uint32_t)(kb / kFirstStages) & 1u) ^ 1u, ep.spin_limit)) {
        atomicExch(&failed, 1);
        break;
      }
      const int row = (int)threadIdx.x & 63;
      patch_row<8>(p, (long long)(kb_first + kb) * 64 + row, smem + s * stage_bytes, row);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive(&full[s]);
    }
  } else {
    const uint32_t idesc = instr_desc_bf16(p.bn, OP_A_MN | OP_B_MN);
    const int boxes = p.bn / 64;
    int issued = 0;
    bool ok = true;
    auto load = [&](int kb) {                   // dz of K block kb
      const int s = kb % kFirstStages;
      if (!mbar_wait(&empty[s], ((uint32_t)(kb / kFirstStages) & 1u) ^ 1u, ep.spin_limit)) return false;
      if (elect_one()) {
        mbar_expect_tx(&full[s], expected((uint32_t)(p.bn * 128), ep.drop_load));
        for (int c = 0; c < boxes; ++c)
          tma_load_2d(&tmB, &full[s], smem + s * stage_bytes + 8192 + 8192 * c, 64 * c, (kb_first + kb) * 64);
      }
      __syncwarp();
      ++issued;
      return true;
    };
    for (int kb = 0; kb < min(kFirstStages - 1, kblocks) && ok; ++kb) ok = load(kb);
    for (int kb = 0; kb < kblocks && ok; ++kb) {
      const int s = kb % kFirstStages;
      if (!mbar_wait(&full[s], (uint32_t)(kb / kFirstStages) & 1u, ep.spin_limit)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t a_addr = smem_u32(smem + s * stage_bytes);
      // 64 rows of M: the second column block is the first one again, and its rows are dropped
      const uint64_t da = smem_desc_sw128_mn(a_addr) & ~((uint64_t)0x3FFFu << 16), db = smem_desc_sw128_mn(a_addr + 8192u);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_bf16(tmem, da + 128u * k, db + 128u * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
        mma_commit(&empty[s]);
      }
      __syncwarp();
      if (kb + kFirstStages - 1 < kblocks) ok = load(kb + kFirstStages - 1);
    }
    if (!ok) atomicExch(&failed, 1);
    if (elect_one()) mma_commit(&done);
    if (lane == 0) issued_loads = issued;
  }
  __syncwarp();
  const bool have = mbar_wait(&done, 0, ep.spin_limit);
  if (!have) atomicExch(&failed, 1);
  asm volatile("tcgen05.fence::after_thread_sync;");
  __syncthreads();
  const bool good = !failed;
  if (!good && threadIdx.x == 0) {
    const int issued = issued_loads;
    for (int kb = issued > kFirstStages ? issued - kFirstStages : 0; kb < issued; ++kb)
      mbar_wait(&full[kb % kFirstStages], (uint32_t)(kb / kFirstStages) & 1u, ep.spin_limit);
    if (ep.err) atomicExch(ep.err, 1);
  }
  if (good && warp < 2) {
    const int row = warp * 32 + lane;
    store_tile(ep, tmem + ((uint32_t)(warp * 32) << 16), p.bn, 0, row < p.kp, (size_t)row, false,
               (float*)ep.out + (size_t)blockIdx.x * ep.split_stride);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 4) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

// ------------------------------------------------------------------ input gradient of a stride-2 layer
// dx[iy, ix, c] = the sum, over the taps (ky, kx) that read the pixel, of sum_n dz[oy, ox, n] w[n, (ky, kx, c)]. Pixels of
// one parity class (iy & 1, ix & 1) are read by the same 1, 2, 2 or 4 taps, each at one offset into dz: a tile is 128
// pixels of a class, each tap a product of its own over n (two accumulators in turn), and the storing warps add the
// taps in order in registers. The sums are those of dz W^T written out in FP32 and gathered by col2im, bit for
// bit; that matrix (9 values for each of dz's pixels and channels) was written and read through HBM: batch 16,
// 128 x 256 pixels 32 <- 64 channels 98 + 121 us -> 41, 64 x 128 64 <- 128 49 + 60 -> 23, 32 x 64 128 <- 256 29 + 23
// -> 20. What is left reads and writes dx once (67 MB each at the first size, 21 us) in 128-byte pieces two pixels apart.
struct Dgrad2Params {
  int units, tiles, tiles_x, tiles_y;   // 4 classes x B x tiles of a class and image
  int bw, bh, log2_bw;
  int H, W, C, chunks;                  // dx; chunks of KC channels n
  int stages, n_valid;
  int accumulate;
  int drop_load;                        // test hook, as EpiParams::drop_load
  float* dx;
  int* err;
  unsigned spin_limit;
};

template <int KC, int BN>
__global__ void __launch_bounds__(kConvThreads, 1) k_dgrad2(const __grid_constant__ CUtensorMap tmA,
                                                            const __grid_constant__ CUtensorMap tmB,
                                                            const __grid_constant__ Dgrad2Params p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kConvMaxStages], empty[kConvMaxStages], tfull[2], tempty[2];
  __shared__ uint32_t tmem_base;
  __shared__ int failed, issued_loads;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n0 = (int)blockIdx.y * BN;
  constexpr int STAGE = conv_stage_bytes<KC>(BN);
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], 4);
    }
    failed = 0;
    issued_loads = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(2u * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_base;
  const int per_class = p.units / 4;            // (the class of four taps first)

  if (threadIdx.x == 0) {
    const uint32_t bytes = expected((uint32_t)STAGE, p.drop_load);
    int s = 0, issued = 0;
    uint32_t phase = 1;
    bool ok = true;
    for (int u = (int)blockIdx.x; u < p.units && ok; u += (int)gridDim.x) {
      const int cls = 3 - u / per_class, v = u % per_class, b = v / p.tiles, q = v - b * p.tiles;
      const int ty = q / p.tiles_x, j0 = (q - ty * p.tiles_x) * p.bw, i0 = ty * p.bh;
      const int py = cls >> 1, px = cls & 1;
      for (int a = 0; a <= py && ok; ++a) {
        for (int e = 0; e <= px && ok; ++e) {
          const int ky = py ? 2 * a : 1, kx = px ? 2 * e : 1, dy = py && a == 0, dx = px && e == 0;
          for (int c = 0; c < p.chunks; ++c) {
            if (!mbar_wait(&empty[s], phase, p.spin_limit)) {
              atomicExch(&failed, 1);
              ok = false;
              break;
            }
            uint8_t* sa = smem + s * STAGE;
            mbar_expect_tx(&full[s], bytes);
            tma_load_4d(&tmA, &full[s], sa, c * KC, j0 + dx, i0 + dy, b);
            tma_load_2d(&tmB, &full[s], sa + BM * KC * 2, c * KC, (ky * 3 + kx) * p.C + n0);
            ++issued;
            if (++s == p.stages) {
              s = 0;
              phase ^= 1;
            }
          }
        }
      }
    }
    issued_loads = issued;
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc_bf16(BN);
    int s = 0, n = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int u = (int)blockIdx.x; u < p.units && ok; u += (int)gridDim.x) {
      const int cls = 3 - u / per_class, taps = (1 + (cls >> 1)) * (1 + (cls & 1));
      for (int t = 0; t < taps && ok; ++t, ++n) {
        const int buf = n & 1;
        if (!mbar_wait(&tempty[buf], ((uint32_t)(n >> 1) & 1u) ^ 1u, p.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        for (int c = 0; c < p.chunks; ++c) {
          if (!mbar_wait(&full[s], phase, p.spin_limit)) {
            atomicExch(&failed, 1);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t a_addr = smem_u32(smem + s * STAGE), b_addr = a_addr + BM * KC * 2;
          const uint64_t da = KC == 64 ? smem_desc_sw128(a_addr) : smem_desc_sw64(a_addr);
          const uint64_t db = KC == 64 ? smem_desc_sw128(b_addr) : smem_desc_sw64(b_addr);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < KC / 16; ++k)
              mma_bf16(tmem + (uint32_t)(buf * BN), da + 2u * k, db + 2u * k, idesc, (c > 0 || k > 0) ? 1u : 0u);
            mma_commit(&empty[s]);
            if (c == p.chunks - 1) mma_commit(&tfull[buf]);
          }
          __syncwarp();
          if (++s == p.stages) {
            s = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp >= 2) {
    const int prow = (warp & 3) * 32, m = prow + lane;
    int n = 0;
    bool ok = true;
    for (int u = (int)blockIdx.x; u < p.units && ok; u += (int)gridDim.x) {
      const int cls = 3 - u / per_class, v = u % per_class, b = v / p.tiles, q = v - b * p.tiles;
      const int ty = q / p.tiles_x, tx = q - ty * p.tiles_x, taps = (1 + (cls >> 1)) * (1 + (cls & 1));
      float acc[BN];
#pragma unroll
      for (int j = 0; j < BN; ++j) acc[j] = 0.0f;
      for (int t = 0; t < taps; ++t, ++n) {
        const int buf = n & 1;
        if (!mbar_wait(&tfull[buf], (uint32_t)(n >> 1) & 1u, p.spin_limit)) {
          atomicExch(&failed, 1);
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {
          uint32_t r[32];
          tmem_ld32(tmem + (uint32_t)(buf * BN + c0) + ((uint32_t)prow << 16), r);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[c0 + j] += __uint_as_float(r[j]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[buf]);
      }
      const int x = 2 * (tx * p.bw + (m & (p.bw - 1))) + (cls & 1), y = 2 * (ty * p.bh + (m >> p.log2_bw)) + (cls >> 1);
      if (ok && x < p.W && y < p.H) {
        float* o = p.dx + (((size_t)b * p.H + y) * p.W + x) * p.C + n0;
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {   // (n_valid: a multiple of 8)
          if (p.accumulate) {
            uint32_t e[32];
#pragma unroll
            for (int j = 0; j < 32; j += 8)
              if (n0 + c0 + j < p.n_valid)
                asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(e[j]), "=r"(e[j + 1]), "=r"(e[j + 2]), "=r"(e[j + 3]), "=r"(e[j + 4]), "=r"(e[j + 5]),
                               "=r"(e[j + 6]), "=r"(e[j + 7])
                             : "l"(o + c0 + j));
              else
#pragma unroll
                for (int i = 0; i < 8; ++i) e[j + i] = 0;
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[c0 + j] = __uint_as_float(e[j]) + acc[c0 + j];
          }
#pragma unroll
          for (int j = c0; j < c0 + 32; j += 8)
            if (n0 + j < p.n_valid)
              asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(o + j), "r"(__float_as_uint(acc[j])),
                           "r"(__float_as_uint(acc[j + 1])), "r"(__float_as_uint(acc[j + 2])), "r"(__float_as_uint(acc[j + 3])),
                           "r"(__float_as_uint(acc[j + 4])), "r"(__float_as_uint(acc[j + 5])), "r"(__float_as_uint(acc[j + 6])),
                           "r"(__float_as_uint(acc[j + 7]))
                           : "memory");
        }
      }
      __syncwarp();
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (failed && threadIdx.x == 0) {
    const int issued = issued_loads;
    for (int it = issued > p.stages ? issued - p.stages : 0; it < issued; ++it)
      mbar_wait(&full[it % p.stages], (uint32_t)(it / p.stages) & 1u, p.spin_limit);
    if (p.err) atomicExch(p.err, 1);
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * BN));
}

}  // namespace gemm
}  // namespace vl
