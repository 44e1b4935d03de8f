// cnn.cu - the convolutional gradient preconditioner (no reference
// counterpart): a small stack of 3x3 convolutions (ReLU between layers)
// that maps the FWI gradient and the source illumination to a search
// direction, with training and inference on the GPU.
//
// Activations and gradients are BF16 in channel-group planes: the channel
// count is rounded up to 16 (zeros above the layer's own count) and group g
// of 8 channels is a plane [x][z][8] of the image (pixel p = x * nz + z), so
// element (p, c) sits at ((c / 8) * npix + p) * 8 + c % 8.  A pixel of a
// plane is 16 bytes: eight consecutive pixels of a column are one core matrix
// of the tensor cores' no-swizzle layout (umma.cuh), at any 16-byte offset.
//
// * Convolution (forward, and the input gradient with mirrored taps and
//   transposed weights): implicit GEMM D[pixel][n] = sum over (tap,
//   channel) on tcgen05 (M = 128 pixels, N = 16 or 32 output channels,
//   K = 9 Cs).  A block is 24 (z) x 16 (x) pixels; one tensor copy brings it
//   with its one-pixel border (26 x 18 pixels, every channel group, zero
//   fill outside the image).  An M = 128 tile is 8 (z) x 16 (x): its core
//   matrices are one column apart, so every tap is the same operand at
//   another start address and nothing is copied per tap.  The epilogue
//   fuses the bias and the ReLU (hidden layers write BF16 activations
//   only), or the ReLU derivative of the layer input (input gradient), or
//   writes the FP32 output of the last layer.
// * Weight gradient: dW[tap, ci][co] = sum_p a[p + off(tap)][ci] dz[p][co]
//   on tcgen05 with both operands MN-major (K = the 16 pixels of a column
//   run).  The columns of a 16 x 16 pixel block are stored one after the
//   other, so the rows of one product are the channels of 4 (8) adjacent
//   columns: the three dx taps (and columns that are not used); dz taps are
//   start addresses.  The bias gradient is summed from the staged gradient
//   by the warps that wait for the accumulators.  Each persistent CTA
//   accumulates its pixels in tensor memory and writes one partial sum, and
//   the partials are added in a fixed order (deterministic).
//
// FP32 master weights and Adam state; the BF16 GEMM copies of the weights
// are rewritten in the tensor cores' layout after every update.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/swave.h"
#include "engine.h"
#include "umma.cuh"

using namespace swave;

namespace {

constexpr int kMaxC = 32;                 // channels per layer
constexpr int kTile = 128;                // GEMM M

int r16(int c);
// Stored channels of a tensor: a multiple of 16, so that one tap of a
// layer's input is a whole number of K = 16 steps.
int cstore(int c) { return (c + 15) / 16 * 16; }
int r16(int c) { return (c + 15) / 16 * 16; }

__device__ __forceinline__ unsigned char *align1024(unsigned char *p) {
  const unsigned a = umma_su32(p);
  return p + ((1024u - (a & 1023u)) & 1023u);
}
__device__ __forceinline__ void cnn_expect_tx(unsigned long long *bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(umma_su32(bar)),
               "r"(bytes)
               : "memory");
}
// Tensor copy (global -> shared memory, on an mbarrier) of the box at pixel
// row z and coordinates c1..c3 of the map's other dimensions.  The innermost
// dimension is (z, channel) flattened, so its coordinate 8 z is a multiple of
// 16 bytes for every z.
__device__ __forceinline__ void cnn_tma4(void *dst, const CUtensorMap *map, int z, int c1, int c2,
                                         int c3, unsigned long long *bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(umma_su32(dst)),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(8 * z), "r"(c1), "r"(c2), "r"(c3),
      "r"(umma_su32(bar))
      : "memory");
}
// The kernels of a pass follow one another by programmatic launches: a
// kernel's CTAs start as those of the one before leave, set themselves up
// and wait here before they touch a tensor.  Tensor memory is allocated
// before the successor is let go, so a CTA that holds some and waits never
// stands in the way of one that it waits for.
__device__ __forceinline__ void cnn_chain() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// Instruction descriptor with both operands MN-major (transposed).
__host__ __device__ constexpr uint32_t umma_idesc_bf16_mn(int M, int N) {
  return umma_idesc_bf16(M, N) | (1u << 15) | (1u << 16);
}

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  const __nv_bfloat16 a = __float2bfloat16(lo), b = __float2bfloat16(hi);
  return (unsigned)__bfloat16_as_ushort(a) | ((unsigned)__bfloat16_as_ushort(b) << 16);
}

// ---------------------------------------------------------------------------
// Warp roles of both kernels (192 threads): warps 0-3 read the tensor-memory
// accumulator (lane quadrant = warp) and run the epilogue, warp 4 issues
// the tensor copies into a ring of shared-memory stages, warp 5 issues the
// tensor-core instructions.  Every wait is bounded; a wait that gives up
// sets the error flag and the CTA's abort flag, and every role leaves its
// loop at its next wait.
// ---------------------------------------------------------------------------
constexpr int kEpiWarps = 4, kProducerWarp = 4, kMmaWarp = 5;
constexpr int kWsThreads = 192;

// Bounded wait that also gives up once another role has aborted.
__device__ __forceinline__ bool cnn_wait(unsigned long long *bar, unsigned parity,
                                         volatile int *abort_flag) {
  for (int it = 0; it < (1 << 22); ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(umma_su32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 63) == 63 && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void cnn_arrive(unsigned long long *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma_su32(bar)) : "memory");
}
__device__ __forceinline__ void cnn_bar_init(unsigned long long *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(umma_su32(bar)), "r"(count)
               : "memory");
}

// ---------------------------------------------------------------------------
// Implicit-GEMM 3x3 (or 3x3x3) convolution.
//   D[p][n] = sum_{tap, c} in[p + s * off(tap)][c] * W[n][tap * Cs + c]
// with s = +1 (forward) or -1 (input gradient) and zero padding outside
// the image.  W: NP x kp BF16 in the tensor cores' K-major layout.  One
// ring stage holds one plane (a dy in 3D) of a block with its border: a
// single tensor copy of kBZ x kBX pixels, every channel group, column pitch
// kPitch bytes.  The M = 128 tile m (rows z0 + 8 m .. + 7 of the 16 columns)
// of tap (dz, dx) starts at column dx + 1, row 8 m + dz + 1: core matrices
// kPitch apart along M and one plane apart along K.  Two sets of kMT
// accumulators in tensor memory let the products of the next block run
// while the epilogue reads the last one.
// Bound by the shared-memory reads of A (4 KB per product of 128 x NP x 16:
// N is only 32).  Three copies per 32 x 4 pixel tile, one per dz, moved 4.5x
// the pixels through L2 and took 26 / 30 us (forward / input gradient, 32
// channels, 301 x 901 pixels, cold L2); this takes 17 / 18 us, and 36 us
// instead of about 95 on 601 x 1801 pixels.
// ---------------------------------------------------------------------------
enum { kFwdHidden = 0, kFwdLast = 1, kBwd = 2 };
constexpr int kMaxRing = 16;
constexpr int kMT = 3;                             // M tiles of a block
constexpr int kCZ = 8 * kMT, kCX = 16;             // pixels of a block
constexpr int kBZ = kCZ + 2, kBX = kCX + 2;        // with the border
constexpr int kPitch = kBZ * 16;                   // bytes of a column
constexpr int kPlane = kBX * kPitch;               // bytes of a channel group

struct ConvArgs {
  int Cs;                        // stored input channels (multiple of 16)
  int nz, nx, ny;
  int taps;                      // 9 (2D) or 27 (3D)
  int kp;                        // GEMM K: taps Cs
  int ntiles, tiles_z, tiles_x;
  int mirror;
  int ring;                      // shared-memory stages (<= kMaxRing)
  const __nv_bfloat16 *W;
  const float *bias;             // forward: nout biases
  int nout;                      // output channels
  int cs_out;                    // stored output channels (BF16 outputs)
  float *out32;                  // kFwdLast: [p][nout]
  __nv_bfloat16 *out16;          // kFwdHidden, kBwd: cs_out / 8 channel-group planes
  const __nv_bfloat16 *mask;     // kBwd: layer input activations (cs_out / 8 planes)
  int *err;
};

__host__ __device__ inline size_t conv_wbytes(int NP, int kp) { return ((size_t)NP * kp * 2 + 1023) / 1024 * 1024; }
size_t conv_smem_bytes(int NP, int kp, int Cs, int ring) {
  return 1024 + conv_wbytes(NP, kp) + (size_t)ring * (Cs / 8) * kPlane;
}

template <int NP, int MODE>
__global__ void __launch_bounds__(kWsThreads, 2)
    k_conv_tma(const __grid_constant__ CUtensorMap amap, const ConvArgs A) {
  extern __shared__ unsigned char cnn_smem[];
  __shared__ __align__(8) unsigned long long full[kMaxRing], empty[kMaxRing];
  __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2];
  __shared__ float sbias[kMaxC];
  __shared__ unsigned tmem_base;
  __shared__ volatile int abort_flag;
  __shared__ volatile int mma_stages;             // stages the MMA warp has consumed
  constexpr unsigned kCols = NP == 32 ? 256 : 128;   // 2 x kMT accumulators of NP columns
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nst = A.taps / 9;                     // ring stages (planes) per block
  const size_t sbytes = (size_t)(A.Cs / 8) * kPlane;
  unsigned char *base = align1024(cnn_smem);
  unsigned char *sW = base;
  unsigned char *ring = base + conv_wbytes(NP, A.kp);
  if (tid == 0) {
    for (int q = 0; q < A.ring; ++q) {
      cnn_bar_init(&full[q], 1);
      cnn_bar_init(&empty[q], 1);
    }
    for (int q = 0; q < 2; ++q) {
      cnn_bar_init(&acc_full[q], 1);
      cnn_bar_init(&acc_empty[q], kEpiWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    mma_stages = 0;
  }
  if (tid < kMaxC) sbias[tid] = MODE != kBwd && tid < A.nout ? A.bias[tid] : 0.f;
  if (warp == kMmaWarp) umma_alloc(&tmem_base, kCols);
#pragma unroll 6
  for (int q = tid; q < NP * A.kp / 8; q += kWsThreads)
    reinterpret_cast<uint4 *>(sW)[q] = reinterpret_cast<const uint4 *>(A.W)[q];
  umma_fence_smem();
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  cnn_chain();
  const unsigned tmem = tmem_base;
  const int first = blockIdx.x, stride = gridDim.x;
  const int nmine = first < A.ntiles ? (A.ntiles - 1 - first) / stride + 1 : 0;
  const int sgn = A.mirror ? -1 : 1;
  if (warp == kProducerWarp) {
    if (lane == 0) {
      int q = 0;
      bool ok = true;
      for (int i = 0; i < nmine && ok; ++i) {
        const int t = first + i * stride;
        const int z0 = (t % A.tiles_z) * kCZ, x0 = ((t / A.tiles_z) % A.tiles_x) * kCX;
        const int y0 = t / (A.tiles_z * A.tiles_x);
        for (int k = 0; k < nst; ++k, ++q) {
          const int slot = q % A.ring;
          if (q >= A.ring && !(ok = cnn_wait(&empty[slot], ((q / A.ring) - 1) & 1, &abort_flag)))
            break;
          cnn_expect_tx(&full[slot], (unsigned)sbytes);
          cnn_tma4(ring + (size_t)slot * sbytes, &amap, z0 - 1, x0 - 1,
                   y0 + (nst == 3 ? sgn * (k - 1) : 0), 0, &full[slot]);
        }
      }
      if (!ok) {
        abort_flag = 1;
        atomicOr(A.err, 1);
      }
      // After a give-up, copies the MMA warp did not consume complete
      // before the CTA leaves (at most one ring of them).
      if (abort_flag)
        for (int r = max(mma_stages, q - A.ring); r < q; ++r)
          umma_mbar_wait(&full[r % A.ring], (r / A.ring) & 1);
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(kTile, NP);
      const int nh = A.Cs / 16;
      const uint64_t bdesc = umma_smem_desc(umma_su32(sW), (NP / 8) * 128, 128);
      int q = 0, committed = -1;
      bool ok = true;
      for (int i = 0; i < nmine && ok; ++i) {
        const int acc = i & 1;
        if (i >= 2 && !(ok = cnn_wait(&acc_empty[acc], ((i >> 1) - 1) & 1, &abort_flag))) break;
        umma_fence_after();
        const unsigned d = tmem + acc * kMT * NP;
        for (int k = 0; k < nst; ++k, ++q) {
          const int slot = q % A.ring;
          if (!(ok = cnn_wait(&full[slot], (q / A.ring) & 1, &abort_flag))) break;
          mma_stages = q + 1;
          umma_fence_after();
          // Descriptors differ in their start address alone (16-byte units):
          // one addition per product, the issuing thread's own instructions
          // would otherwise take longer than the products.
          const uint64_t ad0 =
              umma_smem_desc(umma_su32(ring + (size_t)slot * sbytes), kPlane, kPitch);
          uint64_t ad[3];   // by s dz + 1
          ad[0] = ad0 + (1 - sgn);
          ad[1] = ad0 + 1;
          ad[2] = ad0 + (1 + sgn);
          const uint64_t bd0 = bdesc + (uint64_t)(9 * k * nh) * (2 * NP);
          for (int dz = 0; dz < 3; ++dz)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
              uint64_t a = ad[dz] + (uint64_t)((sgn * (dx - 1) + 1) * (kPitch / 16));
              uint64_t b = bd0 + (uint64_t)((3 * dx + dz) * nh) * (2 * NP);
              for (int h = 0; h < nh; ++h, a += 2 * kPlane / 16, b += 2 * NP) {
                const bool more = k > 0 || dz > 0 || dx > 0 || h > 0;
#pragma unroll
                for (int m = 0; m < kMT; ++m) umma_bf16(d + m * NP, a + m * 8, b, idesc, more);
              }
            }
          umma_commit(&empty[slot]);
        }
        if (!ok) break;
        umma_commit(&acc_full[acc]);
        committed = i;
      }
      if (!ok) {
        abort_flag = 1;
        atomicOr(A.err, 1);
      }
      if (committed >= 0) umma_mbar_wait(&acc_full[committed & 1], (committed >> 1) & 1);
    }
  } else {
    // Epilogue: thread = accumulator lane = row of an M tile, pixel
    // (z0 + 8 m + row % 8, x0 + row / 8).
    const size_t npix = (size_t)A.nz * A.nx * A.ny;
    for (int i = 0; i < nmine; ++i) {
      const int acc = i & 1;
      const int t = first + i * stride;
      const int z0 = (t % A.tiles_z) * kCZ + (tid & 7);
      const int x = ((t / A.tiles_z) % A.tiles_x) * kCX + (tid >> 3);
      const int y = t / (A.tiles_z * A.tiles_x);
      // The ReLU masks are loaded before the products are waited for.
      uint4 mk[MODE == kBwd ? kMT : 1][MODE == kBwd ? NP / 8 : 1];
      if (MODE == kBwd) {
#pragma unroll
        for (int m = 0; m < kMT; ++m)
#pragma unroll
          for (int g = 0; g < NP / 8; ++g)
            mk[m][g] = z0 + 8 * m < A.nz && x < A.nx && 8 * g < A.cs_out
                           ? *reinterpret_cast<const uint4 *>(
                                 A.mask + ((size_t)g * npix + ((size_t)y * A.nx + x) * A.nz + z0 +
                                           8 * m) * 8)
                           : make_uint4(0u, 0u, 0u, 0u);
      }
      bool ok = cnn_wait(&acc_full[acc], (i >> 1) & 1, &abort_flag);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) {
          abort_flag = 1;
          atomicOr(A.err, 1);
        }
        break;
      }
      umma_fence_after();
      const unsigned ta = tmem + ((unsigned)(warp * 32) << 16) + acc * kMT * NP;
#pragma unroll
      for (int m = 0; m < kMT; ++m) {
        float accv[NP];
        umma_ld16(ta + m * NP, accv);
        if (NP == 32) umma_ld16(ta + m * NP + 16, accv + 16);
        if (m == kMT - 1) {
          umma_fence_before();
          __syncwarp();
          if (lane == 0) cnn_arrive(&acc_empty[acc]);
        }
        const int z = z0 + 8 * m;
        if (z >= A.nz || x >= A.nx) continue;
        const size_t p = ((size_t)y * A.nx + x) * A.nz + z;
        if (MODE == kFwdLast) {
#pragma unroll
          for (int n = 0; n < NP; ++n)
            if (n < A.nout) A.out32[p * A.nout + n] = accv[n] + sbias[n];
        } else {
#pragma unroll
          for (int c0 = 0; c0 < NP; c0 += 8) {
            if (c0 >= A.cs_out) break;
            float v[8];
            if (MODE == kFwdHidden) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                v[j] = c0 + j < A.nout ? fmaxf(accv[c0 + j] + sbias[c0 + j], 0.f) : 0.f;
            } else {
              const uint4 mq = mk[MODE == kBwd ? m : 0][MODE == kBwd ? c0 / 8 : 0];
              const unsigned mw[4] = {mq.x, mq.y, mq.z, mq.w};
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const unsigned short bits = (unsigned short)(mw[j >> 1] >> (16 * (j & 1)));
                const bool pos = __bfloat162float(__ushort_as_bfloat16(bits)) > 0.f;
                v[j] = (c0 + j < A.nout && pos) ? accv[c0 + j] : 0.f;
              }
            }
            *reinterpret_cast<uint4 *>(A.out16 + ((size_t)(c0 / 8) * npix + p) * 8) =
                make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                           pack_bf16(v[6], v[7]));
          }
        }
      }
    }
  }
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  if (warp == kMmaWarp) umma_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------------------
// Weight and bias gradient of one layer on the tensor cores.
//   dW[tap, ci][co] = sum_p a[p + off(tap)][ci] dz[p][co]
// A ring stage holds a 16 x 16 pixel block of dz ([group][column][16 z]) and
// one plane (dy) of the activations around it, column by column: 18 columns
// of kWZ rows (z0 - 1 ..; 18 are used, 20 keep what follows 128-byte aligned),
// each [group][row].  Eight-channel groups are then kWPitch bytes apart over
// the groups of a column and on into the next column, so the 128 rows of a
// product for output column c are the channels of columns c, c + 1, ...: row
// dxi * Csi + ci belongs to dx = dxi - 1 (rows of dxi > 2 are not used).  K
// is the column's 16 pixels, dz a start address.  Accumulators: one per (dy,
// dz).
// Bound by the shared-memory reads of A, 4 KB per product; one copy of each
// tap's own 32 x 4 pixel patch took 41 us (32 channels, 301 x 901 pixels, cold
// L2), this takes 21 us.
// ---------------------------------------------------------------------------
struct WgradArgs {
  int Csi, Cin, Cso, Cout;
  int nz, nx, ny, taps, ntiles, tiles_z, tiles_x;
  int ring;                      // shared-memory stages (<= kMaxRing)
  float *part;                   // [cta][tap or bias][kMaxC][kMaxC]
  int *err;
};
constexpr int kWB = 16;                      // pixels of a block along each axis
constexpr int kWZ = 20, kWPitch = kWZ * 16;  // staged rows of a column, bytes per group
constexpr int kWDz = kWB * kWB * 16;         // bytes of a channel group of dz

// Columns of a stage: the rows of the last product reach this far (the ones
// past the 18 copied hold stale data, which only unused rows read).
__host__ __device__ inline int wgrad_cols(int Csi) { return kWB - 1 + kTile / Csi; }
__host__ __device__ inline size_t wgrad_stage(int Csi, int Cso) {
  return (size_t)wgrad_cols(Csi) * (Csi / 8) * kWPitch + (size_t)(Cso / 8) * kWDz;
}

template <int NPO>
__global__ void __launch_bounds__(kWsThreads, 1)
    k_wgrad_umma(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap dmap,
                 const WgradArgs A) {
  extern __shared__ unsigned char cnn_smem[];
  __shared__ __align__(8) unsigned long long full[kMaxRing], empty[kMaxRing], done;
  __shared__ unsigned tmem_base;
  __shared__ volatile int abort_flag;
  __shared__ volatile int mma_stages;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ndy = A.taps / 9;
  const unsigned kCols = ndy == 1 ? 128 : 512;    // 3 ndy accumulators of NPO columns
  const size_t abytes = (size_t)wgrad_cols(A.Csi) * (A.Csi / 8) * kWPitch;
  const size_t sbytes = wgrad_stage(A.Csi, A.Cso);
  const int colb = (A.Csi / 8) * kWPitch;         // bytes of a column
  unsigned char *ring = align1024(cnn_smem);
  if (tid == 0) {
    for (int q = 0; q < A.ring; ++q) {
      cnn_bar_init(&full[q], 1);
      cnn_bar_init(&empty[q], 1 + kEpiWarps);
    }
    cnn_bar_init(&done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_flag = 0;
    mma_stages = 0;
  }
  if (warp == kMmaWarp) umma_alloc(&tmem_base, kCols);
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  cnn_chain();
  const unsigned tmem = tmem_base;
  const int first = blockIdx.x, stride = gridDim.x;
  const int nmine = first < A.ntiles ? (A.ntiles - 1 - first) / stride + 1 : 0;
  if (warp == kProducerWarp) {
    if (lane == 0) {
      int q = 0;
      bool ok = true;
      for (int i = 0; i < nmine && ok; ++i) {
        const int t = first + i * stride;
        const int z0 = (t % A.tiles_z) * kWB, x0 = ((t / A.tiles_z) % A.tiles_x) * kWB;
        const int y0 = t / (A.tiles_z * A.tiles_x);
        for (int k = 0; k < ndy; ++k, ++q) {
          const int slot = q % A.ring;
          if (q >= A.ring && !(ok = cnn_wait(&empty[slot], ((q / A.ring) - 1) & 1, &abort_flag)))
            break;
          unsigned char *dst = ring + (size_t)slot * sbytes;
          cnn_expect_tx(&full[slot], (unsigned)((kWB + 2) * colb + (A.Cso / 8) * kWDz));
          cnn_tma4(dst + abytes, &dmap, z0, x0, y0, 0, &full[slot]);
          cnn_tma4(dst, &amap, z0 - 1, 0, x0 - 1, y0 + (ndy == 3 ? k - 1 : 0), &full[slot]);
        }
      }
      if (!ok) {
        abort_flag = 1;
        atomicOr(A.err, 1);
      }
      if (abort_flag)
        for (int r = max(mma_stages, q - A.ring); r < q; ++r)
          umma_mbar_wait(&full[r % A.ring], (r / A.ring) & 1);
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16_mn(kTile, NPO);
      int q = 0;
      bool ok = true, any = false;
      for (int i = 0; i < nmine && ok; ++i)
        for (int k = 0; k < ndy; ++k, ++q) {
          const int slot = q % A.ring;
          if (!(ok = cnn_wait(&full[slot], (q / A.ring) & 1, &abort_flag))) break;
          mma_stages = q + 1;
          umma_fence_after();
          const unsigned sa = umma_su32(ring + (size_t)slot * sbytes);
          // MN-major, no swizzle: the leading byte offset is the step between
          // the core matrices of 8 pixels along K (128 bytes), the stride
          // byte offset the step between 8-channel groups along M / N.
          uint64_t ad = umma_smem_desc(sa, 128, kWPitch);
          uint64_t bd = umma_smem_desc(sa + (unsigned)abytes, 128, kWDz);
          const unsigned d = tmem + 3 * k * NPO;
#pragma unroll 4
          for (int c = 0; c < kWB; ++c, ad += colb / 16, bd += kWB) {
            const bool more = i > 0 || c > 0;
#pragma unroll
            for (int dz = 0; dz < 3; ++dz) umma_bf16(d + dz * NPO, ad + dz, bd, idesc, more);
          }
          umma_commit(&empty[slot]);
          any = true;
        }
      if (!ok) {
        abort_flag = 1;
        atomicOr(A.err, 1);
      }
      if (any) umma_commit(&done);
      else cnn_arrive(&done);
    }
  } else if (nmine > 0) {
    // While the products run: warp g sums channel group g of dz (once per
    // block) over its pixels.
    float bs[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    bool ok = true;
    for (int q = 0; q < nmine * ndy && ok; ++q) {
      const int slot = q % A.ring;
      ok = __all_sync(0xffffffffu, cnn_wait(&full[slot], (q / A.ring) & 1, &abort_flag));
      if (ok && q % ndy == 0 && warp < A.Cso / 8) {
        const uint4 *g = reinterpret_cast<const uint4 *>(ring + (size_t)slot * sbytes + abytes +
                                                         (size_t)warp * kWDz);
#pragma unroll
        for (int r = 0; r < kWB * kWB / 32; ++r) {
          const uint4 v = g[lane + 32 * r];
          const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 8; ++j)
            bs[j] += __uint_as_float(j & 1 ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
        }
      }
      __syncwarp();
      if (lane == 0) cnn_arrive(&empty[slot]);
    }
    // Epilogue: thread = accumulator lane = row dxi * Csi + ci.
    ok = ok && cnn_wait(&done, 0, &abort_flag) && !abort_flag;
    ok = __all_sync(0xffffffffu, ok);
    umma_fence_after();
    if (ok) {
      float *P = A.part + (size_t)blockIdx.x * (A.taps + 1) * kMaxC * kMaxC;
      const int dxi = tid / A.Csi, ci = tid % A.Csi;
      for (int j = 0; j < 3 * ndy; ++j) {
        float accv[NPO];
        const unsigned ta = tmem + ((unsigned)(warp * 32) << 16) + j * NPO;
        umma_ld16(ta, accv);
        if (NPO == 32) umma_ld16(ta + 16, accv + 16);
        const int tap = 9 * (j / 3) + 3 * dxi + j % 3;
        if (dxi < 3 && ci < A.Cin) {
#pragma unroll
          for (int co = 0; co < NPO; ++co)
            if (co < A.Cout) P[(size_t)tap * kMaxC * kMaxC + co * kMaxC + ci] = accv[co];
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        for (int o = 16; o > 0; o >>= 1) bs[j] += __shfl_xor_sync(0xffffffffu, bs[j], o);
        if (lane == 0 && 8 * warp + j < A.Cout)
          P[(size_t)A.taps * kMaxC * kMaxC + (8 * warp + j) * kMaxC] = bs[j];
      }
    } else if (lane == 0) {
      abort_flag = 1;
      atomicOr(A.err, 1);
    }
  }
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  if (warp == kMmaWarp) {
    // A give-up left products in flight: wait (bounded) for the last commit.
    if (abort_flag && lane == 0) umma_mbar_wait(&done, 0);
    __syncwarp();
    umma_dealloc(tmem, kCols);
  }
}

// Sums the per-CTA partials of every layer into the gradient buffer (FP32,
// per layer [co][tap][ci] then bias[co]) - added to what it holds.  Block
// (tap, co, layer), tap `taps` being the bias: 16 threads per input channel
// take every sixteenth partial, then the 16 sums are added in order.
constexpr int kSumW = 16, kMaxLayers = 16;
struct SumArgs {
  const float *part[kMaxLayers];
  int nchunk, taps;
  int Cin[kMaxLayers], Cout[kMaxLayers];
  size_t off[kMaxLayers];
  float *g;
};
__host__ __device__ inline size_t part_floats(int taps) {
  return (size_t)(taps + 1) * kMaxC * kMaxC;   // of one CTA
}
__global__ void __launch_bounds__(kSumW * kMaxC) k_wgrad_sum(const SumArgs A) {
  __shared__ float sh[kSumW][kMaxC];
  const int tap = blockIdx.x, co = blockIdx.y, l = blockIdx.z;
  const int ci = threadIdx.x % kMaxC, w = threadIdx.x / kMaxC;
  const int Cin = A.Cin[l], Cout = A.Cout[l], taps = A.taps;
  cnn_chain();
  if (co >= Cout) return;
  const bool use = tap == taps ? ci == 0 : ci < Cin;
  const float *P = A.part[l] + (size_t)tap * kMaxC * kMaxC + co * kMaxC + ci;
  float s = 0.f;
#pragma unroll 10
  for (int c = w; c < A.nchunk; c += kSumW) s += use ? P[c * part_floats(taps)] : 0.f;
  sh[w][ci] = s;
  __syncthreads();
  if (w != 0 || !use) return;
  for (int q = 1; q < kSumW; ++q) s += sh[q][ci];
  float *gw = A.g + A.off[l];
  if (tap == taps) gw[(size_t)Cout * taps * Cin + co] += s;
  else gw[((size_t)co * taps + tap) * Cin + ci] += s;
}

// Planar FP32 channels (c, p) -> BF16 channel-group planes; block row y is
// group y, a thread packs the 8 channels of one pixel.
__global__ void k_pack_input(const float *__restrict__ in, int C, int npix,
                             __nv_bfloat16 *__restrict__ out) {
  const int g = blockIdx.y;
  cnn_chain();
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 8 * g + j < C ? in[(size_t)(8 * g + j) * npix + p] : 0.f;
    *reinterpret_cast<uint4 *>(out + ((size_t)g * npix + p) * 8) =
        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]),
                   pack_bf16(v[6], v[7]));
  }
}

// Mean-square loss of a one-channel output: the output gradient
// (out - target) / npix as BF16 in channel 0 of a 16-channel tensor (two
// planes, zero elsewhere), and per-block FP64 partial sums of
// (out - target)^2.  Few blocks: their FP64 tree sums cost more than the
// pixels (1024 blocks: 9.3 us for 301 x 901).
__global__ void k_loss(const float *__restrict__ out, const float *__restrict__ tgt, int npix,
                       __nv_bfloat16 *__restrict__ db, double *__restrict__ part) {
  __shared__ double red[8];
  double s = 0.0;
  cnn_chain();
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
    const float e = out[p] - tgt[p];
    s += (double)e * (double)e;
    *reinterpret_cast<uint4 *>(db + (size_t)p * 8) =
        make_uint4(pack_bf16(e / (float)npix, 0.f), 0u, 0u, 0u);
    *reinterpret_cast<uint4 *>(db + ((size_t)npix + p) * 8) = make_uint4(0u, 0u, 0u, 0u);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) s += red[w];
    part[blockIdx.x] = s;
  }
}

// Adam on the FP32 master weights.
__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2, float gscale) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const float gg = g[q] * gscale;
  const float mm = b1 * m[q] + (1.f - b1) * gg;
  const float vv = b2 * v[q] + (1.f - b2) * gg * gg;
  m[q] = mm;
  v[q] = vv;
  w[q] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

// BF16 GEMM copies of one layer's weights in the tensor cores' K-major
// layout: forward NPo x KPf, element (co, tap * Csi + ci); input gradient
// NPi x KPb, element (ci, tap * Cso + co).  Zero outside the layer.
__global__ void k_weights_bf16(const float *__restrict__ w, int Cout, int Cin, int Csi, int Cso,
                               int taps, int NPo, int KPf, int NPi, int KPb,
                               __nv_bfloat16 *__restrict__ wf, __nv_bfloat16 *__restrict__ wb) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < NPo * KPf; q += gridDim.x * blockDim.x) {
    const int n = q / KPf, k = q % KPf;
    const int tap = k / Csi, ci = k % Csi;
    float v = 0.f;
    if (n < Cout && tap < taps && ci < Cin) v = w[((size_t)n * taps + tap) * Cin + ci];
    wf[umma_off(n, k, NPo) >> 1] = __float2bfloat16(v);
  }
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < NPi * KPb; q += gridDim.x * blockDim.x) {
    const int n = q / KPb, k = q % KPb;
    const int tap = k / Cso, co = k % Cso;
    float v = 0.f;
    if (n < Cin && tap < taps && co < Cout) v = w[((size_t)co * taps + tap) * Cin + n];
    wb[umma_off(n, k, NPi) >> 1] = __float2bfloat16(v);
  }
}

int nblk(long long n) { return (int)std::min<long long>(4096, (n + 255) / 256); }

// BF16 tensor map over Cs / 8 channel-group planes: dimensions (8 nz: z
// and the 8 channels flattened, nx, ny, Cs / 8), box rows x cols pixels of
// one plane, every group; zero fill outside.  by_column: the groups come
// before the columns (dimensions 8 nz, Cs / 8, nx, ny), so that a box lands
// column by column.
bool encode_act_map(CUtensorMap *m, const __nv_bfloat16 *base, int Cs, int nz, int nx, int ny,
                    int rows, int cols, bool by_column = false) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t col = (cuuint64_t)nz * 16, plane = col * nx, grp = plane * ny,
                   G = (cuuint64_t)Cs / 8;
  const cuuint64_t d0[4] = {(cuuint64_t)nz * 8, (cuuint64_t)nx, (cuuint64_t)ny, G},
                   d1[4] = {(cuuint64_t)nz * 8, G, (cuuint64_t)nx, (cuuint64_t)ny};
  const cuuint64_t s0[3] = {col, plane, grp}, s1[3] = {grp, col, plane};
  const cuuint32_t b0[4] = {8 * (cuuint32_t)rows, (cuuint32_t)cols, 1, (cuuint32_t)G},
                   b1[4] = {8 * (cuuint32_t)rows, (cuuint32_t)G, (cuuint32_t)cols, 1};
  const cuuint64_t *dims = by_column ? d1 : d0, *strides = by_column ? s1 : s0;
  const cuuint32_t *box = by_column ? b1 : b0;
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16 *>(base), dims,
             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int num_sms(int dev) {
  int n = 0;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
    n = 1;
  return n;
}

// A kernel of the chain (cnn_chain).
template <typename... P, typename... Q>
cudaError_t launch_chained(void (*k)(P...), dim3 grid, int block, size_t smem, cudaStream_t s,
                           const Q &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}

template <class K>
cudaError_t launch_big(K kernel, int grid, size_t smem, cudaStream_t s, const CUtensorMap &m0,
                       const ConvArgs &a) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  return launch_chained(kernel, dim3(grid), kWsThreads, smem, s, m0, a);
}

// One convolution: input tensor (Cs channels) -> MODE's outputs.
cudaError_t launch_conv(int dev, int mode, int NP, const __nv_bfloat16 *in, int Cs, int nz, int nx,
                        int ny, int taps, ConvArgs a, cudaStream_t s) {
  CUtensorMap m;
  if (!encode_act_map(&m, in, Cs, nz, nx, ny, kBZ, kBX)) return cudaErrorInvalidValue;
  a.Cs = Cs;
  a.nz = nz;
  a.nx = nx;
  a.ny = ny;
  a.taps = taps;
  a.kp = r16(taps * Cs);
  a.tiles_z = (nz + kCZ - 1) / kCZ;
  a.tiles_x = (nx + kCX - 1) / kCX;
  a.ntiles = a.tiles_z * a.tiles_x * ny;
  // Two CTAs per SM where at least two stages fit beside the weights, else
  // one with a longer ring.
  const size_t stage = (size_t)(Cs / 8) * kPlane, w = 1024 + conv_wbytes(NP, a.kp);
  const int per_sm = w + 2 * stage <= 111u * 1024u ? 2 : 1;
  a.ring = (int)std::min<size_t>(kMaxRing, ((per_sm == 2 ? 111u : 224u) * 1024u - w) / stage);
  const size_t smem = conv_smem_bytes(NP, a.kp, Cs, a.ring);
  const int grid = std::min(a.ntiles, num_sms(dev) * per_sm);
  if (NP == 16) {
    if (mode == kFwdHidden) return launch_big(k_conv_tma<16, kFwdHidden>, grid, smem, s, m, a);
    if (mode == kFwdLast) return launch_big(k_conv_tma<16, kFwdLast>, grid, smem, s, m, a);
    return launch_big(k_conv_tma<16, kBwd>, grid, smem, s, m, a);
  }
  if (mode == kFwdHidden) return launch_big(k_conv_tma<32, kFwdHidden>, grid, smem, s, m, a);
  if (mode == kFwdLast) return launch_big(k_conv_tma<32, kFwdLast>, grid, smem, s, m, a);
  return launch_big(k_conv_tma<32, kBwd>, grid, smem, s, m, a);
}

// Weight-gradient partials of one layer; returns the number of partials.
cudaError_t launch_wgrad(int dev, const __nv_bfloat16 *a, int Cin, const __nv_bfloat16 *dz,
                         int Cout, int nz, int nx, int ny, int taps, float *part, int *err,
                         cudaStream_t s, int *nchunk) {
  WgradArgs w;
  w.Csi = cstore(Cin);
  w.Cin = Cin;
  w.Cso = cstore(Cout);
  w.Cout = Cout;
  w.nz = nz;
  w.nx = nx;
  w.ny = ny;
  w.taps = taps;
  w.tiles_z = (nz + kWB - 1) / kWB;
  w.tiles_x = (nx + kWB - 1) / kWB;
  w.ntiles = w.tiles_z * w.tiles_x * ny;
  const size_t stage = wgrad_stage(w.Csi, w.Cso);
  w.ring = (int)std::min<size_t>(kMaxRing, 200u * 1024u / stage);
  w.part = part;
  w.err = err;
  CUtensorMap ma, md;
  if (!encode_act_map(&ma, a, w.Csi, nz, nx, ny, kWZ, kWB + 2, true) ||
      !encode_act_map(&md, dz, w.Cso, nz, nx, ny, kWB, kWB))
    return cudaErrorInvalidValue;
  const int NPO = r16(Cout);
  const size_t smem = 1024 + w.ring * stage;
  const int grid = std::min(w.ntiles, num_sms(dev));
  *nchunk = grid;
  cudaError_t e;
  if (NPO == 16) {
    e = cudaFuncSetAttribute(k_wgrad_umma<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    return launch_chained(k_wgrad_umma<16>, dim3(grid), kWsThreads, smem, s, ma, md, w);
  } else {
    e = cudaFuncSetAttribute(k_wgrad_umma<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
    if (e != cudaSuccess) return e;
    return launch_chained(k_wgrad_umma<32>, dim3(grid), kWsThreads, smem, s, ma, md, w);
  }
}

}  // namespace

struct sw_cnn {
  sw_ctx *ctx = nullptr;
  int nl = 0;
  int taps = 9;                        // 9: 3 x 3 kernels on images, 27: 3 x 3 x 3 on volumes
  std::vector<int> ch;                 // nl + 1 channel counts
  std::vector<size_t> woff;            // offset of layer l in the packed weights
  size_t nw = 0;                       // packed FP32 weights (w then b per layer)
  float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  std::vector<__nv_bfloat16 *> wf, wb; // BF16 GEMM copies per layer
  int step = 0;
  // Per-image buffers (grow-only).
  size_t cap = 0;
  std::vector<__nv_bfloat16 *> a;      // layer inputs, cstore(ch[l]) / 8 channel-group planes
  __nv_bfloat16 *dz[2] = {nullptr, nullptr};   // gradients, up to cstore(max ch) / 8 planes
  float *out32 = nullptr, *in32 = nullptr, *tgt = nullptr, *part = nullptr;
  double *lpart = nullptr;
  int *err = nullptr;
};

namespace {

int cnn_fail(sw_cnn *n, cudaError_t e, const char *what) {
  return cuda_fail(n ? n->ctx : nullptr, e, what);
}

void free_images(sw_cnn *n) {
  for (auto p : n->a) cudaFree(p);
  n->a.clear();
  cudaFree(n->dz[0]); cudaFree(n->dz[1]);
  cudaFree(n->out32); cudaFree(n->in32); cudaFree(n->tgt); cudaFree(n->part); cudaFree(n->lpart);
  n->dz[0] = n->dz[1] = nullptr;
  n->out32 = n->in32 = n->tgt = n->part = nullptr;
  n->lpart = nullptr;
  n->cap = 0;
}

int ensure_images(sw_cnn *n, size_t npix) {
  if (npix <= n->cap) return SW_OK;
  free_images(n);
  auto ck = [&](cudaError_t e) { return e == cudaSuccess; };
  bool ok = true;
  int cmax = 8;
  for (int c : n->ch) cmax = std::max(cmax, cstore(c));
  n->a.assign(n->nl, nullptr);
  for (int l = 0; l < n->nl && ok; ++l)
    ok = ck(dev_malloc(n->ctx, &n->a[l], npix * cstore(n->ch[l]) * sizeof(__nv_bfloat16)));
  ok = ok && ck(dev_malloc(n->ctx, &n->dz[0], npix * cmax * sizeof(__nv_bfloat16))) &&
       ck(dev_malloc(n->ctx, &n->dz[1], npix * cmax * sizeof(__nv_bfloat16))) &&
       ck(dev_malloc(n->ctx, &n->out32, npix * sizeof(float))) &&
       ck(dev_malloc(n->ctx, &n->in32, npix * n->ch[0] * sizeof(float))) &&
       ck(dev_malloc(n->ctx, &n->tgt, npix * sizeof(float))) &&
       ck(dev_malloc(n->ctx, &n->part,
                     (size_t)n->nl * num_sms(n->ctx->device) * part_floats(n->taps) *
                         sizeof(float))) &&
       ck(dev_malloc(n->ctx, &n->lpart, 1024 * sizeof(double)));
  if (!ok) {
    cudaGetLastError();
    free_images(n);
    return fail(n->ctx, SW_OOM_ADMISSION, "cnn image buffers");
  }
  n->cap = npix;
  return SW_OK;
}

// Runs one tensor-core kernel launch; with profiling on, brackets it with
// CUDA events on the context stream and adds its time, algorithmic bytes
// and FLOPs to the context's counters.
template <class L>
cudaError_t timed_launch(sw_cnn *n, uint64_t bytes, uint64_t flops, L launch) {
  sw_ctx *c = n->ctx;
  c->stats.launches_total++;
  if (!c->profiling) return launch();
  cudaEvent_t e0, e1;
  cudaError_t e = cudaEventCreate(&e0);
  if (e != cudaSuccess) return e;
  if ((e = cudaEventCreate(&e1)) != cudaSuccess) {
    cudaEventDestroy(e0);
    return e;
  }
  cudaEventRecord(e0, c->stream);
  e = launch();
  cudaEventRecord(e1, c->stream);
  if (e == cudaSuccess) e = cudaEventSynchronize(e1);
  float ms = 0.f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (e == cudaSuccess) {
    c->stats.cnn_conv_ms += ms;
    c->stats.cnn_conv_timed++;
    c->stats.cnn_conv_bytes += bytes;
    c->stats.cnn_conv_flops += flops;
  }
  return e;
}

int refresh_bf16(sw_cnn *n) {
  cudaStream_t s = n->ctx->stream;
  for (int l = 0; l < n->nl; ++l) {
    const int Cin = n->ch[l], Cout = n->ch[l + 1];
    const int T = n->taps;
    k_weights_bf16<<<16, 256, 0, s>>>(n->w + n->woff[l], Cout, Cin, cstore(Cin), cstore(Cout), T,
                                      r16(Cout), r16(T * cstore(Cin)), r16(Cin), r16(T * cstore(Cout)),
                                      n->wf[l], n->wb[l]);
    n->ctx->stats.launches_total++;
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SW_OK : cnn_fail(n, e, "cnn weights");
}

// Forward pass of one image (volume) already packed into n->a[0]; output
// in n->out32.
int forward(sw_cnn *n, int nz, int nx, int ny) {
  cudaStream_t s = n->ctx->stream;
  const int dev = n->ctx->device;
  const int T = n->taps;
  cudaError_t e;
  for (int l = 0; l < n->nl; ++l) {
    const int Cin = n->ch[l], Cout = n->ch[l + 1];
    const bool last = l + 1 == n->nl;
    ConvArgs a{};
    a.mirror = 0;
    a.W = n->wf[l];
    a.bias = n->w + n->woff[l] + (size_t)Cout * T * Cin;
    a.nout = Cout;
    a.cs_out = cstore(Cout);
    a.out32 = last ? n->out32 : nullptr;
    a.out16 = last ? nullptr : n->a[l + 1];
    a.err = n->err;
    const uint64_t np = (uint64_t)nz * nx * ny;
    const uint64_t bytes = np * cstore(Cin) * 2 + (last ? np * Cout * 4 : np * cstore(Cout) * 2);
    if ((e = timed_launch(n, bytes, 2 * np * Cout * T * Cin, [&] {
           return launch_conv(dev, last ? kFwdLast : kFwdHidden, r16(Cout), n->a[l], cstore(Cin), nz,
                              nx, ny, T, a, s);
         })) != cudaSuccess)
      return cnn_fail(n, e, "cnn conv");
  }
  return SW_OK;
}

int check_err(sw_cnn *n) {
  int h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, n->err, sizeof(int), cudaMemcpyDeviceToHost, n->ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(n->ctx->stream);
  if (e != cudaSuccess) return cnn_fail(n, e, "cnn");
  if (h) {
    cudaMemsetAsync(n->err, 0, sizeof(int), n->ctx->stream);
    return fail(n->ctx, SW_TIMEOUT, "cnn: a tensor-core or tensor-copy wait gave up");
  }
  return SW_OK;
}

// Sum over the batch of the weight gradient into n->g (zeroed first); the
// batch-mean loss into *loss.
int gradient(sw_cnn *n, int nbatch, int nz, int nx, int ny, const float *in, const float *target,
             double *loss) {
  cudaStream_t s = n->ctx->stream;
  const int dev = n->ctx->device;
  const int T = n->taps;
  const size_t npix = (size_t)nz * nx * ny;
  int st = ensure_images(n, npix);
  if (st) return st;
  cudaError_t e;
  if ((e = cudaMemsetAsync(n->g, 0, n->nw * 4, s)) != cudaSuccess) return cnn_fail(n, e, "cnn");
  const int lblocks = (int)std::min<size_t>(304, (npix + 255) / 256);
  double lsum = 0.0;
  std::vector<double> hp(lblocks);
  for (int ib = 0; ib < nbatch; ++ib) {
    const float *xin = in + (size_t)ib * npix * n->ch[0];
    const float *tin = target + (size_t)ib * npix;
    if ((e = cudaMemcpyAsync(n->in32, xin, npix * n->ch[0] * 4, cudaMemcpyHostToDevice, s)) !=
            cudaSuccess ||
        (e = cudaMemcpyAsync(n->tgt, tin, npix * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return cnn_fail(n, e, "cnn batch");
    k_pack_input<<<dim3(nblk(npix), cstore(n->ch[0]) / 8), 256, 0, s>>>(n->in32, n->ch[0], (int)npix,
                                                                        n->a[0]);
    n->ctx->stats.launches_total++;
    if ((st = forward(n, nz, nx, ny))) return st;
    // d loss / d output (one channel), FP64 loss partials.
    int cur = 0;
    if ((e = launch_chained(k_loss, dim3(lblocks), 256, 0, s, n->out32, n->tgt, (int)npix,
                            n->dz[cur], n->lpart)) != cudaSuccess)
      return cnn_fail(n, e, "cnn loss");
    n->ctx->stats.launches_total++;
    SumArgs sum;
    sum.taps = T;
    sum.g = n->g;
    for (int l = n->nl - 1; l >= 0; --l) {
      const int Cin = n->ch[l], Cout = n->ch[l + 1];
      float *part = n->part + (size_t)l * num_sms(dev) * part_floats(T);
      sum.part[l] = part;
      sum.Cin[l] = Cin;
      sum.Cout[l] = Cout;
      sum.off[l] = n->woff[l];
      const uint64_t np = (uint64_t)npix;
      if ((e = timed_launch(n, np * (cstore(Cin) + cstore(Cout)) * 2, 2 * np * T * Cin * Cout, [&] {
             return launch_wgrad(dev, n->a[l], Cin, n->dz[cur], Cout, nz, nx, ny, T, part, n->err,
                                 s, &sum.nchunk);   // the same for every layer
           })) != cudaSuccess)
        return cnn_fail(n, e, "cnn wgrad");
      if (l == 0) break;
      // Input gradient: mirrored taps, transposed weights, then ReLU' of
      // the layer input, into the other gradient buffer.
      ConvArgs a{};
      a.mirror = 1;
      a.W = n->wb[l];
      a.bias = nullptr;
      a.nout = Cin;
      a.cs_out = cstore(Cin);
      a.out16 = n->dz[cur ^ 1];
      a.mask = n->a[l];
      a.err = n->err;
      if ((e = timed_launch(n, np * (cstore(Cout) + 2 * cstore(Cin)) * 2, 2 * np * Cin * T * Cout, [&] {
             return launch_conv(dev, kBwd, r16(Cin), n->dz[cur], cstore(Cout), nz, nx, ny, T, a, s);
           })) != cudaSuccess)
        return cnn_fail(n, e, "cnn dgrad");
      cur ^= 1;
    }
    if ((e = launch_chained(k_wgrad_sum, dim3(T + 1, kMaxC, n->nl), kSumW * kMaxC, 0, s, sum)) !=
        cudaSuccess)
      return cnn_fail(n, e, "cnn backward");
    n->ctx->stats.launches_total++;
    if ((e = cudaMemcpyAsync(hp.data(), n->lpart, lblocks * sizeof(double),
                             cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
      return cnn_fail(n, e, "cnn loss");
    double ls = 0.0;
    for (int b = 0; b < lblocks; ++b) ls += hp[b];
    lsum += ls / (2.0 * (double)npix);
  }
  if (loss) *loss = lsum / nbatch;
  return SW_OK;
}

int create_net(sw_ctx *c, int nlayers, const int *channels, uint64_t seed, int taps,
               sw_cnn **out) {
  if (!c || !channels || !out || nlayers < 1 || nlayers > 16) return SW_BAD_PARAM;
  *out = nullptr;
  for (int l = 0; l <= nlayers; ++l)
    if (channels[l] < 1 || channels[l] > kMaxC)
      return fail(c, SW_BAD_PARAM, "cnn channels must be 1..32");
  cudaSetDevice(c->device);
  sw_cnn *n = new sw_cnn();
  n->ctx = c;
  n->nl = nlayers;
  n->taps = taps;
  n->ch.assign(channels, channels + nlayers + 1);
  for (int l = 0; l < nlayers; ++l) {
    n->woff.push_back(n->nw);
    n->nw += (size_t)n->ch[l + 1] * taps * n->ch[l] + n->ch[l + 1];
  }
  // He initialisation, zero biases.
  std::vector<float> h(n->nw, 0.f);
  std::mt19937_64 rng(seed);
  for (int l = 0; l < nlayers; ++l) {
    const int Cin = n->ch[l], Cout = n->ch[l + 1];
    std::normal_distribution<float> nd(0.f, std::sqrt(2.f / ((float)taps * Cin)));
    for (int q = 0; q < Cout * taps * Cin; ++q) h[n->woff[l] + q] = nd(rng);
  }
  auto ck = [](cudaError_t e) { return e == cudaSuccess; };
  bool ok = ck(dev_malloc(c, &n->w, n->nw * 4)) && ck(dev_malloc(c, &n->g, n->nw * 4)) &&
            ck(dev_malloc(c, &n->m, n->nw * 4)) && ck(dev_malloc(c, &n->v, n->nw * 4)) &&
            ck(dev_malloc(c, &n->err, sizeof(int)));
  n->wf.assign(nlayers, nullptr);
  n->wb.assign(nlayers, nullptr);
  for (int l = 0; l < nlayers && ok; ++l) {
    const int Cin = n->ch[l], Cout = n->ch[l + 1];
    ok = ck(dev_malloc(c, &n->wf[l], (size_t)r16(Cout) * r16(taps * cstore(Cin)) * 2)) &&
         ck(dev_malloc(c, &n->wb[l], (size_t)r16(Cin) * r16(taps * cstore(Cout)) * 2));
  }
  ok = ok && ck(cudaMemcpy(n->w, h.data(), n->nw * 4, cudaMemcpyHostToDevice)) &&
       ck(cudaMemset(n->m, 0, n->nw * 4)) && ck(cudaMemset(n->v, 0, n->nw * 4)) &&
       ck(cudaMemset(n->err, 0, sizeof(int)));
  if (!ok || refresh_bf16(n) != SW_OK) {
    cudaGetLastError();
    sw_cnn_destroy(n);
    return fail(c, SW_CUDA_ERR, "cnn create");
  }
  *out = n;
  return SW_OK;
}

// Shared body of the image (ny = 1, 3 x 3 network) and volume (3 x 3 x 3
// network) entry points.
int cnn_forward(sw_cnn *n, int nz, int nx, int ny, const float *in, float *out) {
  if (n->ch[n->nl] != 1) return fail(n->ctx, SW_BAD_PARAM, "cnn output must have one channel");
  cudaSetDevice(n->ctx->device);
  cudaStream_t s = n->ctx->stream;
  const size_t npix = (size_t)nz * nx * ny;
  int st = ensure_images(n, npix);
  if (st) return st;
  cudaError_t e;
  if ((e = cudaMemcpyAsync(n->in32, in, npix * n->ch[0] * 4, cudaMemcpyHostToDevice, s)) !=
      cudaSuccess)
    return cnn_fail(n, e, "cnn input");
  k_pack_input<<<dim3(nblk(npix), cstore(n->ch[0]) / 8), 256, 0, s>>>(n->in32, n->ch[0], (int)npix,
                                                                        n->a[0]);
  n->ctx->stats.launches_total++;
  if ((st = forward(n, nz, nx, ny))) return st;
  TouchWhileBusy touch(n->ctx);
  touch.add(out, npix * 4);
  populate_touch(n->ctx);
  if ((e = cudaMemcpyAsync(out, n->out32, npix * 4, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cnn_fail(n, e, "cnn output");
  return check_err(n);
}

int cnn_gradient(sw_cnn *n, int nbatch, int nz, int nx, int ny, const float *in,
                 const float *target, float *grad, double *loss) {
  if (n->ch[n->nl] != 1) return fail(n->ctx, SW_BAD_PARAM, "cnn output must have one channel");
  cudaSetDevice(n->ctx->device);
  int st = gradient(n, nbatch, nz, nx, ny, in, target, loss);
  if (st) return st;
  if ((st = check_err(n))) return st;
  std::vector<float> h(n->nw);
  if (cudaMemcpy(h.data(), n->g, n->nw * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
    return SW_CUDA_ERR;
  for (size_t q = 0; q < n->nw; ++q) grad[q] = h[q] / (float)nbatch;
  return SW_OK;
}

int cnn_train_step(sw_cnn *n, int nbatch, int nz, int nx, int ny, const float *in,
                   const float *target, float lr, double *loss) {
  if (n->ch[n->nl] != 1) return fail(n->ctx, SW_BAD_PARAM, "cnn output must have one channel");
  cudaSetDevice(n->ctx->device);
  cudaStream_t s = n->ctx->stream;
  int st = gradient(n, nbatch, nz, nx, ny, in, target, loss);
  if (st) return st;
  // Adam (b1 0.9, b2 0.999, eps 1e-8) on the batch-mean gradient.
  n->step += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - std::pow(b1, (float)n->step), c2 = 1.f - std::pow(b2, (float)n->step);
  k_adam<<<(int)((n->nw + 255) / 256), 256, 0, s>>>(n->w, n->g, n->m, n->v, (int)n->nw, lr, b1, b2,
                                                    1e-8f, c1, c2, 1.f / (float)nbatch);
  n->ctx->stats.launches_total++;
  if ((st = refresh_bf16(n))) return st;
  return check_err(n);
}

}  // namespace

extern "C" {

int sw_cnn_create(sw_ctx *c, int nlayers, const int *channels, uint64_t seed, sw_cnn **out) {
  return create_net(c, nlayers, channels, seed, 9, out);
}

int sw_cnn_create3d(sw_ctx *c, int nlayers, const int *channels, uint64_t seed, sw_cnn **out) {
  return create_net(c, nlayers, channels, seed, 27, out);
}

int sw_cnn_destroy(sw_cnn *n) {
  if (!n) return SW_OK;
  cudaSetDevice(n->ctx->device);
  cudaStreamSynchronize(n->ctx->stream);
  free_images(n);
  cudaFree(n->w); cudaFree(n->g); cudaFree(n->m); cudaFree(n->v); cudaFree(n->err);
  for (auto p : n->wf) cudaFree(p);
  for (auto p : n->wb) cudaFree(p);
  delete n;
  return SW_OK;
}

int sw_cnn_num_weights(const sw_cnn *n) { return n ? (int)n->nw : 0; }

int sw_cnn_get_weights(const sw_cnn *n, float *w) {
  if (!n || !w) return SW_BAD_PARAM;
  cudaSetDevice(n->ctx->device);
  if (cudaMemcpy(w, n->w, n->nw * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return SW_CUDA_ERR;
  return SW_OK;
}

int sw_cnn_set_weights(sw_cnn *n, const float *w) {
  if (!n || !w) return SW_BAD_PARAM;
  cudaSetDevice(n->ctx->device);
  if (cudaMemcpy(n->w, w, n->nw * 4, cudaMemcpyHostToDevice) != cudaSuccess) return SW_CUDA_ERR;
  const int st = refresh_bf16(n);
  if (st) return st;
  return cudaStreamSynchronize(n->ctx->stream) == cudaSuccess ? SW_OK : SW_CUDA_ERR;
}

int sw_cnn_forward(sw_cnn *n, int nz, int nx, const float *in, float *out) {
  if (!n || !in || !out || nz < 1 || nx < 1) return SW_BAD_PARAM;
  if (n->taps != 9) return fail(n->ctx, SW_BAD_PARAM, "a 3x3x3 network takes volumes");
  return cnn_forward(n, nz, nx, 1, in, out);
}

int sw_cnn_gradient(sw_cnn *n, int nbatch, int nz, int nx, const float *in, const float *target,
                    float *grad, double *loss) {
  if (!n || !in || !target || !grad || nbatch < 1 || nz < 1 || nx < 1) return SW_BAD_PARAM;
  if (n->taps != 9) return fail(n->ctx, SW_BAD_PARAM, "a 3x3x3 network takes volumes");
  return cnn_gradient(n, nbatch, nz, nx, 1, in, target, grad, loss);
}

int sw_cnn_train_step(sw_cnn *n, int nbatch, int nz, int nx, const float *in,
                      const float *target, float lr, double *loss) {
  if (!n || !in || !target || nbatch < 1 || nz < 1 || nx < 1) return SW_BAD_PARAM;
  if (n->taps != 9) return fail(n->ctx, SW_BAD_PARAM, "a 3x3x3 network takes volumes");
  return cnn_train_step(n, nbatch, nz, nx, 1, in, target, lr, loss);
}

int sw_cnn_forward3d(sw_cnn *n, int nz, int nx, int ny, const float *in, float *out) {
  if (!n || !in || !out || nz < 1 || nx < 1 || ny < 1) return SW_BAD_PARAM;
  if (n->taps != 27) return fail(n->ctx, SW_BAD_PARAM, "a 3x3 network takes images");
  return cnn_forward(n, nz, nx, ny, in, out);
}

int sw_cnn_gradient3d(sw_cnn *n, int nbatch, int nz, int nx, int ny, const float *in,
                      const float *target, float *grad, double *loss) {
  if (!n || !in || !target || !grad || nbatch < 1 || nz < 1 || nx < 1 || ny < 1)
    return SW_BAD_PARAM;
  if (n->taps != 27) return fail(n->ctx, SW_BAD_PARAM, "a 3x3 network takes images");
  return cnn_gradient(n, nbatch, nz, nx, ny, in, target, grad, loss);
}

int sw_cnn_train_step3d(sw_cnn *n, int nbatch, int nz, int nx, int ny, const float *in,
                        const float *target, float lr, double *loss) {
  if (!n || !in || !target || nbatch < 1 || nz < 1 || nx < 1 || ny < 1) return SW_BAD_PARAM;
  if (n->taps != 27) return fail(n->ctx, SW_BAD_PARAM, "a 3x3 network takes images");
  return cnn_train_step(n, nbatch, nz, nx, ny, in, target, lr, loss);
}

}  // extern "C"
