// vh_nn.cu -- kernels of the learned depth denoiser: a 4-layer 3x3 convolutional net (input 4 channels -> 32
// -> 32 -> 32 -> 1, ReLU between layers, residual output), BF16 weights and activations, FP32 accumulation.
//
// The two 32 -> 32 layers carry ~95 % of the arithmetic and run on the 5th-generation tensor cores
// (tcgen05.mma, kind::f16 with BF16 operands, FP32 accumulator in tensor memory) as an implicit GEMM: each
// output row of a 128-pixel strip is M = 128 pixels x N = 32 output channels, K = 9 taps x 32 input channels,
// issued as 18 MMAs of m128n32k16 into a TMEM accumulator (32 columns; two accumulators).
// Input rows (130 pixels each, 1-pixel halo) are loaded by TMA (4 tensor-map boxes of {8 channels, 130
// pixels} per row, zero fill outside the image) into a ring of row slots in the canonical no-swizzle K-major
// layout: [channel group of 8][pixel][8 channels], 16 bytes per pixel per group (each group's plane padded to
// 2,176 bytes for the TMA's 128-byte destination alignment).  The A operand of tap (dy, dx) is the slot of
// input row y - 1 + dy starting dx pixels further -- a descriptor start address 16 bytes * dx higher; no
// im2col copy.  A CTA streams blocks of output rows of one strip, loading each input row once.  Weights are
// staged once per CTA as [tap][k-step][channel group][output channel][8 channels].  The epilogue reads the
// accumulator with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 = pixels 32w..32w+31), adds the bias and
// applies ReLU, or, for the input gradient, multiplies by the ReLU mask of the layer's input, and stores BF16.
//
// The input gradient of a 32 -> 32 layer is the same convolution with the weights flipped in space and
// transposed in channels, so the backward pass reuses the kernel.  The weight gradient of a 32 -> 32 layer (a
// reduction over pixels) is a second tensor-core kernel, wgrad32_tc_kernel.  The 4-channel input layer, the
// 1-channel output layer, their weight gradients and Adam run on the CUDA cores in FP32, the input channels always
// computed from the depth where they are used.
//
// Safety: the descriptors address only staged bytes: an A operand reads at most 8,608 bytes into its 8,704-byte
// slot (pixels dx .. dx + 127 of each plane), the B operand exactly kBBytes, followed by a margin; the layout is
// checked bit-for-bit against a float64 convolution.  Every mbarrier wait gives up after about a second, sets
// the error word and the kernel still waits (bounded) for its loads and MMAs before freeing tensor memory.
#include <cuda.h>  // CUtensorMap and the tensor-map encoder's types (resolved at run time, no link dependency)
#include <cuda_bf16.h>

#include <cstdint>
#include <cstdlib>

#include "vh_nn.h"

namespace vh {
namespace nn {
namespace {

constexpr int kTile = 128;                 // output pixels per CTA tile (MMA M)
constexpr int kC = 32;                     // channels of the hidden layers (MMA N, and K per tap)
constexpr int kRowPix = kTile + 2;         // staged pixels per input row
constexpr int kGroups = kC / 8;            // channel groups of 8 (16 bytes of BF16)
constexpr int kPlaneData = kRowPix * 16;   // bytes of one channel group of one staged row: one TMA box
constexpr int kPlane = 2176;               // the plane padded to a multiple of 128 (TMA destination alignment);
                                           // the A operand's LBO
constexpr int kRowBytes = kGroups * kPlane;  // one ring slot: 8,704 bytes (8,320 written by a row's 4 boxes)
constexpr int kBBlock = 2 * kC * 16;       // one (tap, k-step) B operand: 2 groups x 32 rows x 16 B = 1,024
constexpr int kBBytes = 18 * kBBlock;      // 18,432
constexpr int kBPad = kBBytes + 1024;
// warps 0-3: epilogue (warp w owns TMEM lanes 32w..32w+31); warp 4: TMA producer; warp 5: TMEM owner, MMA issuer
constexpr int kEpilogueWarps = 4;
constexpr int kThreads = 32 * (kEpilogueWarps + 2);
constexpr int kAccs = 2;  // accumulators in tensor memory (32 columns each)
static_assert(kPlaneData <= kPlane && kPlane % 128 == 0, "TMA destinations 128-byte aligned");
// A wait gives up once kWaitNs of global time have passed since its first poll (kMaxPolls bounds the polls as
// well, should the timer not advance).  Legitimate waits in this kernel last microseconds.
constexpr uint64_t kWaitNs = 1000000000ull;
constexpr uint32_t kMaxPolls = 1u << 28;
constexpr unsigned int kErrorBit = 8u;  // the volume error word's timeout bit

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// tcgen05 shared-memory matrix descriptor, no swizzle (canonical K-major core-matrix layout):
// start address, leading-dimension byte offset (between core matrices along K), stride-dimension byte offset
// (between core matrices along M/N), descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1u) << 46;
  return d;
}

// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, N = 32, M = 128
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(kC >> 3) << 17) |
                            (static_cast<uint32_t>(kTile >> 4) << 24);

__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate));
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
  uint64_t start = 0;
  for (uint32_t i = 0; i < kMaxPolls; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase));
    if (done) return true;
    if ((i & 255u) == 0u) {
      const uint64_t now = global_ns();
      if (i == 0u) {
        start = now;
      } else if (now - start > kWaitNs) {
        return false;
      }
    }
  }
  return false;
}

// The load gate of vh_nn_conv32_gated: true once *gate is nonzero, false if it stays zero for kWaitNs.
__device__ __forceinline__ bool gate_wait(const unsigned int* gate) {
  const uint64_t start = global_ns();
  for (uint32_t i = 0; i < kMaxPolls; ++i) {
    if (*reinterpret_cast<const volatile unsigned int*>(gate) != 0u) return true;
    if (global_ns() - start > kWaitNs) return false;
    __nanosleep(1000);
  }
  return false;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

// A CTA owns blocks of kRows output rows of one 128-pixel strip and streams the block's kRows + 2 input rows
// once each through a ring of kSlots row slots, so an output row costs one new input row (4 TMA boxes) instead
// of three; the three taps' rows are three resident slots.

constexpr uint32_t kRowTxBytes = kGroups * kPlaneData;
static_assert(kRowBytes % 128 == 0, "ring slots keep the TMA destinations 128-byte aligned");

// loads input row y of image img (pixels x0-1 .. x0+128, 4 channel-group boxes, zero fill outside the image)
__device__ __forceinline__ void load_row(const CUtensorMap* map, uint32_t slot_base, uint32_t bar, int img, int y,
                                         int x0) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(kRowTxBytes) : "memory");
  const uint64_t m = reinterpret_cast<uint64_t>(map);
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];\n" ::"r"(slot_base + g * kPlane),
        "l"(m), "r"(8 * g), "r"(x0 - 1), "r"(y), "r"(img), "r"(bar)
        : "memory");
  }
}

// the 18 MMAs of one output row: tap row dy reads the slot r0 / r1 / r2 (input rows y - 1, y, y + 1)
__device__ __forceinline__ void issue_row(uint32_t r0, uint32_t r1, uint32_t r2, uint32_t b_base, uint32_t tmem) {
  int k = 0;
  for (int dy = 0; dy < 3; ++dy) {
    const uint32_t rb = dy == 0 ? r0 : (dy == 1 ? r1 : r2);
    for (int dx = 0; dx < 3; ++dx) {
      for (int ks = 0; ks < 2; ++ks, ++k) {
        const uint64_t a = smem_desc(rb + (2 * ks) * kPlane + dx * 16, kPlane, 128);
        const uint64_t b = smem_desc(b_base + k * kBBlock, kC * 16, 128);
        mma(tmem, a, b, k > 0 ? 1u : 0u);
      }
    }
  }
}

// the epilogue's per-warp transpose buffer: 32 pixels x 64 bytes
constexpr int kEpiStage = 32 * kC * 2;

template <int kSlots>
constexpr int ring_smem_bytes() {
  return 128 + kSlots * kRowBytes + kBPad + kEpilogueWarps * kEpiStage + 8 * (2 * kSlots + 2 * kAccs) + 16;
}

// The epilogue moves a warp's 32 pixels x 64 bytes between registers (lane l: pixel l) and global memory
// through its shared-memory buffer, so that every global access instruction covers 512 contiguous bytes
// (lane l: 16-byte chunk u * 32 + l of the warp's 2 KB), not 32 half sectors.  Chunk q of pixel p sits at
// position 4p + (q ^ ((p >> 1) & 3)): the XOR spreads the lanes of each access phase over distinct banks.
__device__ __forceinline__ int epi_pos(int p, int q) { return 4 * p + (q ^ ((p >> 1) & 3)); }

// One 32 -> 32 3x3 convolution over a batch of images (NHWC BF16, zero padding), tcgen05 implicit GEMM.
// mode kForward: out = relu?(conv(in) + bias); mode kGrad: out = conv(in) * (mask > 0) (mask = the layer
// input's activations; the input gradient of the previous layer's ReLU).
//
// Warp-specialised, handing off through mbarriers only:
//   producer (warp 4, one lane): waits empty[s] (the MMAs that read the slot's previous row completed), then
//     TMA-loads input row q into slot s = q mod kSlots, completing full[s] by transaction bytes;
//   MMA issuer (warp 5, one lane): for each output row waits full[s] of the rows it adds and acc_empty[a] (the
//     epilogue has read accumulator a = row mod kAccs), issues the 18 MMAs and commits them to the top row's
//     empty[s] (that row is not read again) and to acc_full[a]; a block's last two rows are released after
//     its last output row;
//   epilogue (warps 0-3): waits acc_full[a], reads its 32 TMEM lanes, releases the accumulator (acc_empty[a],
//     one arrival per warp) and applies bias / ReLU or the gradient mask and stores BF16.
// Phase j of a barrier completes at its j-th use, so the waits use parity (q / kSlots) & 1 or (row / kAccs) & 1
// and the releases of an earlier use the parity before.  A ring of at least 3 slots cannot deadlock: the row
// an output row still needs to load was released by an earlier output row.  Every wait gives up after about
// a second: that role stops, the error word gets the timeout bit, and the roles waiting on it
// give up in turn; before tensor memory is freed, the loads and MMA groups still in flight are waited for
// (bounded).
template <int kSlots, int kRows>
__global__ void __launch_bounds__(kThreads, 1) conv32_tc_kernel(const __grid_constant__ CUtensorMap in_map,
                                                                  const __nv_bfloat16* __restrict__ wpack,
                                                                  const float* __restrict__ bias,
                                                                  const __nv_bfloat16* __restrict__ mask,
                                                                  __nv_bfloat16* __restrict__ out, int batch,
                                                                  int width, int height, int mode, int relu,
                                                                  const unsigned int* __restrict__ gate,
                                                                  unsigned int* __restrict__ error) {
  static_assert(kSlots >= 3, "an output row needs three resident input rows");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);  // TMA destinations: 128 B
  unsigned char* sB = smem + kSlots * kRowBytes;
  uint4* sEpi = reinterpret_cast<uint4*>(sB + kBPad);  // kEpilogueWarps x kEpiStage
  uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kBPad + kEpilogueWarps * kEpiStage);  // full[S], empty[S],
                                                                                         // acc_full[A], acc_empty[A]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kSlots + 2 * kAccs);
  uint32_t* consumed = tmem_slot + 1;  // rows whose loads the MMA issuer has waited for (teardown)
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  for (int i = tid; i < kBBytes / 16; i += kThreads) {
    reinterpret_cast<uint4*>(sB)[i] = reinterpret_cast<const uint4*>(wpack)[i];
  }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the weights, for the MMAs' async reads
  if (warp == kEpilogueWarps + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"(32 * kAccs));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  if (tid == 0) {
    for (int i = 0; i < 2 * kSlots + kAccs; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bars[i])));
    }
    for (int i = 0; i < kAccs; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&bars[2 * kSlots + kAccs + i])),
                   "r"(kEpilogueWarps));
    }
    *consumed = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  const uint32_t tmem = *tmem_slot;
  const uint32_t ring0 = smem_u32(smem), b_base = smem_u32(sB);
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kSlots]);
  const uint32_t accf0 = smem_u32(&bars[2 * kSlots]), acce0 = smem_u32(&bars[2 * kSlots + kAccs]);
  auto slot_addr = [&](uint32_t q) { return ring0 + (q % kSlots) * static_cast<uint32_t>(kRowBytes); };

  // work item t = blockIdx.x + k gridDim.x: strip xt, row block rb, image img (32-bit: checked by the launcher)
  const uint32_t tiles_x = static_cast<uint32_t>((width + kTile - 1) / kTile);
  const uint32_t blocks_y = static_cast<uint32_t>((height + kRows - 1) / kRows);
  const uint32_t nitems = static_cast<uint32_t>(batch) * blocks_y * tiles_x;
  const uint32_t stride = gridDim.x;
  const int my_items = blockIdx.x < nitems ? static_cast<int>((nitems - 1u - blockIdx.x) / stride + 1u) : 0;
  auto item = [&](int k, int& img, int& y0, int& x0, int& rows) {
    const uint32_t t = blockIdx.x + static_cast<uint32_t>(k) * stride;
    const uint32_t rest = t / tiles_x;
    x0 = static_cast<int>(t - rest * tiles_x) * kTile;
    const uint32_t im = rest / blocks_y;
    y0 = static_cast<int>(rest - im * blocks_y) * kRows;
    img = static_cast<int>(im);
    rows = min(kRows, height - y0);
  };
  bool ok = true;
  uint32_t loaded = 0;  // producer: rows loaded
  uint32_t issued = 0;  // MMA issuer: output rows issued

  if (warp == kEpilogueWarps) {
    if (lane == 0) {  // producer
      if (gate != nullptr && my_items > 0 && !gate_wait(gate)) ok = false;  // nothing loaded, nothing in flight
      for (int k = 0; k < my_items && ok; ++k) {
        int img, y0, x0, rows;
        item(k, img, y0, x0, rows);
        for (int i = 0; i < rows + 2; ++i) {
          const uint32_t q = loaded;
          if (q >= kSlots && !mbar_wait(empty0 + 8 * (q % kSlots), (q / kSlots - 1) & 1u)) {
            ok = false;
            break;
          }
          load_row(&in_map, slot_addr(q), full0 + 8 * (q % kSlots), img, y0 - 1 + i, x0);
          loaded = q + 1;
        }
      }
    }
  } else if (warp == kEpilogueWarps + 1) {
    if (lane == 0) {  // MMA issuer
      uint32_t q = 0;  // first row of the current block
      for (int k = 0; k < my_items && ok; ++k) {
        int img, y0, x0, rows;
        item(k, img, y0, x0, rows);
        for (int r = 0; r < rows && ok; ++r) {
          for (uint32_t w = (r == 0 ? q : q + r + 2); w <= q + r + 2; ++w) {
            if (!mbar_wait(full0 + 8 * (w % kSlots), (w / kSlots) & 1u)) {
              ok = false;
              break;
            }
            *reinterpret_cast<volatile uint32_t*>(consumed) = w + 1;
          }
          if (!ok) break;
          const uint32_t a = issued % kAccs;
          if (issued >= kAccs && !mbar_wait(acce0 + 8 * a, (issued / kAccs - 1) & 1u)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n");
          issue_row(slot_addr(q + r), slot_addr(q + r + 1), slot_addr(q + r + 2), b_base, tmem + 32u * a);
          commit(empty0 + 8 * ((q + r) % kSlots));
          commit(accf0 + 8 * a);
          issued += 1;
        }
        if (!ok) break;
        commit(empty0 + 8 * ((q + rows) % kSlots));
        commit(empty0 + 8 * ((q + rows + 1) % kSlots));
        q += rows + 2;
      }
    }
  } else {  // epilogue: warp w, lane l = output pixel 32w + l of the row
    float bv[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) bv[c] = (mode == kForward && bias) ? __ldg(&bias[c]) : 0.0f;
    uint32_t j = 0;
    for (int k = 0; k < my_items && ok; ++k) {
      int img, y0, x0, rows;
      item(k, img, y0, x0, rows);
      for (int r = 0; r < rows; ++r, ++j) {
        const uint32_t a = j % kAccs;
        const bool got = mbar_wait(accf0 + 8 * a, (j / kAccs) & 1u);
        if (!__all_sync(0xffffffffu, got)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        float acc[32];
        tmem_ld32(tmem + 32u * a + (static_cast<uint32_t>(warp * 32) << 16), acc);
        asm volatile("tcgen05.fence::before_thread_sync;\n");
        __syncwarp();
        if (lane == 0) arrive(acce0 + 8 * a);
        // the warp's 32 pixels start at pixel xw of row y0 + r; chunk u * 32 + lane belongs to pixel
        // xw + 8u + lane / 4, which must lie inside the image
        uint4* buf = sEpi + warp * (kEpiStage / 16);
        const int xw = x0 + warp * 32;
        const size_t row0 = ((static_cast<size_t>(img) * height + (y0 + r)) * width + xw) * kC;
        __align__(16) __nv_bfloat162 res[16];
        if (mode == kForward) {
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            float v0 = acc[2 * c] + bv[2 * c], v1 = acc[2 * c + 1] + bv[2 * c + 1];
            if (relu) {
              v0 = fmaxf(v0, 0.0f);
              v1 = fmaxf(v1, 0.0f);
            }
            res[c] = __floats2bfloat162_rn(v0, v1);
          }
        } else {
          // the gradient mask, read coalesced and transposed to lane = pixel through the buffer
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int p = 8 * u + (lane >> 2), q = lane & 3;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (xw + p < width) v = *reinterpret_cast<const uint4*>(mask + row0 + static_cast<size_t>(p) * kC + 8 * q);
            buf[epi_pos(p, q)] = v;
          }
          __syncwarp();
          __align__(16) __nv_bfloat162 m[16];
#pragma unroll
          for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(m)[q] = buf[epi_pos(lane, q)];
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const float2 mf = __bfloat1622float2(m[c]);
            res[c] = __floats2bfloat162_rn(mf.x > 0.0f ? acc[2 * c] : 0.0f, mf.y > 0.0f ? acc[2 * c + 1] : 0.0f);
          }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) buf[epi_pos(lane, q)] = reinterpret_cast<const uint4*>(res)[q];
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int p = 8 * u + (lane >> 2), q = lane & 3;
          if (xw + p < width) {
            *reinterpret_cast<uint4*>(out + row0 + static_cast<size_t>(p) * kC + 8 * q) = buf[epi_pos(p, q)];
          }
        }
        __syncwarp();  // the buffer is rewritten for the next row
      }
    }
  }
  if (!ok && lane == 0) atomicOr(error, kErrorBit);
  __syncthreads();
  // in-flight work after a timeout (the waits return at once when nothing is pending)
  if (warp == kEpilogueWarps && lane == 0) {
    for (uint32_t w = *consumed; w < loaded; ++w) mbar_wait(full0 + 8 * (w % kSlots), (w / kSlots) & 1u);
  }
  if (warp == kEpilogueWarps + 1 && lane == 0 && issued > 0) {
    mbar_wait(accf0 + 8 * ((issued - 1) % kAccs), ((issued - 1) / kAccs) & 1u);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  if (warp == kEpilogueWarps + 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(32 * kAccs));
  }
}

// cuTensorMapEncodeTiled, resolved through the runtime's driver entry point (no link dependency on libcuda)
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

cudaError_t encode_input_map(const __nv_bfloat16* in, int batch, int width, int height, CUtensorMap* map) {
  static EncodeTiledFn encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qr = cudaDriverEntryPointSymbolNotFound;
    const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &qr);
    if (e != cudaSuccess) return e;
    if (qr != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  if (reinterpret_cast<uintptr_t>(in) % 16 != 0) return cudaErrorInvalidValue;
  // NHWC BF16: dims innermost first {channel, x, y, image}; byte strides of x, y, image
  const cuuint64_t dims[4] = {static_cast<cuuint64_t>(kC), static_cast<cuuint64_t>(width),
                              static_cast<cuuint64_t>(height), static_cast<cuuint64_t>(batch)};
  const cuuint64_t strides[3] = {static_cast<cuuint64_t>(kC) * 2, static_cast<cuuint64_t>(width) * kC * 2,
                                 static_cast<cuuint64_t>(height) * width * kC * 2};
  const cuuint32_t box[4] = {8, static_cast<cuuint32_t>(kRowPix), 1, 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(in), dims, strides,
                            box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 152;
}

// A kernel's limit of dynamic shared memory is raised on the current device only, and is gone after a reset of that device:
// it is set before every launch that needs more than 48 KB, not once in the process (a forward pass's three take 0.5-1 us
// of the 18 us that its launches take on the host).
template <class Kernel>
cudaError_t allow_shared(Kernel* kernel, int bytes) {
  return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

// Launch shapes of conv32_tc_kernel: ring slots, resident CTAs per SM, output rows per block.  Measured on
// 640x480 layers (CUDA events, batch 1 / batch 16): 6 slots x 2 CTAs x 8 rows 18.7 / 169 us; 8 x 2 x 8
// 18.7 / 178; 8 x 2 x 16 24.1 / 171; 6 x 3 x 8 18.7 / 219; 4 x 4 x 8 24.8 / 206; the earlier one-row-tile
// kernel (3 input rows loaded per output row) 22.8 / 277 us.
struct Conv32Variant {
  const void* fn;
  int slots, smem, ctas_per_sm, rows;
};
const Conv32Variant kConv32Variants[] = {
    {reinterpret_cast<const void*>(conv32_tc_kernel<6, 8>), 6, ring_smem_bytes<6>(), 2, 8},
    {reinterpret_cast<const void*>(conv32_tc_kernel<8, 8>), 8, ring_smem_bytes<8>(), 2, 8},
    {reinterpret_cast<const void*>(conv32_tc_kernel<8, 16>), 8, ring_smem_bytes<8>(), 2, 16},
};
constexpr int kConv32Default = 0;  // VH_CONV32_VARIANT selects another for launch-shape sweeps

const Conv32Variant& conv32_variant() {
  static int v = -1;
  if (v < 0) {
    v = kConv32Default;
    if (const char* env = std::getenv("VH_CONV32_VARIANT")) {
      const int x = std::atoi(env);
      if (x >= 0 && x < static_cast<int>(sizeof(kConv32Variants) / sizeof(kConv32Variants[0]))) v = x;
    }
  }
  return kConv32Variants[v];
}

}  // namespace

int conv32_smem_bytes() { return conv32_variant().smem; }

cudaError_t launch_conv32(const __nv_bfloat16* in, const __nv_bfloat16* wpack, const float* bias,
                          const __nv_bfloat16* mask, __nv_bfloat16* out, int batch, int width, int height, int mode,
                          int relu, unsigned int* error, cudaStream_t s, const unsigned int* gate) {
  const Conv32Variant& cv = conv32_variant();
  // persistent CTAs, cv.ctas_per_sm per SM: each CTA stages the weights and allocates tensor memory once
  const int ctas = cv.ctas_per_sm * sm_count();
  const long long ntiles = static_cast<long long>(batch) * height * ((width + kTile - 1) / kTile);
  if (ntiles > 0x7fffffffLL) return cudaErrorInvalidValue;  // the kernels' tile arithmetic is 32-bit
  const long long nitems =
      static_cast<long long>(batch) * ((height + cv.rows - 1) / cv.rows) * ((width + kTile - 1) / kTile);
  const int grid = static_cast<int>(nitems < ctas ? nitems : ctas);
  if (grid <= 0) return cudaSuccess;
  CUtensorMap map;
  cudaError_t e = encode_input_map(in, batch, width, height, &map);
  if (e == cudaSuccess) e = allow_shared(cv.fn, cv.smem);
  if (e != cudaSuccess) return e;
  void* args[] = {&map,    const_cast<__nv_bfloat16**>(&wpack), const_cast<float**>(&bias),
                  const_cast<__nv_bfloat16**>(&mask), &out, &batch, &width, &height, &mode, &relu,
                  const_cast<unsigned int**>(&gate), &error};
  return cudaLaunchKernel(cv.fn, dim3(grid), dim3(kThreads), args, static_cast<size_t>(cv.smem), s);
}

// Packs 32 x 32 x 3 x 3 FP32 weights w[co][ci][ky][kx] (transpose_flip: the input-gradient form, w'[ci][co][2-ky][2-kx])
// into the B operand layout [tap = ky * 3 + kx][ks][g][co][8] in BF16.
__global__ void pack_w32_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ out, int transpose_flip) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // one output element
  if (i >= 9 * kC * kC) return;
  const int c8 = i % 8;
  const int co = (i / 8) % kC;
  const int g = (i / (8 * kC)) % 2;
  const int ks = (i / (16 * kC)) % 2;
  const int tap = i / (32 * kC);
  const int ci = ks * 16 + g * 8 + c8;
  const int ky = tap / 3, kx = tap % 3;
  float v;
  if (!transpose_flip) {
    v = w[((co * kC + ci) * 3 + ky) * 3 + kx];
  } else {
    v = w[((ci * kC + co) * 3 + (2 - ky)) * 3 + (2 - kx)];
  }
  out[i] = __float2bfloat16_rn(v);
}

cudaError_t launch_pack_w32(const float* w, __nv_bfloat16* out, int transpose_flip, cudaStream_t s) {
  pack_w32_kernel<<<(9 * kC * kC + 255) / 256, 256, 0, s>>>(w, out, transpose_flip);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- weight gradient of a 32 -> 32 layer (tensor cores)
//
// dW[co][ci][ky][kx] += sum_p G[p][co] X[p + (ky - 1, kx - 1)][ci] and db[co] += sum_p G[p][co] over a batch of
// NHWC BF16 images (X: the layer's input activations, G: the gradient at its output, zero outside the image).
// As a GEMM per output row: M = (copy kx, input channel) = 3 x 32 rows plus a 32-row pad copy (M = 128), N = the
// 32 output channels, K = the row's pixels, one FP32 accumulator in tensor memory per tap row ky (3 x 32
// columns), summed over every output row the CTA takes and added to dW once at the end.
//
// A CTA takes items of kWgRows output rows of one kWgStrip-pixel strip.  Each input row is staged once, as three
// copies shifted by kx - 1 pixels, transposed into the canonical no-swizzle K-major layout
// [pixel group of 8 (K)][copy][channel][8 pixels]: the A operand of tap row ky of output row y is then the
// staged input row y - 1 + ky, its M rows (copy, channel) at a uniform 128-byte stride per 8 rows.  M rows
// 96..127 (the fourth "copy") read the next pixel group's first copy, or for the last group of the last ring
// slot the gradient ring that follows: staged values, finite, feeding only accumulator rows that are never
// read.  The gradient row is staged the same way as the B operand, [pixel group][output channel][8 pixels].  A
// thread loads a channel pair over 10 (8) pixels as 32-bit words and writes the transposed 16-byte rows with
// byte permutes; the loads of a row are issued a row ahead, so they are in flight while the row before it is
// staged and multiplied (a batch of 16 640x480 frames: 374 -> 330 us on average, 372 and 287 for the two layers; the
// rows' barriers and the loads' latency are the largest stalls).  Rows live in rings (three input rows, two
// gradient rows); thread 0 issues an output row's 12 MMAs (3 tap rows x 4 k-steps of 16 pixels) and commits them to an mbarrier, and a ring slot is
// rewritten only after the MMAs that read it have completed.  Four CTAs per SM (their tensor memory fills the
// SM's 512 columns).  Waits are bounded as in conv32_tc_kernel; a timeout is agreed on by every thread
// (__syncthreads_and) before the CTA leaves its loop.
namespace {

constexpr int kWgStrip = 64;                         // pixels of an output row per item (K of a row)
constexpr int kWgGroups = kWgStrip / 8;              // pixel groups of 8 (16 bytes of BF16)
constexpr int kWgCopies = 3;                         // kx = 0, 1, 2
constexpr int kWgCore = kC * 16;                     // one copy of one pixel group: 32 channels x 16 bytes
constexpr int kWgXLbo = kWgCopies * kWgCore;         // A operand: bytes between pixel groups (K)
constexpr int kWgXRow = kWgGroups * kWgXLbo;         // one staged input row: 12,288 bytes
constexpr int kWgGRow = kWgGroups * kWgCore;         // one staged gradient row: 4,096 bytes
constexpr int kWgXSlots = 3;                         // an output row reads 3 input rows; the slot a new row
                                                     // takes was last read by the previous output row
constexpr int kWgGSlots = 2;
constexpr int kWgRows = 16;                          // output rows per item
constexpr int kWgThreads = 128;                      // thread t stages pixel group t / 16, channel pair t % 16
constexpr int kWgTmemCols = 128;                     // 3 accumulators x 32 columns, allocated as a power of 2
constexpr int kWgCtasPerSm = 4;
constexpr int kWgSmem = 128 + kWgXSlots * kWgXRow + kWgGSlots * kWgGRow + 2 * 8 + 16;
// the A operand reads up to 3,583 bytes from its start (a second pixel group at +LBO, 16 M groups of 128 bytes),
// at most 511 bytes past its ring slot, which the next slot or the gradient ring covers
static_assert(kWgGSlots * kWgGRow >= 4 * kWgCore, "the last slot's pad rows stay inside the gradient ring");
static_assert(kWgCtasPerSm * kWgTmemCols <= 512, "tensor memory of the resident CTAs");
static_assert(kWgThreads == kWgGroups * (kC / 2), "one (pixel group, channel pair) per thread");

__global__ void __launch_bounds__(kWgThreads, kWgCtasPerSm) wgrad32_tc_kernel(const __nv_bfloat16* __restrict__ X,
                                                                    const __nv_bfloat16* __restrict__ G,
                                                                    float* __restrict__ dW, float* __restrict__ db,
                                                                    int batch, int width, int height,
                                                                    unsigned int* __restrict__ error) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  unsigned char* sX = smem;
  unsigned char* sG = smem + kWgXSlots * kWgXRow;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sG + kWgGSlots * kWgGRow);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pg = tid >> 4, cp = tid & 15;  // staging: pixel group, channel pair

  // the rings start zeroed, so that the pad rows read finite values before every slot has been staged
  for (int i = tid; i < (kWgXSlots * kWgXRow + kWgGSlots * kWgGRow) / 16; i += kWgThreads) {
    reinterpret_cast<uint4*>(sX)[i] = make_uint4(0u, 0u, 0u, 0u);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"(kWgTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bars[i])));
    asm volatile("fence.mbarrier_init.release.cluster;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  const uint32_t tmem = *tmem_slot;
  const uint32_t xs0 = smem_u32(sX), gs0 = smem_u32(sG), bar0 = smem_u32(&bars[0]);

  const uint32_t strips = static_cast<uint32_t>((width + kWgStrip - 1) / kWgStrip);
  const uint32_t rblocks = static_cast<uint32_t>((height + kWgRows - 1) / kWgRows);
  const uint32_t nitems = static_cast<uint32_t>(batch) * rblocks * strips;

  bool ok = true;
  uint32_t xq = 0;      // input rows staged
  uint32_t oq = 0;      // output rows issued (MMA groups), group g commits to bars[g & 1]
  uint32_t waited = 0;  // groups whose completion has been waited for, in order
  int reader[kWgXSlots];  // the last group that reads each input-row slot
#pragma unroll
  for (int k = 0; k < kWgXSlots; ++k) reader[k] = -1;
  float bsum0 = 0.0f, bsum1 = 0.0f;

  // waits, in order, for the groups up to g: a group's barrier phase is waited for before the group two later
  // commits to the same barrier, so a parity never refers to a phase two completions old
  auto wait_through = [&](int g) {
    while (ok && static_cast<int>(waited) <= g) {
      if (!mbar_wait(bar0 + 8u * (waited & 1u), (waited >> 1) & 1u)) {
        ok = false;
        break;
      }
      ++waited;
    }
  };

  // the words of input row y0 + i + 1 and, for i >= 0, gradient row y0 + i of an item
  auto load_rows = [&](uint32_t it, int i, uint32_t (&wv)[10], uint32_t (&gv)[8]) {
    const uint32_t rest = it / strips;
    const int xs = static_cast<int>(it - rest * strips) * kWgStrip;
    const uint32_t img = rest / rblocks;
    const int y0 = static_cast<int>(rest - img * rblocks) * kWgRows;
    const size_t img_base = static_cast<size_t>(img) * height;
    const int y = y0 + i + 1;
    const bool rok = y >= 0 && y < height;
    const unsigned int* rowp = reinterpret_cast<const unsigned int*>(X + (img_base + (rok ? y : 0)) * width * kC) + cp;
#pragma unroll
    for (int j = 0; j < 10; ++j) {
      const int px = xs - 1 + 8 * pg + j;
      wv[j] = (rok && px >= 0 && px < width) ? __ldg(rowp + static_cast<size_t>(px) * (kC / 2)) : 0u;
    }
    if (i >= 0) {
      const unsigned int* growp = reinterpret_cast<const unsigned int*>(G + (img_base + (y0 + i)) * width * kC) + cp;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int px = xs + 8 * pg + j;
        gv[j] = px < width ? __ldg(growp + static_cast<size_t>(px) * (kC / 2)) : 0u;
      }
    }
  };
  uint32_t nwv[10], ngv[8];  // the next row's words: in flight while this row is staged and multiplied
#pragma unroll
  for (int j = 0; j < 8; ++j) ngv[j] = 0u;
  if (blockIdx.x < nitems) load_rows(blockIdx.x, -2, nwv, ngv);

  for (uint32_t it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
    const uint32_t rest = it / strips;
    const uint32_t img = rest / rblocks;
    const int y0 = static_cast<int>(rest - img * rblocks) * kWgRows;
    const int rows = min(kWgRows, height - y0);
    const uint32_t xa = xq;  // ring index of input row y0 - 1
    for (int i = -2; i < rows; ++i) {
      // stage input row y0 + i + 1 and, for i >= 0, gradient row y0 + i; then issue output row y0 + i
      uint32_t wv[10], gv[8];
#pragma unroll
      for (int j = 0; j < 10; ++j) wv[j] = nwv[j];
#pragma unroll
      for (int j = 0; j < 8; ++j) gv[j] = ngv[j];
      if (i + 1 < rows) {
        load_rows(it, i + 1, nwv, ngv);
      } else if (it + gridDim.x < nitems) {
        load_rows(it + gridDim.x, -2, nwv, ngv);
      }
      const uint32_t sx = xq % kWgXSlots;
      if (reader[sx] >= 0) wait_through(reader[sx]);
      if (i >= 0 && oq >= 2) wait_through(static_cast<int>(oq) - 2);
      if (ok) {
        unsigned char* dst = sX + sx * kWgXRow + pg * kWgXLbo + (2 * cp) * 16;
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          uint4 lo, hi;
          lo.x = __byte_perm(wv[kx + 0], wv[kx + 1], 0x5410);
          lo.y = __byte_perm(wv[kx + 2], wv[kx + 3], 0x5410);
          lo.z = __byte_perm(wv[kx + 4], wv[kx + 5], 0x5410);
          lo.w = __byte_perm(wv[kx + 6], wv[kx + 7], 0x5410);
          hi.x = __byte_perm(wv[kx + 0], wv[kx + 1], 0x7632);
          hi.y = __byte_perm(wv[kx + 2], wv[kx + 3], 0x7632);
          hi.z = __byte_perm(wv[kx + 4], wv[kx + 5], 0x7632);
          hi.w = __byte_perm(wv[kx + 6], wv[kx + 7], 0x7632);
          *reinterpret_cast<uint4*>(dst + kx * kWgCore) = lo;
          *reinterpret_cast<uint4*>(dst + kx * kWgCore + 16) = hi;
        }
        if (i >= 0) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            bsum0 += __uint_as_float(gv[j] << 16);
            bsum1 += __uint_as_float(gv[j] & 0xffff0000u);
          }
          unsigned char* gdst = sG + (oq % kWgGSlots) * kWgGRow + pg * kWgCore + (2 * cp) * 16;
          uint4 lo, hi;
          lo.x = __byte_perm(gv[0], gv[1], 0x5410);
          lo.y = __byte_perm(gv[2], gv[3], 0x5410);
          lo.z = __byte_perm(gv[4], gv[5], 0x5410);
          lo.w = __byte_perm(gv[6], gv[7], 0x5410);
          hi.x = __byte_perm(gv[0], gv[1], 0x7632);
          hi.y = __byte_perm(gv[2], gv[3], 0x7632);
          hi.z = __byte_perm(gv[4], gv[5], 0x7632);
          hi.w = __byte_perm(gv[6], gv[7], 0x7632);
          *reinterpret_cast<uint4*>(gdst) = lo;
          *reinterpret_cast<uint4*>(gdst + 16) = hi;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the staged rows, for the MMAs' reads
      ok = __syncthreads_and(ok) != 0;
      ++xq;
      if (!ok) break;
      if (i < 0) continue;
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        const uint32_t b_row = gs0 + (oq % kWgGSlots) * kWgGRow;
        for (int ky = 0; ky < 3; ++ky) {
          const uint32_t a_row = xs0 + ((xa + static_cast<uint32_t>(i + ky)) % kWgXSlots) * kWgXRow;
          for (int ks = 0; ks < kWgStrip / 16; ++ks) {
            const uint64_t a = smem_desc(a_row + ks * 2 * kWgXLbo, kWgXLbo, 128);
            const uint64_t b = smem_desc(b_row + ks * 2 * kWgCore, kWgCore, 128);
            mma(tmem + 32u * ky, a, b, (oq == 0 && ks == 0) ? 0u : 1u);
          }
        }
        commit(bar0 + 8u * (oq & 1u));
      }
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) reader[(xa + static_cast<uint32_t>(i + ky)) % kWgXSlots] = static_cast<int>(oq);
      ++oq;
    }
  }
  if (ok && oq > 0) wait_through(static_cast<int>(oq) - 1);
  ok = __syncthreads_and(ok) != 0;
  if (ok && oq > 0 && warp < 3) {  // warp kx reads TMEM lanes 32 kx .. 32 kx + 31 = input channel `lane`
    asm volatile("tcgen05.fence::after_thread_sync;\n");
    for (int ky = 0; ky < 3; ++ky) {
      float acc[32];
      tmem_ld32(tmem + 32u * ky + (static_cast<uint32_t>(warp * 32) << 16), acc);
#pragma unroll
      for (int co = 0; co < kC; ++co) atomicAdd(&dW[(co * kC + lane) * 9 + ky * 3 + warp], acc[co]);
    }
  }
  if (ok) {
    // pixel groups pg and pg + 1 of a channel pair are lanes l and l ^ 16 of one warp
    bsum0 += __shfl_xor_sync(0xffffffffu, bsum0, 16);
    bsum1 += __shfl_xor_sync(0xffffffffu, bsum1, 16);
    if (lane < 16 && oq > 0) {
      atomicAdd(&db[2 * cp], bsum0);
      atomicAdd(&db[2 * cp + 1], bsum1);
    }
  }
  if (!ok) {
    if (lane == 0) atomicOr(error, kErrorBit);
    // the MMA groups still in flight complete before tensor memory is freed (bounded waits)
    if (tid == 0) {
      for (uint32_t w = waited; w < oq; ++w) mbar_wait(bar0 + 8u * (w & 1u), (w >> 1) & 1u);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kWgTmemCols));
  }
}

}  // namespace

cudaError_t launch_wgrad32(const __nv_bfloat16* x, const __nv_bfloat16* g, float* dw, float* db, int batch, int width,
                           int height, unsigned int* error, cudaStream_t s) {
  const int ctas = kWgCtasPerSm * sm_count();
  if (reinterpret_cast<uintptr_t>(x) % 4 != 0 || reinterpret_cast<uintptr_t>(g) % 4 != 0) return cudaErrorInvalidValue;
  const long long nitems = static_cast<long long>(batch) * ((height + kWgRows - 1) / kWgRows) *
                           ((width + kWgStrip - 1) / kWgStrip);
  if (nitems > 0x7fffffffLL) return cudaErrorInvalidValue;  // the item arithmetic is 32-bit
  const int grid = static_cast<int>(nitems < ctas ? nitems : ctas);
  if (grid <= 0) return cudaSuccess;
  const cudaError_t e = allow_shared(wgrad32_tc_kernel, kWgSmem);
  if (e != cudaSuccess) return e;
  wgrad32_tc_kernel<<<grid, kWgThreads, kWgSmem, s>>>(x, g, dw, db, batch, width, height, error);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- the rest of the net (CUDA cores)
//
// Parameters, one FP32 array (kParamCount): w1[32][4][3][3] b1[32] w2[32][32][3][3] b2[32] w3[32][32][3][3] b3[32]
// w4[32][3][3] b4.  Input channels per pixel (FP32): the depth's local high-pass (d - m) * 100 (centimetres;
// m = mean of the valid depths of the 3x3 neighbourhood), the validity mask, and m / 4 (the depth level); the
// output is the residual r in centimetres, depth' = d + r / 100 on valid pixels (clamped at 0).  The
// high-pass keeps the BF16 activations' 8 significant bits on the noise rather than on metres of depth.
namespace {

constexpr int kCin = 4;
constexpr float kScale = 100.0f, kInvScale = 0.01f;
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kC * kCin * 9, kOffW2 = kOffB1 + kC, kOffB2 = kOffW2 + kC * kC * 9;
constexpr int kOffW3 = kOffB2 + kC, kOffB3 = kOffW3 + kC * kC * 9, kOffW4 = kOffB3 + kC, kOffB4 = kOffW4 + kC * 9;
constexpr int kParams = kOffB4 + 1;
// depth-discontinuity threshold max(base, rel * depth) of the reference's GPU path (cuda_tsdf_integrator.cu:27-28):
// training ignores pixels whose raw depth and target differ by more (they see different surfaces), and at
// inference a correction larger than it falls back to the bilateral filter's value
constexpr float kGateBase = 0.012f, kGateRel = 0.025f;

__device__ __forceinline__ float gate(float d) { return fmaxf(kGateBase, kGateRel * d); }

__device__ __forceinline__ bool inside(int x, int y, int w, int h) { return x >= 0 && x < w && y >= 0 && y < h; }

// ---- packed single-precision arithmetic: two FP32 multiply-adds per instruction ----
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// two BF16 of one word as FP32
__device__ __forceinline__ f32x2 bf2_to_f32x2(uint32_t v) {
  return pack2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// The tiles of the CUDA-core layers: kTileW x kTileH pixels of one image, 256 threads, warp w on rows w and w + 8
// (thread: pixels (lane, w) and (lane, w + 8)).
constexpr int kTileW = 32, kTileH = 16, kTileThreads = 256;

struct TileGrid {
  int tx, ty;
  long long count;
};
__host__ __device__ inline TileGrid tile_grid(int batch, int w, int h, int tw, int th) {
  TileGrid g{(w + tw - 1) / tw, (h + th - 1) / th, 0};
  g.count = static_cast<long long>(batch) * g.tx * g.ty;
  return g;
}
__device__ __forceinline__ void tile_at(const TileGrid& g, long long t, int tw, int th, int& img, int& x0, int& y0) {
  const uint32_t i = static_cast<uint32_t>(t), row = i / static_cast<uint32_t>(g.tx);
  x0 = static_cast<int>(i - row * static_cast<uint32_t>(g.tx)) * tw;
  img = static_cast<int>(row / static_cast<uint32_t>(g.ty));
  y0 = static_cast<int>(row - static_cast<uint32_t>(img) * static_cast<uint32_t>(g.ty)) * th;
}

// The input channels (see above) of the tile at (x0, y0) and a ring of one pixel around it, from the depth, staged
// with a ring of two (0 outside the image, which counts as invalid).
template <int TW, int TH>
struct InputTile {
  float depth[TH + 4][TW + 4];
  float4 X[TH + 2][TW + 2];
};
// the depth words of a tile that a thread stages, in flight while the tile before is worked on
template <int TW, int TH>
struct DepthAhead {
  static constexpr int kPer = ((TH + 4) * (TW + 4) + kTileThreads - 1) / kTileThreads;
  float v[kPer];
  __device__ __forceinline__ void load(const float* __restrict__ depth, int img, int x0, int y0, int w, int h) {
    const float* d0 = depth + static_cast<size_t>(img) * w * h;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = threadIdx.x + k * kTileThreads, r = i / (TW + 4), c = i - r * (TW + 4);
      const int x = x0 + c - 2, y = y0 + r - 2;
      v[k] = r < TH + 4 && inside(x, y, w, h) ? __ldg(d0 + static_cast<size_t>(y) * w + x) : 0.0f;
    }
  }
};
template <int TW, int TH>
__device__ __forceinline__ void stage_input(InputTile<TW, TH>& S, const DepthAhead<TW, TH>& ahead) {
#pragma unroll
  for (int k = 0; k < DepthAhead<TW, TH>::kPer; ++k) {
    const int i = threadIdx.x + k * kTileThreads;
    if (i < (TH + 4) * (TW + 4)) (&S.depth[0][0])[i] = ahead.v[k];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < (TH + 2) * (TW + 2); i += kTileThreads) {
    const int r = i / (TW + 2), c = i - r * (TW + 2);
    const float d = S.depth[r + 1][c + 1];
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (d > 0.0f) {
      float sum = 0.0f;
      int cnt = 0;
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        const float n = S.depth[r + t / 3][c + t % 3];
        if (n > 0.0f) {
          sum += n;
          ++cnt;
        }
      }
      const float m = sum / static_cast<float>(cnt);  // at least the pixel itself
      v = make_float4((d - m) * kScale, 1.0f, m * 0.25f, 0.0f);
    }
    S.X[r][c] = v;
  }
  __syncthreads();
}

// a warp's 32 pixels of row y from (x0, y), 64 bytes each, between a lane per pixel and global memory through its
// shared-memory buffer (epi_pos): 512 contiguous bytes per access instruction
__device__ __forceinline__ void store_row32(uint4* buf, const uint4 (&v)[4], __nv_bfloat16* __restrict__ out, size_t row,
                                            int x0, int w, int lane) {
#pragma unroll
  for (int q = 0; q < 4; ++q) buf[epi_pos(lane, q)] = v[q];
  __syncwarp();
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int p = 8 * u + (lane >> 2), q = lane & 3;
    if (x0 + p < w) *reinterpret_cast<uint4*>(out + (row + x0 + p) * kC + 8 * q) = buf[epi_pos(p, q)];
  }
  __syncwarp();
}
// The 32 pixels from (x0, row) copied into a warp's buffer without passing through registers (0 outside the image),
// pixel p's chunk q at epi_pos(p, q) or, kLinear, at 4 p + q: read by the same warp once async_wait has passed.
template <bool kLinear>
__device__ __forceinline__ void async_row32(uint4* buf, const __nv_bfloat16* __restrict__ in, size_t row, int x0, int w,
                                            bool row_in, int lane) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int p = 8 * u + (lane >> 2), q = lane & 3, x = x0 + p;
    const bool ok = row_in && x >= 0 && x < w;
    const __nv_bfloat16* src = ok ? in + (row + x) * kC + 8 * q : in;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(&buf[kLinear ? 4 * p + q : epi_pos(p, q)])),
                 "l"(src), "r"(ok ? 16 : 0)
                 : "memory");
  }
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// all but the newest kAhead groups of this thread have arrived; the warp's lanes see each other's
template <int kAhead>
__device__ __forceinline__ void async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kAhead) : "memory");
  __syncwarp();
}

// layer 1: the input channels from the depth (in shared memory only), 4 -> 32, ReLU; the fourth channel is always 0 and
// takes no products.  Two pixels per thread share the weights' shared-memory reads, and two output channels go
// through one packed multiply-add: 27 x 16 of them a pixel.  Bound by FP32 arithmetic (105 us at the full rate for a batch
// of 16 640x480 frames): 260 us, against 457 with the channels in global memory, one pixel a thread and scalar
// multiply-adds; the next tile's depth is loaded during this one's products (283 us without).
__global__ void __launch_bounds__(kTileThreads, 2) conv_in_kernel(const float* __restrict__ depth,
                                                                  const float* __restrict__ params,
                                                                  __nv_bfloat16* __restrict__ A1, int batch, int w, int h) {
  __shared__ InputTile<kTileW, kTileH> S;
  __shared__ __align__(16) float sw[9][3][kC];
  __shared__ __align__(16) float sb[kC];
  __shared__ uint4 sbuf[kTileThreads / 32][128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 9 * 3 * kC; i += kTileThreads) {
    const int t = i / (3 * kC), ci = (i / kC) % 3, co = i % kC;
    sw[t][ci][co] = params[kOffW1 + (co * kCin + ci) * 9 + t];
  }
  if (threadIdx.x < kC) sb[threadIdx.x] = params[kOffB1 + threadIdx.x];
  const TileGrid g = tile_grid(batch, w, h, kTileW, kTileH);
  int img, x0, y0;
  DepthAhead<kTileW, kTileH> ahead;
  if (blockIdx.x < g.count) {
    tile_at(g, blockIdx.x, kTileW, kTileH, img, x0, y0);
    ahead.load(depth, img, x0, y0, w, h);
  }
  for (long long tile = blockIdx.x; tile < g.count; tile += gridDim.x) {
    tile_at(g, tile, kTileW, kTileH, img, x0, y0);
    __syncthreads();  // the previous tile has been read
    stage_input(S, ahead);
    if (tile + gridDim.x < g.count) {
      int nimg, nx0, ny0;
      tile_at(g, tile + gridDim.x, kTileW, kTileH, nimg, nx0, ny0);
      ahead.load(depth, nimg, nx0, ny0, w, h);
    }
    f32x2 acc[2][kC / 2];
#pragma unroll
    for (int c = 0; c < kC / 2; ++c) acc[0][c] = acc[1][c] = reinterpret_cast<const f32x2*>(sb)[c];
#pragma unroll 1
    for (int t = 0; t < 9; ++t) {
      const float4 xa = S.X[warp + t / 3][lane + t % 3], xb = S.X[warp + 8 + t / 3][lane + t % 3];
      const float va[3] = {xa.x, xa.y, xa.z}, vb[3] = {xb.x, xb.y, xb.z};
#pragma unroll
      for (int ci = 0; ci < 3; ++ci) {
        const f32x2 pa = pack2(va[ci], va[ci]), pb = pack2(vb[ci], vb[ci]);
        const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(sw[t][ci]);
#pragma unroll
        for (int c = 0; c < kC / 4; ++c) {
          const ulonglong2 wv = wp[c];
          acc[0][2 * c] = fma2(wv.x, pa, acc[0][2 * c]);
          acc[0][2 * c + 1] = fma2(wv.y, pa, acc[0][2 * c + 1]);
          acc[1][2 * c] = fma2(wv.x, pb, acc[1][2 * c]);
          acc[1][2 * c + 1] = fma2(wv.y, pb, acc[1][2 * c + 1]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int y = y0 + warp + 8 * r;
      __align__(16) __nv_bfloat162 res[kC / 2];
#pragma unroll
      for (int c = 0; c < kC / 2; ++c) {
        float lo, hi;
        unpack2(acc[r][c], lo, hi);
        res[c] = __floats2bfloat162_rn(fmaxf(lo, 0.0f), fmaxf(hi, 0.0f));
      }
      uint4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const uint4*>(res)[q];
      if (y < h) store_row32(sbuf[warp], v, A1, (static_cast<size_t>(img) * h + y) * w, x0, w, lane);
    }
  }
}

// layer 4: 32 -> 1 residual, depth' = d + r / 100 on valid pixels.  Every input pixel's products with the 9 taps'
// weights are summed over its channels once (9 sums a pixel, packed multiply-adds over channel pairs, two pixels a
// thread sharing the weights' reads) and an output pixel adds 9 of those sums from shared memory; a CTA's 32 x 16
// input pixels give 30 x 14 outputs.  148 us for a batch of 16 640x480 frames; one thread per (output pixel, 8
// channels) read and converted every activation 9 times: 380 us.
constexpr int kOutW = kTileW - 2, kOutH = kTileH - 2, kOutCtas = 3;
constexpr int kOutRowBytes = kTileThreads / 32 * 2 * 128 * 16, kOutSmem = kOutRowBytes + 9 * kTileH * kTileW * 4;

__global__ void __launch_bounds__(kTileThreads, kOutCtas) conv_out_kernel(const __nv_bfloat16* __restrict__ A3,
                                                                   const float* __restrict__ params,
                                                                   const float* __restrict__ depth,
                                                                   const float* __restrict__ fallback,
                                                                   float* __restrict__ out, int batch, int w, int h) {
  extern __shared__ __align__(16) unsigned char out_smem[];
  uint4(*rows)[2][128] = reinterpret_cast<uint4(*)[2][128]>(out_smem);  // [warp][row][chunk]
  float(*S)[kTileH][kTileW] = reinterpret_cast<float(*)[kTileH][kTileW]>(out_smem + kOutRowBytes);
  __shared__ __align__(16) float sw[9][kC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 9 * kC; i += kTileThreads) sw[i / kC][i % kC] = params[kOffW4 + (i % kC) * 9 + i / kC];
  const float sb = params[kOffB4];
  const TileGrid g = tile_grid(batch, w, h, kOutW, kOutH);
  auto fetch = [&](long long tile) {  // this warp's two rows of a tile, in flight while the tile before is worked on
    if (tile < g.count) {
      int img, x0, y0;
      tile_at(g, tile, kOutW, kOutH, img, x0, y0);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int y = y0 - 1 + warp + 8 * r;
        const bool in = y >= 0 && y < h;
        async_row32<false>(rows[warp][r], A3, (static_cast<size_t>(img) * h + (in ? y : 0)) * w, x0 - 1, w, in, lane);
      }
    }
    async_commit();
  };
  fetch(blockIdx.x);
  for (long long tile = blockIdx.x; tile < g.count; tile += gridDim.x) {
    int img, x0, y0;
    tile_at(g, tile, kOutW, kOutH, img, x0, y0);
    const size_t base = static_cast<size_t>(img) * h;
    uint4 a[2][4];
    async_wait<0>();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[r][q] = rows[warp][r][epi_pos(lane, q)];
    }
    __syncwarp();
    fetch(tile + gridDim.x);
    __syncthreads();  // the weights; the previous tile's sums have been read
    f32x2 acc[2][9];
#pragma unroll
    for (int t = 0; t < 9; ++t) acc[0][t] = acc[1][t] = 0ULL;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t w0[4] = {a[0][q].x, a[0][q].y, a[0][q].z, a[0][q].w};
      const uint32_t w1[4] = {a[1][q].x, a[1][q].y, a[1][q].z, a[1][q].w};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const f32x2 p0 = bf2_to_f32x2(w0[2 * j]), p1 = bf2_to_f32x2(w0[2 * j + 1]);
        const f32x2 r0 = bf2_to_f32x2(w1[2 * j]), r1 = bf2_to_f32x2(w1[2 * j + 1]);
#pragma unroll
        for (int t = 0; t < 9; ++t) {
          const ulonglong2 wv = *reinterpret_cast<const ulonglong2*>(&sw[t][8 * q + 4 * j]);
          acc[0][t] = fma2(wv.y, p1, fma2(wv.x, p0, acc[0][t]));
          acc[1][t] = fma2(wv.y, r1, fma2(wv.x, r0, acc[1][t]));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        float lo, hi;
        unpack2(acc[r][t], lo, hi);
        S[t][warp + 8 * r][lane] = lo + hi;
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kOutW * kOutH; i += kTileThreads) {
      const int oy = i / kOutW, ox = i - oy * kOutW;
      const int x = x0 + ox, y = y0 + oy;
      if (x >= w || y >= h) continue;
      const size_t at = (base + y) * w + x;
      const float d = depth[at];
      if (!(d > 0.0f)) {
        out[at] = 0.0f;
        continue;
      }
      float r = 0.0f;
#pragma unroll
      for (int t = 0; t < 9; ++t) r += S[t][oy + t / 3][ox + t % 3];
      const float corr = (sb + r) * kInvScale;
      out[at] = (fallback && fabsf(corr) > gate(d)) ? fallback[at] : fmaxf(d + corr, 0.0f);
    }
  }
}

// The output layer's backward pass in one read of the activations A3:
//   the loss (sum over pixels valid in input, target and output whose input and target agree within the discontinuity
//   threshold, of (out - target)^2 / n_pixels) and dr = dloss/dr of the tile and a ring around it, in shared memory;
//   dA3[q][c] = (A3[q][c] > 0) * sum_t w4[c][t] dr[q - off(t)], BF16 (packed multiply-adds over channel pairs, two
//   pixels a thread);
//   dw4[c][t] += sum_q A3[q][c] dr[q - off(t)], db4 += sum_q dr[q]: lane = (channel pair, half of the warp's 32
//   pixels), the 9 taps' dr sliding along the row in registers; summed over the CTA's tiles, one atomic per weight.
// 283 us for a batch of 16 640x480 frames (HBM needs 92, FP32 arithmetic 70); as three kernels, the weight gradients
// from segments staged three rows at a time, 723 us.
constexpr int kOutBackSmem = 2 * kTileThreads / 32 * 2 * 128 * 16;  // two stages of a tile's activations

__global__ void __launch_bounds__(kTileThreads, 2) out_backward_kernel(
    const __nv_bfloat16* __restrict__ A3, const float* __restrict__ params, const float* __restrict__ depth,
    const float* __restrict__ target, const float* __restrict__ out, __nv_bfloat16* __restrict__ dA3,
    float* __restrict__ dw4, float* __restrict__ db4, float* __restrict__ loss, int batch, int w, int h) {
  constexpr int kWarps = kTileThreads / 32, kRing = (kTileH + 2) * (kTileW + 2);
  constexpr int kPer = (kRing + kTileThreads - 1) / kTileThreads;
  extern __shared__ __align__(16) unsigned char out_smem[];
  uint4(*rows)[kWarps][2][128] = reinterpret_cast<uint4(*)[kWarps][2][128]>(out_smem);  // [stage][warp][row][chunk]
  __shared__ __align__(16) float sw[9][kC];
  __shared__ float sdr[kTileH + 2][kTileW + 2];
  __shared__ uint4 sbuf[kWarps][128];
  __shared__ float sred[9][kC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < 9 * kC; i += kTileThreads) {
    sw[i / kC][i % kC] = params[kOffW4 + (i % kC) * 9 + i / kC];
    sred[i / kC][i % kC] = 0.0f;
  }
  const float inv_n = 1.0f / static_cast<float>(static_cast<long long>(batch) * w * h);
  const int pair = lane & 15, part = lane >> 4;
  f32x2 wacc[9];
#pragma unroll
  for (int t = 0; t < 9; ++t) wacc[t] = 0ULL;
  float se = 0.0f, cnt = 0.0f, dsum = 0.0f;
  const TileGrid g = tile_grid(batch, w, h, kTileW, kTileH);
  // a tile's activations (this warp's two rows) and the depth, target and output of its ring: in flight while the
  // tile before is worked on
  float fd[kPer], ft[kPer], fo[kPer];
  auto fetch = [&](long long tile, int stage) {
    if (tile < g.count) {
      int img, x0, y0;
      tile_at(g, tile, kTileW, kTileH, img, x0, y0);
      const size_t base = static_cast<size_t>(img) * h;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int y = y0 + warp + 8 * r;
        async_row32<false>(rows[stage][warp][r], A3, (base + min(y, h - 1)) * w, x0, w, y < h, lane);
      }
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const int i = threadIdx.x + k * kTileThreads, r = i / (kTileW + 2), c = i - r * (kTileW + 2);
        const int x = x0 + c - 1, y = y0 + r - 1;
        fd[k] = ft[k] = fo[k] = 0.0f;
        if (i < kRing && inside(x, y, w, h)) {
          const size_t at = (base + y) * w + x;
          fd[k] = __ldg(depth + at);
          ft[k] = __ldg(target + at);
          fo[k] = __ldg(out + at);
        }
      }
    }
    async_commit();
  };
  fetch(blockIdx.x, 0);
  int stage = 0;
  for (long long tile = blockIdx.x; tile < g.count; tile += gridDim.x, stage ^= 1) {
    int img, x0, y0;
    tile_at(g, tile, kTileW, kTileH, img, x0, y0);
    const size_t base = static_cast<size_t>(img) * h;
    __syncthreads();  // the previous tile's dr has been read
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = threadIdx.x + k * kTileThreads, r = i / (kTileW + 2), c = i - r * (kTileW + 2);
      if (i >= kRing) break;
      const float d = fd[k], t = ft[k], o = fo[k];  // 0 outside the image
      const bool m = d > 0.0f && t > 0.0f && o > 0.0f && fabsf(d - t) <= gate(t);
      const float diff = m ? o - t : 0.0f;
      const float v = 2.0f * diff * kInvScale * inv_n;
      if (r >= 1 && r <= kTileH && c >= 1 && c <= kTileW) {
        se += diff * diff;
        cnt += m ? 1.0f : 0.0f;
        dsum += v;
      }
      sdr[r][c] = v;
    }
    __syncthreads();
    fetch(tile + gridDim.x, stage ^ 1);
    async_wait<1>();
    const uint4(*act)[128] = rows[stage][warp];
    // the activations' gradient
    f32x2 acc[2][kC / 2];
#pragma unroll
    for (int c = 0; c < kC / 2; ++c) acc[0][c] = acc[1][c] = 0ULL;
#pragma unroll 1
    for (int t = 0; t < 9; ++t) {
      const float ga = sdr[warp + 2 - t / 3][lane + 2 - t % 3], gb = sdr[warp + 10 - t / 3][lane + 2 - t % 3];
      const f32x2 pa = pack2(ga, ga), pb = pack2(gb, gb);
      const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(sw[t]);
#pragma unroll
      for (int c = 0; c < kC / 4; ++c) {
        const ulonglong2 wv = wp[c];
        acc[0][2 * c] = fma2(wv.x, pa, acc[0][2 * c]);
        acc[0][2 * c + 1] = fma2(wv.y, pa, acc[0][2 * c + 1]);
        acc[1][2 * c] = fma2(wv.x, pb, acc[1][2 * c]);
        acc[1][2 * c + 1] = fma2(wv.y, pb, acc[1][2 * c + 1]);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int y = y0 + warp + 8 * r;
      __align__(16) __nv_bfloat162 res[kC / 2];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 a4 = act[r][epi_pos(lane, q)];
        const uint32_t words[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float lo, hi, alo, ahi;
          unpack2(acc[r][4 * q + j], lo, hi);
          unpack2(bf2_to_f32x2(words[j]), alo, ahi);
          res[4 * q + j] = __floats2bfloat162_rn(alo > 0.0f ? lo : 0.0f, ahi > 0.0f ? hi : 0.0f);
        }
      }
      uint4 v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = reinterpret_cast<const uint4*>(res)[q];
      if (y < h) store_row32(sbuf[warp], v, dA3, (base + y) * w, x0, w, lane);
    }
    // the weights' gradients: word `pair` of pixel p is in its chunk pair / 4
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
      const uint32_t* words = reinterpret_cast<const uint32_t*>(act[r]);
      const int row = warp + 8 * r, p0 = 16 * part;
      // dr at column p + 2 - kx of rows row + 2 - ky: the window's columns p (kx = 2), p + 1, p + 2 (kx = 0)
      f32x2 win[3][3];  // [ky][column]
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const float v = sdr[row + 2 - ky][p0 + c];
          win[ky][c + 1] = pack2(v, v);
        }
      }
#pragma unroll 4
      for (int p = p0; p < p0 + 16; ++p) {
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          const float v = sdr[row + 2 - ky][p + 2];
          win[ky][0] = win[ky][1];
          win[ky][1] = win[ky][2];
          win[ky][2] = pack2(v, v);
        }
        const f32x2 av = bf2_to_f32x2(words[4 * epi_pos(p, pair >> 2) + (pair & 3)]);
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
#pragma unroll
          for (int kx = 0; kx < 3; ++kx) wacc[3 * ky + kx] = fma2(av, win[ky][2 - kx], wacc[3 * ky + kx]);
        }
      }
    }
    __syncwarp();  // the stage is refilled after the next tile's start
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    float lo, hi;
    unpack2(wacc[t], lo, hi);
    lo += __shfl_xor_sync(0xffffffffu, lo, 16);
    hi += __shfl_xor_sync(0xffffffffu, hi, 16);
    if (part == 0) {
      atomicAdd(&sred[t][2 * pair], lo);
      atomicAdd(&sred[t][2 * pair + 1], hi);
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    se += __shfl_down_sync(0xffffffffu, se, o);
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    dsum += __shfl_down_sync(0xffffffffu, dsum, o);
  }
  if (lane == 0) {
    atomicAdd(&loss[0], se);
    atomicAdd(&loss[1], cnt);
    atomicAdd(db4, dsum);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 9 * kC; i += kTileThreads) atomicAdd(&dw4[(i % kC) * 9 + i / kC], sred[i / kC][i % kC]);
}

// The input layer's weight gradients dw1[co][ci][t] += sum_p dY[p][co] X[p + off(t)][ci], db1[co] += sum_p dY[p][co]:
// lane = output channel, a warp runs along its row's 32 pixels with the 9 taps' input channels (from the depth, as in
// conv_in_kernel) sliding in registers, two input channels per packed multiply-add; summed over the CTA's tiles, one
// atomic per weight.  Bound by FP32 arithmetic and issue: 274 us for a batch of 16 640x480 frames, against 472 with
// (output, input) channel threads over staged segments.
constexpr int kWgInH = 8;  // rows of a tile: one per warp

__global__ void __launch_bounds__(kTileThreads, 2) wgrad_in_kernel(const float* __restrict__ depth,
                                                                   const __nv_bfloat16* __restrict__ dY,
                                                                   float* __restrict__ dw1, float* __restrict__ db1,
                                                                   int batch, int w, int h) {
  constexpr int kWarps = kTileThreads / 32;
  static_assert(kWarps == kWgInH, "one row per warp");
  __shared__ InputTile<kTileW, kWgInH> S;
  __shared__ uint4 sbuf[2][kWarps][128];  // two stages of a row's gradients, 64 bytes a pixel
  __shared__ float sred[kC * 3 * 9 + kC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kC * 3 * 9 + kC; i += kTileThreads) sred[i] = 0.0f;
  f32x2 acc[9];   // channels 0 and 1
  float acc2[9];  // channel 2
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    acc[t] = 0ULL;
    acc2[t] = 0.0f;
  }
  float bacc = 0.0f;
  const TileGrid g = tile_grid(batch, w, h, kTileW, kWgInH);
  DepthAhead<kTileW, kWgInH> ahead;
  auto fetch = [&](long long tile, int stage) {
    if (tile < g.count) {
      int img, x0, y0;
      tile_at(g, tile, kTileW, kWgInH, img, x0, y0);
      const int y = y0 + warp;
      async_row32<true>(sbuf[stage][warp], dY, (static_cast<size_t>(img) * h + min(y, h - 1)) * w, x0, w, y < h, lane);
      ahead.load(depth, img, x0, y0, w, h);
    }
    async_commit();
  };
  fetch(blockIdx.x, 0);
  int stage = 0;
  for (long long tile = blockIdx.x; tile < g.count; tile += gridDim.x, stage ^= 1) {
    __syncthreads();  // the previous tile has been read
    stage_input(S, ahead);
    fetch(tile + gridDim.x, stage ^ 1);
    async_wait<1>();
    const uint16_t* gr = reinterpret_cast<const uint16_t*>(sbuf[stage][warp]);
    f32x2 win[3][3];  // [ky][column]: a pixel's channels 0 and 1
    float win2[3][3];  // channel 2
    auto column = [&](int ky, int c, int to) {
      const float4 v = S.X[warp + ky][c];
      win[ky][to] = pack2(v.x, v.y);
      win2[ky][to] = v.z;
    };
#pragma unroll
    for (int ky = 0; ky < 3; ++ky) {
      column(ky, 0, 1);
      column(ky, 1, 2);
    }
#pragma unroll 3
    for (int p = 0; p < kTileW; ++p) {
      const float gv = __uint_as_float(static_cast<uint32_t>(gr[p * kC + lane]) << 16);
      const f32x2 gp = pack2(gv, gv);
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        win[ky][0] = win[ky][1];
        win[ky][1] = win[ky][2];
        win2[ky][0] = win2[ky][1];
        win2[ky][1] = win2[ky][2];
        column(ky, p + 2, 2);
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
          acc[3 * ky + kx] = fma2(gp, win[ky][kx], acc[3 * ky + kx]);
          acc2[3 * ky + kx] = fmaf(gv, win2[ky][kx], acc2[3 * ky + kx]);
        }
      }
      bacc += gv;
    }
    __syncwarp();
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    float v[3];
    unpack2(acc[t], v[0], v[1]);
    v[2] = acc2[t];
#pragma unroll
    for (int ci = 0; ci < 3; ++ci) atomicAdd(&sred[(lane * 3 + ci) * 9 + t], v[ci]);
  }
  atomicAdd(&sred[kC * 3 * 9 + lane], bacc);
  __syncthreads();
  // [co][ci][t]; the gradients of the fourth channel, which is always 0, stay 0
  for (int i = threadIdx.x; i < kC * 3 * 9; i += kTileThreads) atomicAdd(&dw1[i / 27 * (kCin * 9) + i % 27], sred[i]);
  if (threadIdx.x < kC) atomicAdd(&db1[threadIdx.x], sred[kC * 3 * 9 + threadIdx.x]);
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// CTAs of a tile kernel: at most per_sm resident ones per SM, each taking tiles in turn
int tile_ctas(int batch, int w, int h, int tw, int th, int per_sm) {
  const long long tiles = tile_grid(batch, w, h, tw, th).count, cap = static_cast<long long>(per_sm) * sm_count();
  return static_cast<int>(tiles < cap ? tiles : cap);
}

}  // namespace

int param_count() { return kParams; }

size_t workspace_bytes(int batch, int width, int height) {
  const size_t n = static_cast<size_t>(batch) * width * height;
  // A1, A2, A3 (32 x BF16), dA x 2 (32 x BF16)
  return n * (3 * 64 + 2 * 64) + 4096;
}

static void carve(unsigned char* ws, size_t n, __nv_bfloat16** A1, __nv_bfloat16** A2, __nv_bfloat16** A3,
                  __nv_bfloat16** G1, __nv_bfloat16** G2) {
  size_t o = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = ws + o;
    o += (bytes + 255) & ~static_cast<size_t>(255);
    return reinterpret_cast<__nv_bfloat16*>(p);
  };
  *A1 = take(n * 64);
  *A2 = take(n * 64);
  *A3 = take(n * 64);
  *G1 = take(n * 64);
  *G2 = take(n * 64);
}

cudaError_t pack_weights(const float* params, __nv_bfloat16* packed, cudaStream_t s) {
  cudaError_t e = launch_pack_w32(params + kOffW2, packed, 0, s);
  if (e == cudaSuccess) e = launch_pack_w32(params + kOffW3, packed + 9 * kC * kC, 0, s);
  if (e == cudaSuccess) e = launch_pack_w32(params + kOffW2, packed + 2 * 9 * kC * kC, 1, s);
  if (e == cudaSuccess) e = launch_pack_w32(params + kOffW3, packed + 3 * 9 * kC * kC, 1, s);
  return e;
}

cudaError_t forward(const float* params, const __nv_bfloat16* packed, const float* depth, const float* fallback,
                    float* out, int batch, int width, int height, unsigned char* ws, unsigned int* error,
                    cudaStream_t s) {
  const size_t n = static_cast<size_t>(batch) * width * height;
  if (n > 0x7fffffffULL) return cudaErrorInvalidValue;  // the layers' pixel arithmetic is 32-bit
  __nv_bfloat16 *A1, *A2, *A3, *G1, *G2;
  carve(ws, n, &A1, &A2, &A3, &G1, &G2);
  conv_in_kernel<<<tile_ctas(batch, width, height, kTileW, kTileH, 2), kTileThreads, 0, s>>>(depth, params, A1, batch, width,
                                                                                          height);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_conv32(A1, packed, params + kOffB2, nullptr, A2, batch, width, height, kForward, 1, error, s);
  if (e == cudaSuccess) {
    e = launch_conv32(A2, packed + 9 * kC * kC, params + kOffB3, nullptr, A3, batch, width, height, kForward, 1, error, s);
  }
  if (e != cudaSuccess) return e;
  e = allow_shared(conv_out_kernel, kOutSmem);
  if (e != cudaSuccess) return e;
  conv_out_kernel<<<tile_ctas(batch, width, height, kOutW, kOutH, kOutCtas), kTileThreads, kOutSmem, s>>>(
      A3, params, depth, fallback, out, batch, width, height);
  return cudaGetLastError();
}

cudaError_t backward(const float* params, const __nv_bfloat16* packed, const float* depth, const float* target,
                     const float* out, int batch, int width, int height, unsigned char* ws, float* grads, float* loss,
                     unsigned int* error, cudaStream_t s) {
  const size_t n = static_cast<size_t>(batch) * width * height;
  __nv_bfloat16 *A1, *A2, *A3, *G1, *G2;
  carve(ws, n, &A1, &A2, &A3, &G1, &G2);
  cudaError_t e = cudaMemsetAsync(grads, 0, kParams * sizeof(float), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(loss, 0, 2 * sizeof(float), s);
  // the loss, layer 4's weights and the gradient into A3
  if (e == cudaSuccess) e = allow_shared(out_backward_kernel, kOutBackSmem);
  if (e != cudaSuccess) return e;
  out_backward_kernel<<<tile_ctas(batch, width, height, kTileW, kTileH, 2), kTileThreads, kOutBackSmem, s>>>(
      A3, params, depth, target, out, G1, grads + kOffW4, grads + kOffB4, loss, batch, width, height);
  // layer 3
  e = cudaGetLastError();
  if (e == cudaSuccess) e = launch_wgrad32(A2, G1, grads + kOffW3, grads + kOffB3, batch, width, height, error, s);
  if (e == cudaSuccess) {
    e = launch_conv32(G1, packed + 3 * 9 * kC * kC, nullptr, A2, G2, batch, width, height, kGrad, 0, error, s);
  }
  if (e != cudaSuccess) return e;
  // layer 2
  e = launch_wgrad32(A1, G2, grads + kOffW2, grads + kOffB2, batch, width, height, error, s);
  if (e == cudaSuccess) {
    e = launch_conv32(G2, packed + 2 * 9 * kC * kC, nullptr, A1, G1, batch, width, height, kGrad, 0, error, s);
  }
  if (e != cudaSuccess) return e;
  // layer 1
  wgrad_in_kernel<<<tile_ctas(batch, width, height, kTileW, kWgInH, 2), kTileThreads, 0, s>>>(
      depth, G1, grads + kOffW1, grads + kOffB1, batch, width, height);
  return cudaGetLastError();
}

cudaError_t adam(float* params, const float* grads, float* m, float* v, float lr, float b1, float b2, float eps,
                 int step, cudaStream_t s) {
  const float c1 = 1.0f - powf(b1, static_cast<float>(step)), c2 = 1.0f - powf(b2, static_cast<float>(step));
  adam_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(params, grads, m, v, kParams, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

}  // namespace nn
}  // namespace vh
