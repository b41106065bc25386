// vh_misc.cu -- pool-wide maintenance kernels: observed-voxel recount and export to the reference layout.
#include "vh_common.cuh"
#include "vh_kernels.h"

namespace vh {
namespace {

// countObservedVoxelsKernel (src/cuda_tsdf_integrator.cu:905-930) with a warp reduction and one atomic per
// warp; the integrate kernel maintains the same number incrementally, this pass re-derives it from the pool.
__global__ void __launch_bounds__(256) recount_kernel(const Volume V, unsigned long long* __restrict__ out) {
  const uint32_t nblocks = min(V.counters->num_blocks, V.max_blocks);
  const size_t nvox = static_cast<size_t>(nblocks) * kBlockVoxels;
  unsigned long long local = 0ULL;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < nvox;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t b = static_cast<uint32_t>(i / kBlockVoxels);
    const int li = static_cast<int>(i % kBlockVoxels);
    bool obs = false;
    for (int d = 0; d < kDirs && !obs; ++d) obs = bin_observed(V, b, d, li);
    local += obs ? 1ULL : 0ULL;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffU, local, o);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(out, local);
}

// Blocks (list[i], or first + i without a list) in the reference Voxel layout voxels[i][li][d][l], transposed from the
// pool's direction-major one through shared memory: a CTA takes 64 voxels of a block, reads each direction's bins as
// one run (3 KB of FP32 layers, 2 KB of FP16 bins, each decoded once) and writes the 18 KB of records as one run.
// A direction that no layer was ever stored in (its bit of dir_mask) is zeros without a read.
// Bound by HBM: with one thread per output record, which read 48-byte pieces and decoded an FP16 bin three times,
// 1,024 blocks took 60 us (FP32) and 95 us (FP16).
constexpr int kExportVoxels = 64, kExportThreads = kExportVoxels * kDirs;
constexpr int kExportPitch = kDirs * kLayers + 1;  // records of a voxel, padded: conflict-free 16-byte accesses

template <bool kFp16>
__global__ void __launch_bounds__(kExportThreads) export_kernel(const Volume V, const uint32_t* __restrict__ list,
                                                                uint32_t first, float4* __restrict__ voxels) {
  __shared__ float4 S[kExportVoxels * kExportPitch];
  constexpr uint32_t kParts = kBlockVoxels / kExportVoxels;
  constexpr int kRecords = kExportVoxels * kDirs * kLayers;
  const int tid = threadIdx.x;
  const uint32_t i = blockIdx.x / kParts;
  const int li0 = static_cast<int>(blockIdx.x % kParts) * kExportVoxels;
  const uint32_t b = list ? list[i] : first + i;
  const uint32_t dirs = V.dir_mask[b];
  if (kFp16) {  // one bin per thread
    const int d = tid / kExportVoxels, v = tid % kExportVoxels;
    float4* o = S + v * kExportPitch + d * kLayers;
    if ((dirs >> d) & 1U) {  // uniform in the warp
      const uint4* q = V.layers16 + bin16_index(b, d, li0 + v);
      const uint4 A = q[0], B = q[1];
      decode_bin16(A, B, voxel_centre(V.block_keys[b], li0 + v, V.voxel_size), d, V.voxel_size, o[0], o[1], o[2]);
    } else {
      o[0] = o[1] = o[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  } else {  // three records per thread
#pragma unroll
    for (int k = 0; k < kLayers; ++k) {
      const int r = k * kExportThreads + tid;
      const int d = r / (kExportVoxels * kLayers), vl = r % (kExportVoxels * kLayers);
      S[(vl / kLayers) * kExportPitch + d * kLayers + vl % kLayers] =
          (dirs >> d) & 1U ? V.layers[layer_index(b, d, li0, 0) + vl] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
  __syncthreads();
  float4* out = voxels + (static_cast<size_t>(i) * kBlockVoxels + li0) * (kDirs * kLayers);
#pragma unroll
  for (int k = 0; k < kRecords / kExportThreads; ++k) {
    const int r = k * kExportThreads + tid;
    out[r] = S[(r / (kDirs * kLayers)) * kExportPitch + r % (kDirs * kLayers)];
  }
}

__global__ void __launch_bounds__(256) export_keys_kernel(const Volume V, const uint32_t* __restrict__ list,
                                                          uint32_t first, uint32_t count, int* __restrict__ keys) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const int4 k = V.block_keys[list ? list[i] : first + i];
    keys[3 * i] = k.x;
    keys[3 * i + 1] = k.y;
    keys[3 * i + 2] = k.z;
  }
}

// Zeros into the directions of blocks [0, count) that layers were stored in (dir_mask; the others are zeros already):
// one CTA per block, the next block's mask in flight.  Bound by HBM writes: a surface block has one to three directions of
// six, and the blocks around it that the neighbourhood rule allocates mostly none, so clearing whole blocks wrote several
// times as much.  With the same test in export_kernel, a volume reset, fused from 7 room frames of 640x480 and exported
// (plain form) takes 11.04 instead of 11.56 ms, from 15 orbit frames of 320x240 5.75 instead of 6.13.
__global__ void __launch_bounds__(256) clear_blocks_kernel(const Volume V, uint32_t count, uint4* __restrict__ pool,
                                                           uint32_t dir_words) {
  uint32_t dirs = blockIdx.x < count ? V.dir_mask[blockIdx.x] : 0U;
  for (uint32_t b = blockIdx.x; b < count; b += gridDim.x) {
    const uint32_t next = b + gridDim.x < count ? V.dir_mask[b + gridDim.x] : 0U;
    for (int d = 0; d < kDirs; ++d) {
      if (!((dirs >> d) & 1U)) continue;
      uint4* p = pool + (static_cast<size_t>(b) * kDirs + d) * dir_words;
      for (uint32_t w = threadIdx.x; w < dir_words; w += blockDim.x) p[w] = make_uint4(0U, 0U, 0U, 0U);
    }
    dirs = next;
  }
}

}  // namespace

cudaError_t launch_clear_blocks(const Volume& V, uint32_t count, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  uint4* pool = V.layers16 != nullptr ? V.layers16 : reinterpret_cast<uint4*>(V.layers);
  const uint32_t dir_words = kBlockVoxels * (V.layers16 != nullptr ? kBinWords16 : kLayers);
  const uint32_t grid = count < 152U * 8U ? count : 152U * 8U;
  clear_blocks_kernel<<<grid, 256, 0, s>>>(V, count, pool, dir_words);
  return cudaGetLastError();
}

cudaError_t launch_recount(const Volume& V, unsigned long long* out, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  recount_kernel<<<152 * 8, 256, 0, s>>>(V, out);
  return cudaGetLastError();
}

cudaError_t launch_export(const Volume& V, const uint32_t* list, uint32_t first, uint32_t count, int* keys,
                          float4* voxels, cudaStream_t s) {
  if (count == 0) return cudaSuccess;
  if (keys) export_keys_kernel<<<(count + 255) / 256, 256, 0, s>>>(V, list, first, count, keys);
  if (voxels) {
    const uint32_t grid = count * static_cast<uint32_t>(kBlockVoxels / kExportVoxels);  // count <= 2^23
    if (V.layers16 != nullptr) {
      export_kernel<true><<<grid, kExportThreads, 0, s>>>(V, list, first, voxels);
    } else {
      export_kernel<false><<<grid, kExportThreads, 0, s>>>(V, list, first, voxels);
    }
  }
  return cudaGetLastError();
}

}  // namespace vh

namespace vh {
namespace {

__device__ __forceinline__ bool any_word(const float4& L) {
  return (__float_as_uint(L.x) | __float_as_uint(L.y) | __float_as_uint(L.z) | __float_as_uint(L.w)) != 0U;
}

// Insert (or find) each imported key; idx[i] receives its pool block (kInvalidBlock when the pool is full).
__global__ void import_keys_kernel(const Volume V, const int* __restrict__ keys, uint32_t n, uint32_t* __restrict__ idx) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int x = keys[3 * i], y = keys[3 * i + 1], z = keys[3 * i + 2];
    unsigned long long key;
    idx[i] = kInvalidBlock;
    if (!pack_block_key(x, y, z, key)) {
      atomicOr(&V.counters->error, kErrKeyRange);
      continue;
    }
    uint32_t slot = hash_block_key(x, y, z) & V.mask;
    bool done = false;
    for (uint32_t probe = 0; probe < V.capacity && !done; ++probe) {
      unsigned long long cur = atomicCAS(&V.slot_keys[slot], kEmptyKey, key);
      if (cur == kEmptyKey) {
        uint32_t b = atomicAdd(&V.counters->num_blocks, 1U);
        if (b >= V.max_blocks) {
          atomicOr(&V.counters->error, kErrPoolFull);
          b = kInvalidBlock;
        } else {
          V.block_keys[b] = make_int4(x, y, z, 0);
        }
        V.slot_block[slot] = b;
        idx[i] = b;
        done = true;
      } else if (cur == key) {
        idx[i] = V.slot_block[slot];
        done = true;
      } else {
        slot = (slot + 1U) & V.mask;
      }
    }
    if (!done) atomicOr(&V.counters->error, kErrHashFull);
  }
}

// reference Voxel layout [i][li][d][l] -> pool (direction-major); rebuilds the observed mask, and flags the directions
// that hold any word (a caller's record without weight too)
__global__ void __launch_bounds__(256) import_voxels_kernel(const Volume V, const float4* __restrict__ voxels,
                                                            uint32_t n, const uint32_t* __restrict__ idx) {
  for (size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; t < static_cast<size_t>(n) * kBlockVoxels;
       t += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t i = static_cast<uint32_t>(t / kBlockVoxels);
    const int li = static_cast<int>(t % kBlockVoxels);
    const uint32_t b = idx[i];
    bool obs = false;
    uint32_t dirs = 0U;
    if (b != kInvalidBlock) {
      const float4* src = voxels + t * kDirs * kLayers;
      const int4 bk = V.block_keys[b];
      for (int d = 0; d < kDirs; ++d) {
        const float4 L0 = src[d * kLayers], L1 = src[d * kLayers + 1], L2 = src[d * kLayers + 2];
        store_bin(V, b, d, li, bk, V.voxel_size, L0, L1, L2);
        if (L0.x > 0.0f || L1.x > 0.0f || L2.x > 0.0f) obs = true;
        if (any_word(L0) || any_word(L1) || any_word(L2)) dirs |= 1U << d;
      }
    }
    const unsigned ballot = __ballot_sync(__activemask(), obs);
    if (b != kInvalidBlock) {
      if ((li & 31) == 0) V.obs_mask[static_cast<size_t>(b) * (kBlockVoxels / 32) + (li >> 5)] = ballot;
      if (dirs) atomicOr(&V.dir_mask[b], dirs);
    }
  }
}

}  // namespace

cudaError_t launch_import_keys(const Volume& V, const int* keys, uint32_t n, uint32_t* idx, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  import_keys_kernel<<<(n + 255) / 256, 256, 0, s>>>(V, keys, n, idx);
  return cudaGetLastError();
}

cudaError_t launch_import(const Volume& V, const int* keys, const float4* voxels, uint32_t n, uint32_t* idx,
                          cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  import_keys_kernel<<<(n + 255) / 256, 256, 0, s>>>(V, keys, n, idx);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  import_voxels_kernel<<<152 * 8, 256, 0, s>>>(V, voxels, n, idx);
  return cudaGetLastError();
}

}  // namespace vh
