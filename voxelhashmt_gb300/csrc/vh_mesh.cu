// vh_mesh.cu -- directional multi-layer marching cubes: near cells, their counts, a scan, their triangles.
//
// Reference: extractMeshCuda (src/cuda_mesh_extractor.cu:636-720) rebuilds a host lookup table per call and
// runs count + extract kernels once per direction (12 launches, 12 syncs, 6 readbacks); every cell copies
// its 8 corner voxels whole (288 B each) through a device hash lookup, twice.  Here:
//   1. prepare_kernel: each block's 7 (+x, +y, +z) neighbours through the persistent hash, cleared masks;
//   2. near_kernel: every observed voxel's planes, read once as the pool stores them, mark the cells of their
//      direction whose centre they pass near enough to produce triangles (a bit per cell; a plane marks up to 8 cells,
//      some of them in a neighbour block);
//   3. cells_kernel, counting: one thread per marked cell evaluates it from the corner voxels' bins; its count;
//   4. rounds_kernel, scan_kernel: the direction totals, and the block offsets;
//   5. cells_kernel, emitting: the cells that have triangles again, each writing them at its offset.
// The output is deterministic (block, direction, cell, cluster, table order).
//
// One cell in ten or so has a plane near its centre.  Staging every direction of every block in shared memory and
// evaluating all its 512 cells ran on 9-21 of 32 threads, with the CTA waiting at its barriers for the few warps with
// work; marking first fills the warps: 9 cells in 10 are never looked at, and a warp takes 32 marked cells.  A room of
// 26,000 FP32 blocks: 9.2 -> 2.7 ms, a tenth of it in near_kernel (3.6 TB/s), the rest in cells_kernel, which is bound
// by instruction issue (62 % of the slots, 17 of 32 threads active).
//
// Per cell the arithmetic is the reference's collectSurfaceClusters / loadCubeForSurface /
// completeCubeValuesWithFallbackGpu / emitCubeTriangles (:259-551) in the same operation order.
#include "vh_common.cuh"
#include "vh_kernels.h"

#define VH_MC_TABLE_QUALIFIER static __constant__
#include "vh_mc_tables.h"

namespace vh {
namespace {

constexpr int kCorners = 8;
constexpr int kMaxCand = kCorners * kLayers;  // cuda_mesh_extractor.cu:18
constexpr int kMaskWords = kBlockVoxels / 32;  // cell mask of one (block, direction)

__constant__ int c_corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                   {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
__constant__ int c_edge_corners[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                          {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};

// planeSignedDistanceGpu (:259-262)
__device__ __forceinline__ float plane_sd(const float4& pl, f3 p) {
  return pl.x * p.x + pl.y * p.y + pl.z * p.z - pl.w;
}

// interpolateVertexGpu (:358-374)
__device__ __forceinline__ f3 interp(f3 p0, f3 p1, float v0, float v1, float iso) {
  const float delta = v1 - v0;
  if (fabsf(delta) < 1e-6f) return p0;
  const float t = fminf(1.0f, fmaxf(0.0f, (iso - v0) / delta));
  return mk3(p0.x + (p1.x - p0.x) * t, p0.y + (p1.y - p0.y) * t, p0.z + (p1.z - p0.z) * t);
}

// corner k of the cell at grid (gx, gy, gz): ((g + corner) + 0.5) * vs per axis (loadCubeForSurface, :276-303)
__device__ __forceinline__ f3 corner_pos(int gx, int gy, int gz, int k, float vs) {
  return mk3((static_cast<float>(gx + c_corner[k][0]) + 0.5f) * vs, (static_cast<float>(gy + c_corner[k][1]) + 0.5f) * vs,
             (static_cast<float>(gz + c_corner[k][2]) + 0.5f) * vs);
}

// A bin as the pool stores it, in flight while the one before it is used, and layer l of it as an FP32 record (the
// voxel at grid (gx, gy, gz): the FP16 codec's centre).
template <bool kFp16>
struct RawBin;
template <>
struct RawBin<false> {
  float4 L[kLayers];
  __device__ __forceinline__ void clear() { L[0] = L[1] = L[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
  __device__ __forceinline__ void load(const Volume& V, uint32_t b, int d, int li) {
    const float4* q = V.layers + layer_index(b, d, li, 0);
#pragma unroll
    for (int l = 0; l < kLayers; ++l) L[l] = q[l];
  }
  __device__ __forceinline__ bool any() const { return L[0].x > 0.0f || L[1].x > 0.0f || L[2].x > 0.0f; }
  __device__ __forceinline__ float4 layer(int l, int, int, int, int, float) const {
    return l == 0 ? L[0] : (l == 1 ? L[1] : L[2]);
  }
};
template <>
struct RawBin<true> {
  uint4 A, B;
  __device__ __forceinline__ void clear() { A = B = make_uint4(0U, 0U, 0U, 0U); }
  __device__ __forceinline__ void load(const Volume& V, uint32_t b, int d, int li) {
    const uint4* q = V.layers16 + bin16_index(b, d, li);
    A = q[0];
    B = q[1];
  }
  __device__ __forceinline__ bool any() const { return (A.x & 0xffffU) || (A.y >> 16) || (A.w & 0xffffU); }
  __device__ __forceinline__ float4 layer(int l, int d, int gx, int gy, int gz, float vs) const {
    const uint32_t w = l == 0 ? A.x & 0xffffU : (l == 1 ? A.y >> 16 : A.w & 0xffffU);
    if (w == 0U) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const uint32_t sc = l == 0 ? A.x >> 16 : (l == 1 ? A.z & 0xffffU : A.w >> 16);
    const uint32_t po = l == 0 ? A.y & 0xffffU : (l == 1 ? A.z >> 16 : B.x & 0xffffU);
    const uint32_t nk = l == 0 ? B.y : (l == 1 ? B.z : B.w);
    const f3 c = voxel_centre(make_int4(gx >> 3, gy >> 3, gz >> 3, 0),
                              (gx & 7) + kBlockSide * ((gy & 7) + kBlockSide * (gz & 7)), vs);
    return decode_layer16(w, sc, po, nk, bin_normal(nk), c, axis_coordinate(c, d), vs);
  }
};

__device__ __forceinline__ uint32_t block_count(const Volume& V) { return min(V.counters->num_blocks, V.max_blocks); }

// 1. every block's cell masks (and, with a list, direction totals) cleared; neighbours[8 b + k] = the block at +(k & 1, k >> 1 & 1,
// k >> 2).  With a list (incremental meshing), only for its blocks, and they and their neighbours get need[] = epoch:
// the blocks whose voxels may be corners of a listed block's cells.
__global__ void __launch_bounds__(256) prepare_kernel(const Volume V, const MeshBuffers M, const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ list_count, uint32_t epoch) {
  const uint32_t n = block_count(V);
  const uint32_t items = list ? *list_count : n;
  const size_t t0 = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  if (t0 < 4) M.queue[t0] = 0U;
  uint4* masks = reinterpret_cast<uint4*>(M.cell_mask);
  for (size_t i = t0; i < static_cast<size_t>(n) * (kDirs * kMaskWords / 4); i += stride) {
    masks[i] = make_uint4(0U, 0U, 0U, 0U);
  }
  for (size_t i = t0; list && i < static_cast<size_t>(n) * kDirs; i += stride) M.dir_totals[i] = 0U;
  for (size_t i = t0; i < static_cast<size_t>(items) * 8; i += stride) {
    const uint32_t b = list ? list[i >> 3] : static_cast<uint32_t>(i >> 3);
    const int k = static_cast<int>(i & 7);
    const int4 bk = V.block_keys[b];
    const uint32_t nb = k == 0 ? b : lookup_block(V, bk.x + (k & 1), bk.y + ((k >> 1) & 1), bk.z + (k >> 2));
    M.neighbours[static_cast<size_t>(b) * 8 + k] = nb;
    if (list && nb != kInvalidBlock) M.need[nb] = epoch;
  }
}

// Distance from iso of a plane at a cell centre beyond which the cell has no triangles: every corner value of a cell
// is a candidate's plane evaluated at a corner, at most sqrt(3)/2 voxel from the centre (plus a rounding margin for
// the two float evaluations); means of same-sign values keep the sign.
__device__ __forceinline__ float reject_distance(float vs, f3 cc) {
  return 0.8660254f * vs * 1.00001f + 1e-5f * (1.0f + fabsf(cc.x) + fabsf(cc.y) + fabsf(cc.z));
}

// 2. One warp per 8 x 4 voxels (a word of the observed mask) of a block, no barriers.  A layer's plane at the 8 cell
// centres around its voxel is its distance at the voxel's centre +- half a voxel along each axis; the cells within the
// reject distance (with a margin for this form of the sum: marking too many cells is harmless) are marked, a few words
// per warp and direction.  The bins of the flagged directions are read once, the next direction's while this one's are
// used.
constexpr int kNearThreads = 256;

template <bool kFp16>
__global__ void __launch_bounds__(kNearThreads) near_kernel(const Volume V, const Params p, const MeshBuffers M,
                                                            bool selected, uint32_t epoch) {
  const int lane = threadIdx.x & 31;
  const float vs = p.voxel_size, half = 0.5f * vs;
  const uint32_t items = block_count(V) * kMaskWords;
  for (uint32_t item = blockIdx.x * (kNearThreads / 32) + (threadIdx.x >> 5); item < items;
       item += gridDim.x * (kNearThreads / 32)) {
    const uint32_t b = item / kMaskWords;
    const int word = static_cast<int>(item % kMaskWords), li = word * 32 + lane;
    if (selected && M.need[b] != epoch) continue;  // uniform in the warp, as are the tests below
    uint32_t dirs = V.dir_mask[b];
    const uint32_t observed = V.obs_mask[static_cast<size_t>(b) * kMaskWords + word];
    if (!dirs || !observed) continue;
    const int4 bk = V.block_keys[b];
    const bool mine = (observed >> lane) & 1U;
    int d = __ffs(dirs) - 1;
    RawBin<kFp16> next;
    next.clear();
    if (mine) next.load(V, b, d, li);
    // lane k: the block at -(k & 1, k >> 1 & 1, k >> 2)
    uint32_t down = b;
    if (lane > 0 && lane < 8) down = lookup_block(V, bk.x - (lane & 1), bk.y - ((lane >> 1) & 1), bk.z - (lane >> 2));
    const int gx = bk.x * kBlockSide + (lane & 7), gy = bk.y * kBlockSide + ((li >> 3) & 7),
              gz = bk.z * kBlockSide + (word >> 1);
    const f3 vc = mk3((static_cast<float>(gx) + 0.5f) * vs, (static_cast<float>(gy) + 0.5f) * vs,
                      (static_cast<float>(gz) + 0.5f) * vs);
    const float reach = 0.8660254f * vs * 1.0001f + 4e-5f * (1.0f + vs + fabsf(vc.x) + fabsf(vc.y) + fabsf(vc.z));
    while (dirs) {
      const RawBin<kFp16> bin = next;
      const int dir = d;
      dirs &= dirs - 1U;
      if (dirs) {
        d = __ffs(dirs) - 1;
        if (mine) next.load(V, b, d, li);
      }
      if (!__any_sync(0xffffffffU, bin.any())) continue;
      uint32_t near = 0U;  // bit k: the cell whose corner (k & 1, k >> 1 & 1, k >> 2) this voxel is
#pragma unroll 1
      for (int l = 0; l < kLayers; ++l) {
        const float4 L = bin.layer(l, dir, gx, gy, gz, vs);
        if (!(L.x > 0.0f)) continue;
        const f3 m = unpack_normal_mesh(__float_as_uint(L.w));
        const float s = plane_sd(make_float4(m.x, m.y, m.z, L.z), vc) - p.iso;
        const float a = m.x * half, c = m.y * half, e = m.z * half;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float t = s + ((k & 1) ? -a : a) + ((k & 2) ? -c : c) + ((k & 4) ? -e : e);
          if (fabsf(t) <= reach) near |= 1U << k;
        }
      }
      if (!__any_sync(0xffffffffU, near != 0U)) continue;
      uint32_t w = 0U;  // lane k (and k + 8, ...): the voxels of this warp that mark through corner k
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t ballot = __ballot_sync(0xffffffffU, (near >> k) & 1U);
        if ((lane & 7) == k) w = ballot;
      }
      // The marked cells are one step down along each axis of corner k.  Along x, column 0 goes to column 7 of the -x
      // block; along y, row 0 of the word to row 3 of the word before (the -y block's last for the lower word).
      // Quantity j = lane >> 3: bit 0 the word before, bit 1 the -x block.  Corners of the same z step (lanes k and
      // k ^ 1, k ^ 2, k ^ 3) mark the same words.
      const bool kx = lane & 1, ky = lane & 2, before = lane & 8, out = lane & 16;
      uint32_t v = out ? (kx ? (w & 0x01010101U) << 7 : 0U) : (kx ? (w & 0xfefefefeU) >> 1 : w);
      v = before ? (ky ? (v & 0xffU) << 24 : 0U) : (ky ? v >> 8 : v);
      v |= __shfl_xor_sync(0xffffffffU, v, 1);
      v |= __shfl_xor_sync(0xffffffffU, v, 2);
      const int z = (word >> 1) - ((lane >> 2) & 1), yq = word & 1;
      const int nb = (z < 0 ? 4 : 0) | (before && !yq ? 2 : 0) | (out ? 1 : 0);
      const uint32_t to = __shfl_sync(0xffffffffU, down, nb);
      if ((lane & 3) == 0 && v && to != kInvalidBlock) {
        atomicOr(&M.cell_mask[(static_cast<size_t>(to) * kDirs + dir) * kMaskWords + (z & 7) * 2 + (before ? yq ^ 1 : yq)],
                 v);
      }
    }
  }
}

// The rounds of 32 marked cells of every (block, direction), 16 bd + r, appended to M.rounds in no particular order, so
// that the cells kernel's warps share them evenly (a flat surface gives one (block, direction) a dozen rounds and the
// next none; by (block, direction), the longest held up the kernel: 319 instead of 85 us for 2,000 blocks).  kCounted:
// after the count, the cells without triangles leave the mask first, and the direction's total is written.
constexpr int kRoundThreads = 256;

template <bool kCounted>
__global__ void __launch_bounds__(kRoundThreads) rounds_kernel(const Volume V, const MeshBuffers M,
                                                               const uint32_t* __restrict__ list,
                                                               const uint32_t* __restrict__ list_count) {
  constexpr int kWarps = kRoundThreads / 32;
  __shared__ uint32_t s_rounds[kWarps], s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t items = (list ? *list_count : block_count(V)) * kDirs;
  for (uint32_t i0 = blockIdx.x * kWarps; i0 < items; i0 += gridDim.x * kWarps) {
    const uint32_t item = i0 + warp;
    uint32_t cells = 0U, code = 0U;
    if (item < items) {  // uniform in the warp
      const size_t bd = static_cast<size_t>(list ? list[item / kDirs] : item / kDirs) * kDirs + item % kDirs;
      code = static_cast<uint32_t>(bd) * 16U;
      uint32_t* mask = M.cell_mask + bd * kMaskWords;
      const uint32_t word = lane < kMaskWords ? mask[lane] : 0U;
      cells = __reduce_add_sync(0xffffffffU, __popc(word));
      if (kCounted) {
        uint32_t sum = 0U;
        if (cells) {
          // 16 cells per lane
          uint32_t bits = (__shfl_sync(0xffffffffU, word, lane >> 1) >> (16 * (lane & 1))) & 0xffffU;
          if (bits) {
            const uint4 c4 = *reinterpret_cast<const uint4*>(M.cell_counts + bd * kBlockVoxels + 16 * lane);
            const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const uint32_t n = (bits >> j) & 1U ? (c[j >> 2] >> (8 * (j & 3))) & 0xffU : 0U;
              sum += n;
              if (n == 0U) bits &= ~(1U << j);
            }
          }
          sum = __reduce_add_sync(0xffffffffU, sum);
          cells = __reduce_add_sync(0xffffffffU, __popc(bits));
          const uint32_t high = __shfl_down_sync(0xffffffffU, bits, 1);
          if (!(lane & 1)) mask[lane >> 1] = bits | (high << 16);
        }
        if (lane == 0) M.dir_totals[bd] = sum;
      }
    }
    const uint32_t rounds = (cells + 31U) / 32U;
    if (lane == 0) s_rounds[warp] = rounds;
    __syncthreads();
    uint32_t before = 0U, all = 0U;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) before += s_rounds[w];
      all += s_rounds[w];
    }
    if (threadIdx.x == 0 && all) s_base = atomicAdd(&M.queue[kCounted ? 1 : 0], all);
    __syncthreads();
    if (static_cast<uint32_t>(lane) < rounds) M.rounds[s_base + before + lane] = code + static_cast<uint32_t>(lane);
    __syncthreads();
  }
}

// 3 and 5. One warp per round of 32 marked cells from a device work queue, one thread per cell.  A thread's
// candidate distances and corner values live in its column of shared memory; every loop over candidates is rolled:
// with the corners unrolled (70 KB of code instead of 16) the same instructions took twice as long, waiting to be
// fetched.
constexpr int kCellThreads = 128;

struct CellShared {
  float centre[kMaxCand][kCellThreads];  // candidate i = 3 corner + layer: its plane at the cell centre
  float corner[kMaxCand][kCellThreads];  // at its corner
  float key[kMaxCand][kCellThreads];     // sorted candidate keys, then cluster centres
  float val[kCorners][kCellThreads];     // a cluster's corner values
  uint8_t ntri[256];
  int8_t tri[256][16];  // emitting only
};
constexpr size_t kCountSmem = offsetof(CellShared, tri), kEmitSmem = sizeof(CellShared);

// the 3 corners that share an edge with corner k, in the order of the edges
__constant__ int c_adjacent[8][3] = {{1, 3, 4}, {0, 2, 5}, {1, 3, 6}, {2, 0, 7},
                                     {5, 7, 0}, {4, 6, 1}, {5, 7, 2}, {6, 4, 3}};

// One cell (grid position gx, gy, gz; local lx, ly, lz) of direction d: returns its triangle count; with kEmit writes
// them to out (9 floats each).  nbr: lane k holds the block at corner offset k of the warp's block.
template <bool kEmit, bool kFp16>
__device__ __forceinline__ int process_cell(CellShared& S, const Volume& V, const Params& p, int d, uint32_t nbr, bool live,
                                            int gx, int gy, int gz, int lx, int ly, int lz, int t,
                                            float* __restrict__ out) {
  const float vs = p.voxel_size;
  const f3 cc = mk3((static_cast<float>(gx) + 1.0f) * vs, (static_cast<float>(gy) + 1.0f) * vs,
                    (static_cast<float>(gz) + 1.0f) * vs);
  // collectSurfaceClusters (:439-507): the corners' layers; the next corner's bin is loaded while this one's is used
  uint32_t valid = 0U;
  int nc = 0;
  float nearest = 3.0e38f;  // smallest |candidate - iso|
  RawBin<kFp16> next;
  next.clear();
#pragma unroll 1
  for (int k = -1; k < kCorners; ++k) {
    const RawBin<kFp16> bin = next;
    if (k + 1 < kCorners) {
      const int x = lx + c_corner[k + 1][0], y = ly + c_corner[k + 1][1], z = lz + c_corner[k + 1][2];
      const uint32_t nb = __shfl_sync(0xffffffffU, nbr, (x >> 3) | ((y >> 3) << 1) | ((z >> 3) << 2));
      next.clear();
      if (live && nb != kInvalidBlock) next.load(V, nb, d, (x & 7) + kBlockSide * ((y & 7) + kBlockSide * (z & 7)));
    }
    if (k < 0 || !bin.any()) continue;
    const f3 cp = corner_pos(gx, gy, gz, k, vs);
#pragma unroll 1
    for (int l = 0; l < kLayers; ++l) {
      const float4 L = bin.layer(l, d, gx + c_corner[k][0], gy + c_corner[k][1], gz + c_corner[k][2], vs);
      if (!(L.x > 0.0f)) continue;
      const f3 n = unpack_normal_mesh(__float_as_uint(L.w));
      const float4 pl = make_float4(n.x, n.y, n.z, L.z);
      const float c = plane_sd(pl, cc);
      const int i = k * kLayers + l;
      S.centre[i][t] = c;
      S.corner[i][t] = plane_sd(pl, cp);
      S.key[nc][t] = c;
      nearest = fminf(nearest, fabsf(c - p.iso));
      valid |= 1U << i;
      ++nc;
    }
  }
  // Every corner value below is a candidate's plane evaluated at a corner: cells without a plane near their centre
  // have cube index 0 or 255 for every cluster, no triangles, and are skipped without changing the output.
  const float reject = reject_distance(vs, cc);
  if (nc == 0 || nearest > reject) return 0;
#pragma unroll 1
  for (int i = 1; i < nc; ++i) {  // insertion sort (:264-274)
    const float x = S.key[i][t];
    int j = i - 1;
    while (j >= 0 && S.key[j][t] > x) {
      S.key[j + 1][t] = S.key[j][t];
      --j;
    }
    S.key[j + 1][t] = x;
  }
  // greedy clustering with running means; centre c is written to slot c <= i after slot i has been read,
  // and only the last cluster's size is ever used
  const float tol = p.extract_tol;
  int ncl = 0;
  float last = 0.0f, last_size = 0.0f;
#pragma unroll 1
  for (int i = 0; i < nc; ++i) {
    const float key = S.key[i][t];
    if (ncl == 0 || fabsf(key - last) > tol) {
      last = key;
      last_size = 1.0f;
      ++ncl;
    } else {
      last = (last * last_size + key) / (last_size + 1.0f);
      last_size += 1.0f;
    }
    S.key[ncl - 1][t] = last;
  }

  // A cluster's corner values are planes within tol of its key at the cell centre, evaluated at most sqrt(3)/2
  // voxel away (and means of such values): a key farther than tol + that from iso (with the rounding margin)
  // gives cube index 0 or 255, no triangles.  Skipped without changing the output.
  const float cluster_reject = tol * 1.00001f + reject;
  int total = 0;
#pragma unroll 1
  for (int ci = 0; ci < ncl; ++ci) {
    const float key = S.key[ci][t];
    if (fabsf(key - p.iso) > cluster_reject) continue;
    // loadCubeForSurface + selectClosestLayerForSurfaceGpu (:276-303, :509-551)
    uint32_t mask = 0U;
    int cnt = 0;
    float sum = 0.0f;
#pragma unroll 1
    for (int k = 0; k < kCorners; ++k) {
      int best = -1;
      float best_delta = 1e30f;
#pragma unroll
      for (int l = 0; l < kLayers; ++l) {
        const int i = k * kLayers + l;
        if (!((valid >> i) & 1U)) continue;
        const float delta = fabsf(S.centre[i][t] - key);
        if (delta <= tol && delta < best_delta) {
          best_delta = delta;
          best = i;
        }
      }
      if (best >= 0) {
        const float v = S.corner[best][t];
        S.val[k][t] = v;
        mask |= 1U << k;
        ++cnt;
        sum += v;
      }
    }
    // completeCubeValuesWithFallbackGpu (:305-356)
    if (cnt < 6) continue;
    int cube = 0;
    if (mask != 0xffU) {
      const float global = sum / static_cast<float>(cnt);
#pragma unroll 1
      for (int k = 0; k < kCorners; ++k) {
        if (mask & (1U << k)) continue;
        float ns = 0.0f;
        int nn = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int nb = c_adjacent[k][j];
          if (!(mask & (1U << nb))) continue;
          ns += S.val[nb][t];
          ++nn;
        }
        S.val[k][t] = nn > 0 ? (ns / static_cast<float>(nn)) : global;
        mask |= 1U << k;
      }
    }
    // computeCubeIndex / countCubeTriangles / emitCubeTriangles (:376-437)
#pragma unroll
    for (int k = 0; k < kCorners; ++k)
      if (S.val[k][t] < p.iso) cube |= 1 << k;
    const int ntri = S.ntri[cube];
    if (kEmit) {
      float* o = out + static_cast<size_t>(total) * 9;
#pragma unroll 1
      for (int q = 0; q < 3 * ntri; ++q) {
        // the vertex on edge e (interpolateVertexGpu, :358-374), computed where it is used: the same
        // operations on the same values wherever an edge's vertex is needed
        const int e = S.tri[cube][q];
        const int c0 = c_edge_corners[e][0], c1 = c_edge_corners[e][1];
        const f3 v = interp(corner_pos(gx, gy, gz, c0, vs), corner_pos(gx, gy, gz, c1, vs), S.val[c0][t], S.val[c1][t],
                            p.iso);
        o[3 * q] = v.x;
        o[3 * q + 1] = v.y;
        o[3 * q + 2] = v.z;
      }
    }
    total += ntri;
  }
  return total;
}

// the t-th set bit (t < popc) of a (block, direction) mask whose word lane holds `word` and `before` bits precede it
__device__ __forceinline__ int nth_cell(uint32_t word, uint32_t before, uint32_t t) {
  int w = 0;
#pragma unroll
  for (int step = 8; step > 0; step >>= 1) {  // the last of the 16 words with at most t bits before it
    if (__shfl_sync(0xffffffffU, before, w + step) <= t) w += step;
  }
  uint32_t m = __shfl_sync(0xffffffffU, word, w);
  t -= __shfl_sync(0xffffffffU, before, w);
  int bit = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    const uint32_t low = __popc(m & ((1U << step) - 1U));
    if (t >= low) {
      t -= low;
      m >>= step;
      bit += step;
    }
  }
  return w * 32 + bit;
}

template <bool kEmit, bool kFp16>
__global__ void __launch_bounds__(kCellThreads, 5) cells_kernel(const Volume V, const Params p, const MeshBuffers M,
                                                                float* __restrict__ tris) {
  extern __shared__ __align__(16) unsigned char mc_smem[];
  CellShared& S = *reinterpret_cast<CellShared*>(mc_smem);
  const int t = threadIdx.x, lane = t & 31;
  for (int i = t; i < 256; i += kCellThreads) {
    int ntri = 0;
    if (vh_mc_edge_table[i] != 0) {
      while (ntri < 5 && vh_mc_tri_table[i][3 * ntri] >= 0) ++ntri;
    }
    S.ntri[i] = static_cast<uint8_t>(ntri);
  }
  if (kEmit) {
    for (int i = t; i < 256 * 16; i += kCellThreads) S.tri[i / 16][i % 16] = vh_mc_tri_table[i / 16][i % 16];
  }
  __syncthreads();
  const uint32_t items = M.queue[kEmit ? 1 : 0];
  uint32_t* queue = M.queue + (kEmit ? 3 : 2);
  uint32_t fetched = 0U;
  if (lane == 0) fetched = atomicAdd(queue, 1U);
  for (;;) {
    const uint32_t item = __shfl_sync(0xffffffffU, fetched, 0);
    if (item >= items) break;
    if (lane == 0) fetched = atomicAdd(queue, 1U);
    const uint32_t code = M.rounds[item];
    const uint32_t first = (code & 15U) * 32U;
    const size_t bd = code >> 4;
    const uint32_t b = static_cast<uint32_t>(bd) / kDirs;
    const int d = static_cast<int>(static_cast<uint32_t>(bd) - b * kDirs);
    const uint32_t word = lane < kMaskWords ? M.cell_mask[bd * kMaskWords + lane] : 0U;
    uint32_t before = __popc(word);
#pragma unroll
    for (int o = 1; o < kMaskWords; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffU, before, o);
      if (lane >= o) before += x;
    }
    const uint32_t cells = __shfl_sync(0xffffffffU, before, kMaskWords - 1);
    before -= __popc(word);
    const int4 bk = V.block_keys[b];
    uint32_t nbr = lane < 8 ? M.neighbours[static_cast<size_t>(b) * 8 + lane] : kInvalidBlock;
    if (nbr != kInvalidBlock && !((V.dir_mask[nbr] >> d) & 1U)) nbr = kInvalidBlock;  // no observed layer there
    uint8_t* counts = M.cell_counts + bd * kBlockVoxels;
    const bool live = first + lane < cells;
    const int c = nth_cell(word, before, min(first + lane, cells - 1U));
    const int lx = c & 7, ly = (c >> 3) & 7, lz = c >> 6;
    float* o = nullptr;
    if (kEmit) {
      // this round's first triangle: the block's, after those of its earlier directions and of the cells before
      uint32_t skip = lane < d ? M.dir_totals[static_cast<size_t>(b) * kDirs + lane] : 0U;
      if (first) {
        const int c0 = __shfl_sync(0xffffffffU, c, 0);
        uint32_t bits = (__shfl_sync(0xffffffffU, word, lane >> 1) >> (16 * (lane & 1))) & 0xffffU;
        const int below = min(max(c0 - 16 * lane, 0), 16);
        bits &= (1U << below) - 1U;
        if (bits) {
          const uint4 c4 = *reinterpret_cast<const uint4*>(counts + 16 * lane);
          const uint32_t w4[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
          for (int j = 0; j < 16; ++j) skip += (bits >> j) & 1U ? (w4[j >> 2] >> (8 * (j & 3))) & 0xffU : 0U;
        }
      }
      skip = __reduce_add_sync(0xffffffffU, skip);
      const uint32_t n = live ? counts[c] : 0U;
      uint32_t incl = n;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffU, incl, s);
        if (lane >= s) incl += x;
      }
      o = tris + (M.offsets[b] + skip + incl - n) * 9ULL;
    }
    const int n = process_cell<kEmit, kFp16>(S, V, p, d, nbr, live, bk.x * kBlockSide + lx, bk.y * kBlockSide + ly,
                                             bk.z * kBlockSide + lz, lx, ly, lz, t, o);
    if (!kEmit && live) counts[c] = static_cast<uint8_t>(n);  // one byte: at most 5 triangles x 24 clusters
  }
}

// pool blocks updated in frames (frame - frames, frame]: the subset of incremental meshing
__global__ void recent_blocks_kernel(const Volume V, uint32_t frames, uint32_t* __restrict__ list,
                                     uint32_t* __restrict__ count) {
  const uint32_t n = min(V.counters->num_blocks, V.max_blocks);
  const uint32_t frame = V.counters->frame;
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < n; b += gridDim.x * blockDim.x) {
    const uint32_t st = V.block_stamp[b];
    if (st != 0U && frame - st < frames) list[atomicAdd(count, 1U)] = b;
  }
}

// 4. exclusive scan of the block totals (the sums of their 6 direction totals) -> offsets, total; one CTA, 8 blocks per
// thread and pass
__global__ void __launch_bounds__(1024) scan_kernel(const Volume V, const MeshBuffers M,
                                                    unsigned long long* __restrict__ total) {
  constexpr uint32_t kPer = 8;
  __shared__ unsigned long long s_w[32];
  __shared__ unsigned long long s_carry;
  const uint32_t n = block_count(V);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_carry = 0ULL;
  __syncthreads();
  for (uint32_t start = 0; start < n; start += 1024U * kPer) {
    const uint32_t i0 = start + tid * kPer;
    uint32_t v[kPer];
    unsigned long long sum = 0ULL;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
      v[j] = 0U;
      if (i0 + j < n) {
        const uint2* q = reinterpret_cast<const uint2*>(M.dir_totals + static_cast<size_t>(i0 + j) * kDirs);
        const uint2 a = q[0], b = q[1], c = q[2];
        v[j] = a.x + a.y + b.x + b.y + c.x + c.y;
      }
      sum += v[j];
    }
    unsigned long long incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffU, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s_w[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const unsigned long long w = s_w[lane];
      unsigned long long wi = w;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffU, wi, o);
        if (lane >= o) wi += t;
      }
      s_w[lane] = wi - w;
    }
    __syncthreads();
    const unsigned long long carry = s_carry;
    unsigned long long at = carry + s_w[warp] + incl - sum;
#pragma unroll
    for (uint32_t j = 0; j < kPer; ++j) {
      if (i0 + j < n) M.offsets[i0 + j] = at;
      at += v[j];
    }
    __syncthreads();
    if (tid == 1023) s_carry = at;
    __syncthreads();
  }
  if (tid == 0) *total = s_carry;
}

template <bool kEmit, bool kFp16>
cudaError_t launch_cells(const Volume& V, const Params& p, const MeshBuffers& M, float* tris, cudaStream_t s) {
  constexpr size_t smem = kEmit ? kEmitSmem : kCountSmem;
  static int grid = 0;
  if (grid == 0) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const cudaError_t e = cudaFuncSetAttribute(cells_kernel<kEmit, kFp16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cells_kernel<kEmit, kFp16>, kCellThreads, smem);
    grid = (sms > 0 ? sms : 152) * (per_sm > 0 ? per_sm : 1);
  }
  cells_kernel<kEmit, kFp16><<<grid, kCellThreads, smem, s>>>(V, p, M, tris);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_mc_count(const Volume& V, const Params& p, const MeshBuffers& M, const uint32_t* list,
                            const uint32_t* list_count, uint32_t epoch, unsigned long long* total, cudaStream_t s) {
  prepare_kernel<<<152 * 8, 256, 0, s>>>(V, M, list, list_count, epoch);
  const bool fp16 = V.layers16 != nullptr;
  if (fp16) {
    near_kernel<true><<<152 * 8, kNearThreads, 0, s>>>(V, p, M, list != nullptr, epoch);
  } else {
    near_kernel<false><<<152 * 8, kNearThreads, 0, s>>>(V, p, M, list != nullptr, epoch);
  }
  rounds_kernel<false><<<152 * 4, kRoundThreads, 0, s>>>(V, M, list, list_count);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    e = fp16 ? launch_cells<false, true>(V, p, M, nullptr, s) : launch_cells<false, false>(V, p, M, nullptr, s);
  }
  if (e != cudaSuccess) return e;
  rounds_kernel<true><<<152 * 4, kRoundThreads, 0, s>>>(V, M, list, list_count);
  scan_kernel<<<1, 1024, 0, s>>>(V, M, total);
  return cudaGetLastError();
}

cudaError_t launch_recent_blocks(const Volume& V, uint32_t frames, uint32_t* list, uint32_t* count, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(count, 0, sizeof(uint32_t), s);
  if (e != cudaSuccess) return e;
  recent_blocks_kernel<<<1024, 256, 0, s>>>(V, frames, list, count);
  return cudaGetLastError();
}

cudaError_t launch_mc_emit(const Volume& V, const Params& p, const MeshBuffers& M, float* tris, cudaStream_t s) {
  return V.layers16 != nullptr ? launch_cells<true, true>(V, p, M, tris, s) : launch_cells<true, false>(V, p, M, tris, s);
}

}  // namespace vh
