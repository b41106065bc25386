// vh_raycast.cu -- depth ray-cast of the fused volume (the TSDF ray-caster that produces depth maps of the
// fused surface, e.g. as training targets for a depth denoiser).  The reference has no ray-caster; the
// surface definition is the one its marching cubes uses: a voxel's observed layers are planes
// (planeSignedDistanceGpu, cuda_mesh_extractor.cu:259-262, normals unpacked as at :237-257).
//
// The ray through the pixel centre is parameterised by camera depth z (camera-frame direction
// ((u - cx)/fx, (v - cy)/fy, 1)); it is sampled every `step` voxels of path length from min_depth
// to max_depth.  A voxel's distance at a point x is the plane distance n.x - offset of its heaviest observed
// layer, over all directions, whose normal faces the ray (n.d < 0; first such layer on ties): the
// best-supported surface of the voxel, so that the low-weight layers a few noisy observations leave in front
// of a surface do not stop the ray.  The distance at a sample x is the trilinear blend, with the weights of x
// among the 8 surrounding voxel centres, of those voxels' distances at x (over the voxels that have one,
// renormalised; none when they carry less than half of the weight).  The first step from a positive to a
// non-positive distance, with a drop of at most the truncation distance, is the hit; its depth is
// interpolated linearly.
// Unallocated blocks are skipped to the point where the ray leaves them.  Output: depth (camera z) per
// pixel, 0 where nothing is hit.
//
// Eight lanes per pixel, one per voxel around the sample; a warp's four rays run in step.  A ray is a serial chain
// of samples and a sample is 8 voxels of up to 18 layers each: with one thread per ray a 640x480 view of a room
// fused from 6 frames took 16-20 ms, 12 of 32 threads active and 8 % of the issue slots used.  Lane q of a ray's
// eight holds the voxel of the neighbourhood whose coordinates' parities are the bits of q, so that when the
// neighbourhood moves one voxel along an axis half of the lanes keep theirs: a voxel's plane (its choice depends on
// the ray's direction alone, not on the sample) stays in registers until its lane moves on.  A voxel without an
// observed layer is known from its bit of the observed-voxel mask, without reading bins.  The same view takes
// 6.3 ms; the kernel is bound by instruction issue (75 % of the slots, 21 of 32 threads active).  Measured and not
// kept: one lane per ray through unallocated space and eight through blocks, handing over inside a warp
// (12-21 ms) or inside a CTA with a list of rays (6.7-25 ms): rays that run through blocks out of step execute both
// parts of the loop.
#include "vh_common.cuh"
#include "vh_kernels.h"

namespace vh {
namespace {

constexpr int kRTX = 8, kRTY = 4;  // pixels per CTA
constexpr int kMaxGridY = 65535;   // CTAs that a grid holds along y, 262,140 rows: the rest of a taller image goes along z
constexpr int kRayThreads = 8 * kRTX * kRTY;
constexpr int kMaxRaySteps = 1 << 16;

// x / b correctly rounded, inv_b = 1 / b correctly rounded: two corrections of x * inv_b by the exact remainder
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990: a faithful quotient
// corrected with a correctly rounded reciprocal is the correctly rounded one).  5 instructions without a branch
// where the quotient is of ordinary size; the division itself elsewhere (overflow, infinities, NaN, and
// operands so small that the remainder could underflow).
__device__ __forceinline__ float div_by(float x, float b, float inv_b) {
  float q = __fmul_rn(x, inv_b);
  q = __fmaf_rn(__fmaf_rn(-q, b, x), inv_b, q);
  q = __fmaf_rn(__fmaf_rn(-q, b, x), inv_b, q);
  const float a = fabsf(q);
  return a < 0x1p60f && ((a > 0x1p-60f && fabsf(x) > 0x1p-90f) || x == 0.0f) ? q : __fdiv_rn(x, b);
}

// the heaviest camera-facing layer (n, off) of observed voxel li of block b, its centre at grid (gx, gy, gz) + 0.5;
// false: no such layer
__device__ __forceinline__ bool voxel_plane(const Volume& V, uint32_t b, int li, int gx, int gy, int gz, float vs,
                                            f3 dw, f3& n, float& off) {
  const uint32_t dirs = V.dir_mask[b];
  // The weights of every flagged direction's bin first: independent loads that bring the bins in together.
  constexpr int kN = kDirs * kLayers;
  float w[kN];
  if (V.layers16 == nullptr) {
#pragma unroll
    for (int d = 0; d < kDirs; ++d) {
      const float4* L = V.layers + layer_index(b, d, li, 0);
      const bool use = (dirs >> d) & 1U;
#pragma unroll
      for (int l = 0; l < kLayers; ++l) w[d * kLayers + l] = use ? L[l].x : 0.0f;
    }
  } else {
#pragma unroll
    for (int d = 0; d < kDirs; ++d) {
      uint4 A = make_uint4(0U, 0U, 0U, 0U);
      if ((dirs >> d) & 1U) A = V.layers16[bin16_index(b, d, li)];
      w[d * kLayers] = h2f(A.x & 0xffffU);
      w[d * kLayers + 1] = h2f(A.y >> 16);
      w[d * kLayers + 2] = h2f(A.w & 0xffffU);
    }
  }
  // Candidates from the heaviest down (the first of equal weights first) until one faces the camera: one or two
  // normals are decoded instead of one per layer.
  for (;;) {
    float best = 0.0f;
    int k = -1;
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      if (w[i] > best) {
        best = w[i];
        k = i;
      }
    }
    if (k < 0) return false;
    const int d = k / kLayers, l = k - d * kLayers;
    if (V.layers16 == nullptr) {
      // plane offset, packed normal
      const float2 pn = *reinterpret_cast<const float2*>(&(V.layers + layer_index(b, d, li, l))->z);
      n = unpack_normal_mesh(__float_as_uint(pn.y));
      off = pn.x;
    } else {
      const uint32_t* bin = reinterpret_cast<const uint32_t*>(V.layers16 + bin16_index(b, d, li));
      const uint32_t nk = bin[5 + l];
      const uint32_t pw = bin[l == 0 ? 1 : (l == 1 ? 2 : 4)];
      const uint32_t p16 = l == 1 ? pw >> 16 : pw & 0xffffU;
      const f3 c = mk3(__fmul_rn(__fadd_rn(static_cast<float>(gx), 0.5f), vs),
                       __fmul_rn(__fadd_rn(static_cast<float>(gy), 0.5f), vs),
                       __fmul_rn(__fadd_rn(static_cast<float>(gz), 0.5f), vs));
      n = unpack_normal_mesh(nk);
      off = __fadd_rn(dot_rn(bin_normal(nk), c), __fmul_rn(h2f(p16), vs));  // decode_layer16
    }
    if (dot3(n, dw) < 0.0f) return true;
#pragma unroll
    for (int i = 0; i < kN; ++i) w[i] = i == k ? 0.0f : w[i];
  }
}

// where the ray leaves the unallocated block (bx, by, bz) that holds its sample at z, and a little further
__device__ __forceinline__ float skip_block(float z, float dz, f3 o, f3 dw, f3 inv_dw, int bx, int by, int bz, float vs) {
  float zexit = 3.0e38f;
  const int bb[3] = {bx, by, bz};
  const float oo[3] = {o.x, o.y, o.z}, dd[3] = {dw.x, dw.y, dw.z}, id[3] = {inv_dw.x, inv_dw.y, inv_dw.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int side = dd[k] > 0.0f ? bb[k] + 1 : bb[k];
    const float t = div_by(static_cast<float>(side * kBlockSide) * vs - oo[k], dd[k], id[k]);
    if (dd[k] > 0.0f || dd[k] < 0.0f) zexit = fminf(zexit, t);
  }
  return fmaxf(z + dz, zexit + 0.25f * dz);
}

// A ray's eight lanes hold the same ray state and take the same branches; the warp's four rays run in step (full
// warp shuffles) until the last one has ended.  Four resident CTAs per SM (64 registers): 6.3 ms for the view above
// against 8.7 ms without the bound (96 registers), 7.1 with three and 6.6 with five.
__global__ void __launch_bounds__(kRayThreads, 4) raycast_kernel(const Volume V, const Params p, float min_depth,
                                                                 float max_depth, float step, float* __restrict__ out) {
  const int lane = threadIdx.x & 31, q = lane & 7, base = lane & 24, ray = threadIdx.x >> 3;
  const int px = q & 1, py = (q >> 1) & 1, pz = q >> 2;  // parities of this lane's voxel
  // a warp's four rays are 2x2 pixels, a CTA's eight warps 4x2 of those
  const int warp = ray >> 2, r = ray & 3;
  const int u = blockIdx.x * kRTX + 2 * (warp & 3) + (r & 1);
  const uint32_t v = (blockIdx.z * kMaxGridY + blockIdx.y) * kRTY + 2 * (warp >> 2) + (r >> 1);
  const bool inside = u < p.width && v < static_cast<uint32_t>(p.height);
  const f3 dc = mk3((static_cast<float>(u) - p.cx) / p.fx, (static_cast<float>(v) - p.cy) / p.fy, 1.0f);
  const f3 dw = xform_vector(p.T_wc, dc);
  const f3 inv_dw = mk3(1.0f / dw.x, 1.0f / dw.y, 1.0f / dw.z);
  const f3 o = mk3(p.T_wc.t[0], p.T_wc.t[1], p.T_wc.t[2]);
  const float dz = step * p.voxel_size / norm3(dc);
  const float vs = p.voxel_size, inv_vs = 1.0f / vs;
  float z = min_depth;
  bool prev_ok = false;
  float prev_sdf = 0.0f, prev_z = 0.0f, result = 0.0f;
  // this lane's voxel (its plane once read) and the last block it looked up
  bool vox_known = false, vox_has = false;
  int vx = 0, vy = 0, vz = 0;
  f3 vn = mk3(0.0f, 0.0f, 0.0f);
  float voff = 0.0f;
  bool blk_known = false;
  int kx = 0, ky = 0, kz = 0;
  uint32_t kb = kInvalidBlock;
  // the block of the ray's last sample
  bool c_known = false;
  int cx = 0, cy = 0, cz = 0;
  uint32_t cb = kInvalidBlock;
  bool active = inside;
  for (int it = 0; it < kMaxRaySteps; ++it) {
    active = active && z <= max_depth;
    if (!__any_sync(0xffffffffU, active)) break;
    const f3 x = mk3(o.x + dw.x * z, o.y + dw.y * z, o.z + dw.z * z);
    const float qx = div_by(x.x, vs, inv_vs), qy = div_by(x.y, vs, inv_vs), qz = div_by(x.z, vs, inv_vs);
    // the sample's block, then its neighbourhood's
    const int sx = static_cast<int>(floorf(qx)) >> 3;  // floor division by 8
    const int sy = static_cast<int>(floorf(qy)) >> 3;
    const int sz = static_cast<int>(floorf(qz)) >> 3;
    if (active && !(c_known && sx == cx && sy == cy && sz == cz)) {
      cb = lookup_block(V, sx, sy, sz);
      cx = sx;
      cy = sy;
      cz = sz;
      c_known = true;
    }
    const bool sampled = active && cb != kInvalidBlock;
    if (active && !sampled) {
      prev_ok = false;
      z = skip_block(z, dz, o, dw, inv_dw, sx, sy, sz, vs);
    }
    if (!__any_sync(0xffffffffU, sampled)) continue;
    const float fx = qx - 0.5f, fy = qy - 0.5f, fz = qz - 0.5f;
    const float x0f = floorf(fx), y0f = floorf(fy), z0f = floorf(fz);
    const int x0 = static_cast<int>(x0f), y0 = static_cast<int>(y0f), z0 = static_cast<int>(z0f);
    // this lane's voxel of the neighbourhood [x0, x0 + 1] x [y0, y0 + 1] x [z0, z0 + 1]
    const int ax = (x0 & 1) ^ px, ay = (y0 & 1) ^ py, az = (z0 & 1) ^ pz;
    const int nx = x0 + ax, ny = y0 + ay, nz = z0 + az;
    const bool same = vox_known && nx == vx && ny == vy && nz == vz;
    const int bx = nx >> 3, by = ny >> 3, bz = nz >> 3;
    if (sampled && !(blk_known && bx == kx && by == ky && bz == kz)) {
      kb = lookup_block(V, bx, by, bz);
      kx = bx;
      ky = by;
      kz = bz;
      blk_known = true;
    }
    if (sampled && !same) {
      vx = nx;
      vy = ny;
      vz = nz;
      vox_known = true;
      vox_has = false;
      if (kb != kInvalidBlock) {
        const int li = (nx & 7) + kBlockSide * ((ny & 7) + kBlockSide * (nz & 7));
        if ((V.obs_mask[static_cast<size_t>(kb) * (kBlockVoxels / 32) + (li >> 5)] >> (li & 31)) & 1U) {
          vox_has = voxel_plane(V, kb, li, nx, ny, nz, vs, dw, vn, voff);
        }
      }
    }
    const uint32_t has_all = __ballot_sync(0xffffffffU, sampled && vox_has);
    float ws = 0.0f, acc = 0.0f;
    if (has_all) {
      // the blend over the voxels that have a distance, summed in the order of the corners (x fastest)
      const uint32_t has = (has_all >> base) & 0xffU;
      const float tx = fx - x0f, ty = fy - y0f, tz = fz - z0f;
      const float w = (ax ? tx : 1.0f - tx) * (ay ? ty : 1.0f - ty) * (az ? tz : 1.0f - tz);
      const float wsd = w * (vn.x * x.x + vn.y * x.y + vn.z * x.z - voff);
      const int par = (x0 & 1) | ((y0 & 1) << 1) | ((z0 & 1) << 2);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int ql = k ^ par;
        const float wk = __shfl_sync(0xffffffffU, w, base | ql);
        const float sk = __shfl_sync(0xffffffffU, wsd, base | ql);
        if ((has >> ql) & 1U) {
          acc += sk;
          ws += wk;
        }
      }
    }
    if (!sampled) continue;
    if (!(ws >= 0.5f)) {
      prev_ok = false;
      z += dz;
      continue;
    }
    const float sdf = acc / ws;
    if (prev_ok && prev_sdf > 0.0f && sdf <= 0.0f && prev_sdf - sdf <= p.truncation) {
      result = prev_z + (z - prev_z) * (prev_sdf / (prev_sdf - sdf));
      active = false;
      continue;
    }
    prev_ok = true;
    prev_sdf = sdf;
    prev_z = z;
    z += dz;
  }
  if (inside && q == 0) out[static_cast<size_t>(v) * p.width + u] = result;
}

}  // namespace

cudaError_t launch_raycast(const Volume& V, const Params& p, float min_depth, float max_depth, float step, float* out,
                           cudaStream_t s) {
  const int ty = (p.height + kRTY - 1) / kRTY;
  const dim3 grid((p.width + kRTX - 1) / kRTX, ty < kMaxGridY ? ty : kMaxGridY, (ty + kMaxGridY - 1) / kMaxGridY);
  raycast_kernel<<<grid, kRayThreads, 0, s>>>(V, p, min_depth, max_depth, step, out);
  return cudaGetLastError();
}

}  // namespace vh
