// Learned absorbing boundary: a thin layer around the interior whose outer
// cells are advanced by a one-way (outgoing-wave) update with a per-cell
// coefficient predicted by a small MLP.
//
// Geometry.  The grid is interior + a layer of L cells + bord zero cells on
// every side; the plain update runs over interior and layer alike (the
// medium is extended into the layer, no random velocities).  A layer cell d
// cells outside the interior along an axis has an update stencil (radius 4)
// reaching d + 4 cells out; for the layer's outer 4 cells (d = L-3 .. L,
// the ghost zone) that reaches the zero border, where an unbounded medium
// would hold the outgoing wave.  After the plain step those cells are
// overwritten with the box-scheme update of the one-way wave equation
// u_t + c u_n = 0 along the outward normal n,
//
//     u_g(t+1) = u_i(t) + k (u_g(t) - u_i(t+1)),   k = (1 - r) / (1 + r),  r = c dt / h
//
// (g the ghost cell, i its inward neighbour), applied outward from d = L-3
// (whose inward neighbour carries the plain update) to d = L, for p and q,
// face by face: the z faces, then the y faces, then the x faces (edge and
// corner cells keep the last face's value).  For r > 0 the box scheme of
// the one-way equation is unconditionally stable and 0 < k < 1.
//
//  * FLETCHER_BOUNDARY_ONEWAY: k from the medium, c = vpz along z and
//    vpz sqrt(1 + 2 epsilon) along x and y (the normal-incidence P-wave
//    velocities of a vertical-axis medium);
//  * FLETCHER_BOUNDARY_LEARNED: (k_p, k_q) = sigmoid(network(inputs)) per
//    ghost cell and step.  The inputs are the 9-point stencils of p and q
//    along the outward normal at t and t-1 (points beyond the layer read as
//    zero) divided by their largest magnitude s, vpz / 4000, epsilon, delta
//    and d / L; the network learns the coefficient with which the update
//    reproduces the unbounded medium's next value (oblique incidence,
//    tilted anisotropy, the wave's own apparent velocity).
//
// Network: 40 -> 32 -> 32 -> 2, tanh, FP16 weights and FP16 activations
// between layers, FP32 accumulation and FP32 biases.
//   * inference runs on the tensor cores (mma.sync m16n8k16, f16 x f16 ->
//     f32) inside the boundary kernel (k_abc_boundary, one cooperative launch
//     after the plain step that also applies the one-way update): one warp
//     evaluates 16 ghost cells, the layer-1 and layer-2 outputs stay in
//     registers as the next layer's A fragments, and k stays in registers
//     until the update uses it; the weights' B fragments are read from a
//     shared-memory copy (in registers they took 62 of 128, and the SM held
//     16 warps instead of 24: 119 against 90 us per evaluating step at
//     256^3);
//   * training (k_abc_train) is a per-sample forward and backward pass in
//     FP32 with the same roundings (straight-through), block sums of the
//     gradients added up in block order (k_abc_reduce: training is
//     reproducible bit for bit), and Adam (k_abc_adam) on FP32 master
//     weights.  The loss of
//     a sample is sum_c (sigmoid(y_c) a_c - b_c)^2 with a = (u_g(t) -
//     u_i(t+1)) / s and b = (u_g(t+1) - u_i(t)) / s: the update's error
//     when the neighbour's next value is the true one.
//
// Training data (k_abc_collect) come from plain-method runs on padded
// domains: around a virtual interior box, the ghost cells' inputs are read
// with everything beyond the virtual layer set to zero, and the next values
// u(t+1) are the plain update on the padded field (an unbounded medium as
// far as the ghost cells can tell).
#include <cuda_fp16.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <vector>

#include "../../include/fletcher_gb300.h"
#include "device_util.cuh"
#include "fletcher_internal.h"
#include "stencil_common.cuh"

int flt_record_error(int code, const char *msg);

namespace flt {

constexpr int kIn = 40, kHid = 32, kOut = 2;
constexpr int kTgt = 4;   // targets of a sample: a_p, a_q, b_p, b_q
constexpr int kSt = 36;   // stencil inputs (4 x 9)
// Master parameter layout (FP32): W1 [32][40], b1, W2 [32][32], b2, W3 [2][32], b3.
constexpr int oW1 = 0, oB1 = oW1 + kHid * kIn, oW2 = oB1 + kHid, oB2 = oW2 + kHid * kHid, oW3 = oB2 + kHid,
              oB3 = oW3 + kOut * kHid, kNP = oB3 + kOut;
static_assert(kNP == FLETCHER_ABC_PARAMS, "parameter count");
constexpr int kK1 = 48;      // layer-1 K padded to a multiple of 16
constexpr int kXs = 56;      // row stride (halves) of a warp's feature tile: conflict-free A loads
constexpr float kVScale = 1.0f / 4000.0f;
constexpr float kMinScale = 1e-30f;  // smallest stencil magnitude the network sees
constexpr int kGhostD = kRadius;     // ghost cells per ray: the layer's outer 4
constexpr float kInitBias = 0.85f;   // initial output bias: k ~ 0.7 (r ~ 0.18)

// Inference copy of the network: FP16 weights in mma B-operand order
// (row n = output, contiguous k), FP32 biases.
struct NetHalf {
  __half w1[kHid * kK1];
  __half w2[kHid * kHid];
  __half w3[8 * kHid];
  float b1[kHid], b2[kHid], b3[8];
};

// A box [lo, hi) per axis.
struct Box {
  int lo[3], hi[3];
};

// One layer cell (the taper's list): position and distance d.
struct LayerCell {
  int x, y, z, d;
};

// The ghost zone of a layer: the interior box, the layer, the kept box
// (interior grown by L) and the first cell of each face.  Faces 0..5 are
// z-, z+, y-, y+, x-, x+; a face is a set of rays along its outward normal,
// one per transverse position of the kept box (first transverse axis
// fastest), 4 cells per ray (d = L-3 .. L, d fastest).
struct Ghost {
  Box in, keep;
  int L;
  long off[7];
};

__host__ __device__ __forceinline__ int face_axis(int f) { return 2 - f / 2; }
__host__ __device__ __forceinline__ int face_sign(int f) { return (f & 1) ? 1 : -1; }
__host__ __device__ __forceinline__ void transverse(int a, int &t0, int &t1) {
  t0 = a == 0 ? 1 : 0;
  t1 = a == 2 ? 1 : 2;
}

Ghost make_ghost(const Box &in, int L) {
  Ghost G;
  G.in = in;
  G.L = L;
  for (int a = 0; a < 3; ++a) {
    G.keep.lo[a] = in.lo[a] - L;
    G.keep.hi[a] = in.hi[a] + L;
  }
  G.off[0] = 0;
  for (int f = 0; f < 6; ++f) {
    int t0, t1;
    transverse(face_axis(f), t0, t1);
    const long rays = (long)(G.keep.hi[t0] - G.keep.lo[t0]) * (G.keep.hi[t1] - G.keep.lo[t1]);
    G.off[f + 1] = G.off[f] + rays * kGhostD;
  }
  return G;
}

// Ghost cell i: coordinates c, face f, normal axis a, outward sign; returns d.
__host__ __device__ __forceinline__ int ghost_cell(const Ghost &G, long i, int (&c)[3], int &f, int &a, int &sgn) {
  f = 0;
  while (f < 5 && i >= G.off[f + 1]) ++f;
  const long j = i - G.off[f];
  a = face_axis(f);
  sgn = face_sign(f);
  int t0, t1;
  transverse(a, t0, t1);
  const int e0 = G.keep.hi[t0] - G.keep.lo[t0];
  const int ray = (int)(j / kGhostD);  // a face holds fewer than 2^31 rays
  const int d = G.L - kGhostD + 1 + (int)(j % kGhostD);
  c[t0] = G.keep.lo[t0] + ray % e0;
  c[t1] = G.keep.lo[t1] + ray / e0;
  c[a] = sgn < 0 ? G.in.lo[a] - d : G.in.hi[a] - 1 + d;
  return d;
}

__host__ __device__ __forceinline__ int face_of(const Ghost &G, long i) {
  int f = 0;
  while (f < 5 && i >= G.off[f + 1]) ++f;
  return f;
}

// Index step of one cell outward along face f's normal.
__host__ __device__ __forceinline__ int normal_step(int f, int sy, int pitch) {
  const int a = face_axis(f);
  const int s = a == 0 ? 1 : (a == 1 ? pitch : sy * pitch);
  return face_sign(f) > 0 ? s : -s;
}

__host__ __device__ __forceinline__ long cell_index(int x, int y, int z, int sy, int pitch) {
  return ((long)z * sy + y) * pitch + x;
}

// Index in the field of ghost cell i and its face (ghost_cell without an
// indexed coordinate array, for the hot kernels).
__device__ __forceinline__ long ghost_index(const Ghost &G, long i, int sy, int pitch, int &f) {
  f = face_of(G, i);
  const long j = i - G.off[f];
  const int a = face_axis(f);
  const int t0 = a == 0 ? 1 : 0, t1 = a == 2 ? 1 : 2;
  const int e0 = G.keep.hi[t0] - G.keep.lo[t0];
  const int ray = (int)(j / kGhostD);
  const int d = G.L - kGhostD + 1 + (int)(j % kGhostD);
  const int u = G.keep.lo[t0] + ray % e0, v = G.keep.lo[t1] + ray / e0;
  const int n = face_sign(f) < 0 ? G.in.lo[a] - d : G.in.hi[a] - 1 + d;
  const int x = a == 0 ? n : u;
  const int y = a == 1 ? n : (a == 0 ? u : v);
  const int z = a == 2 ? n : v;
  return cell_index(x, y, z, sy, pitch);
}

// ---- features -------------------------------------------------------------------

// vpz, epsilon, delta of a cell of the updated region from its coefficients (v2pz = vpz^2,
// v2px = vpz^2 (1 + 2 eps), v2pn = vpz^2 (1 + 2 delta): original/precomp.h).
__device__ __forceinline__ float4 medium_of(const float *coef, int x, int y, int z, int sy, int pitch) {
  const float *c = coef + coef_index(x - kRadius, y, z, sy, pitch);
  const float v2px = c[DC_V2PX * kTileX], v2pz = c[DC_V2PZ * kTileX], v2pn = c[DC_V2PN * kTileX];
  float4 m;
  m.x = sqrtf(v2pz);
  m.y = v2pz > 0.f ? 0.5f * (v2px / v2pz - 1.0f) : 0.f;
  m.z = v2pz > 0.f ? 0.5f * (v2pn / v2pz - 1.0f) : 0.f;
  m.w = 0.f;
  return m;
}

// The 9 (p, q) values of field F along axis a from (x, y, z), offsets
// sign * (-4 .. 4); points outside `keep` read as zero.
__device__ __forceinline__ void normal_stencil(const float2 *F, int x, int y, int z, int a, int sgn, const Box &keep,
                                               int sy, int pitch, float *p9, float *q9) {
#pragma unroll
  for (int j = -kRadius; j <= kRadius; ++j) {
    int c[3] = {x, y, z};
    c[a] += sgn * j;
    float2 v = make_float2(0.f, 0.f);
    if (c[0] >= keep.lo[0] && c[0] < keep.hi[0] && c[1] >= keep.lo[1] && c[1] < keep.hi[1] && c[2] >= keep.lo[2] &&
        c[2] < keep.hi[2])
      v = F[cell_index(c[0], c[1], c[2], sy, pitch)];
    p9[j + kRadius] = v.x;
    q9[j + kRadius] = v.y;
  }
}

// One-way coefficient of the medium along axis a: k = (1 - r) / (1 + r),
// r = c dt / h, c = vpz (z) or vpz sqrt(1 + 2 eps) (x, y).
__host__ __device__ __forceinline__ float oneway_k(float vpz, float eps, int a, float dt, float h) {
  const float c = a == 2 ? vpz : vpz * sqrtf(1.0f + 2.0f * eps);
  const float r = c * dt / h;
  return (1.0f - r) / (1.0f + r);
}

// ---- the plain update's rhs over the cells outside a box (an empty box: every cell) ----

// (p, q) of the current field at a cell, if it lies outside `keep`.
__device__ __forceinline__ float2 outer(const float2 *F, int x, int y, int z, const Box &keep, int sy, int pitch) {
  const bool in = x >= keep.lo[0] && x < keep.hi[0] && y >= keep.lo[1] && y < keep.hi[1] && z >= keep.lo[2] &&
                  z < keep.hi[2];
  if (in) return make_float2(0.f, 0.f);
  return F[((size_t)z * sy + y) * pitch + x];
}

// dt^2 * (rhsp, rhsq) of original/sample.h:32-89 evaluated on the field
// outside `keep` (it is linear in the field; an empty `keep` gives the
// whole update).
__device__ float2 outer_update(const float2 *F, const float *coef, int x, int y, int z, const Box &keep, int sy,
                               int pitch, float dx, float dy, float dz, float dt) {
  const float K[5] = {cK0, cK1, cK2, cK3, cK4};
  const float Lw[5] = {0.f, cL1, cL2, cL3, cL4};
  // The centre term counts when the cell itself lies outside `keep`.
  const float2 u0 = outer(F, x, y, z, keep, sy, pitch);
  float2 d2[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) d2[a] = make_float2(K[0] * u0.x, K[0] * u0.y);
  const int cx[3] = {1, 0, 0}, cy[3] = {0, 1, 0}, cz[3] = {0, 0, 1};
#pragma unroll
  for (int a = 0; a < 3; ++a)
    for (int k = 1; k <= kRadius; ++k) {
      const float2 u = outer(F, x + k * cx[a], y + k * cy[a], z + k * cz[a], keep, sy, pitch);
      const float2 w = outer(F, x - k * cx[a], y - k * cy[a], z - k * cz[a], keep, sy, pitch);
      d2[a].x += K[k] * (u.x + w.x);
      d2[a].y += K[k] * (u.y + w.y);
    }
  // Mixed derivatives: xy, yz, xz.
  const int pa[3] = {0, 1, 0}, pb[3] = {1, 2, 2};
  float2 dc[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
  for (int m = 0; m < 3; ++m)
    for (int i = 1; i <= kRadius; ++i)
      for (int j = 1; j <= kRadius; ++j) {
        int o1[3] = {0, 0, 0}, o2[3] = {0, 0, 0};
        o1[pa[m]] = i;
        o2[pb[m]] = j;
        const float2 pp = outer(F, x + o1[0] + o2[0], y + o1[1] + o2[1], z + o1[2] + o2[2], keep, sy, pitch);
        const float2 pm = outer(F, x + o1[0] - o2[0], y + o1[1] - o2[1], z + o1[2] - o2[2], keep, sy, pitch);
        const float2 mp = outer(F, x - o1[0] + o2[0], y - o1[1] + o2[1], z - o1[2] + o2[2], keep, sy, pitch);
        const float2 mm = outer(F, x - o1[0] - o2[0], y - o1[1] - o2[1], z - o1[2] - o2[2], keep, sy, pitch);
        const float w = Lw[i] * Lw[j];
        dc[m].x += w * (pp.x - pm.x - mp.x + mm.x);
        dc[m].y += w * (pp.y - pm.y - mp.y + mm.y);
      }
  const float sx2 = 1.0f / (dx * dx), sy2 = 1.0f / (dy * dy), sz2 = 1.0f / (dz * dz);
  const float sxy = 1.0f / (dx * dy), syz = 1.0f / (dy * dz), sxz = 1.0f / (dx * dz);
  const float pxx = d2[0].x * sx2, pyy = d2[1].x * sy2, pzz = d2[2].x * sz2;
  const float qxx = d2[0].y * sx2, qyy = d2[1].y * sy2, qzz = d2[2].y * sz2;
  const float pxy = dc[0].x * sxy, pyz = dc[1].x * syz, pxz = dc[2].x * sxz;
  const float qxy = dc[0].y * sxy, qyz = dc[1].y * syz, qxz = dc[2].y * sxz;
  const float *c0 = coef + coef_index(x - kRadius, y, z, sy, pitch);
  auto C = [&](int k) { return c0[k * kTileX]; };
  const float cxx = C(DC_XX), cyy = C(DC_YY), czz = C(DC_ZZ), cxy = C(DC_XY), cyz = C(DC_YZ), cxz = C(DC_XZ);
  const float h1p = cxx * pxx + cyy * pyy + czz * pzz + cxy * pxy + cyz * pyz + cxz * pxz;
  const float h1q = cxx * qxx + cyy * qyy + czz * qzz + cxy * qxy + cyz * qyz + cxz * qxz;
  const float h2p = pxx + pyy + pzz - h1p, h2q = qxx + qyy + qzz - h1q;
  const float rhsp = C(DC_V2PX) * h2p + C(DC_V2PZ) * h1q + C(DC_V2SZ) * (h1p - h1q);
  const float rhsq = C(DC_V2PN) * h2p + C(DC_V2PZ) * h1q - C(DC_V2SZ) * (h2p - h2q);
  const float dt2 = dt * dt;
  return make_float2(rhsp * dt2, rhsq * dt2);
}

__device__ __forceinline__ uint32_t mix32(uint32_t a, uint32_t b) {
  uint32_t h = a * 0x9E3779B1u ^ (b + 0x7F4A7C15u + (a << 6) + (a >> 2));
  h ^= h >> 16;
  h *= 0x85EBCA6Bu;
  h ^= h >> 13;
  h *= 0xC2B2AE35u;
  h ^= h >> 16;
  return h;
}

// Training samples from the ghost cells of the layer around a virtual
// interior box: features, targets (a_p, a_q, b_p, b_q) over s, and the
// cell (x, y, z, face + 8 d).  A random fraction `keep_frac` of the cells is
// taken; cells whose stencils are below `min_scale` carry no wave and are
// skipped.  The next values are the plain update of original/sample.h:32-89
// (u(t+1) = 2 u(t) - u(t-1) + dt^2 rhs) on the padded field.
//
// The samples land in cell order, so the training set does not depend on
// thread timing: block b takes the cells [b per, (b+1) per); a counting
// pass gives each block's number of samples, their prefix sums (host) its
// first slot, and the writing pass ranks each cell inside its block with
// warp ballots.

// Whether ghost cell i becomes a sample; its stencils and scale.
__device__ __forceinline__ bool collect_cell(const float2 *cur, const float2 *prev, const Ghost &G, long i, int sy,
                                             int pitch, float keep_frac, uint32_t seed, float min_scale, float (&v)[kSt],
                                             float &s, int (&c)[3], int &f, int &a, int &sgn, int &d) {
  if ((mix32(seed, (uint32_t)i) >> 8) * (1.0f / 16777216.0f) >= keep_frac) return false;
  d = ghost_cell(G, i, c, f, a, sgn);
  normal_stencil(cur, c[0], c[1], c[2], a, sgn, G.keep, sy, pitch, v, v + 9);
  normal_stencil(prev, c[0], c[1], c[2], a, sgn, G.keep, sy, pitch, v + 18, v + 27);
  s = 0.f;
#pragma unroll
  for (int k = 0; k < kSt; ++k) s = fmaxf(s, fabsf(v[k]));
  return (s > min_scale) && (s > kMinScale);
}

constexpr int kCollectBlock = 256;

__global__ void __launch_bounds__(kCollectBlock) k_abc_collect_count(const float2 *cur, const float2 *prev,
                                                                     const __grid_constant__ Ghost G, int sy,
                                                                     int pitch, float keep_frac, uint32_t seed,
                                                                     float min_scale, long per, int *block_count) {
  __shared__ int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  const long n = G.off[6];
  const long lo = blockIdx.x * per, hi = min(n, lo + per);
  int mine = 0;
  for (long i = lo + threadIdx.x; i < hi; i += kCollectBlock) {
    float v[kSt], sc;
    int c[3], f, a, sgn, d;
    mine += collect_cell(cur, prev, G, i, sy, pitch, keep_frac, seed, min_scale, v, sc, c, f, a, sgn, d) ? 1 : 0;
  }
  atomicAdd(&cnt, mine);  // an integer count: the order does not matter
  __syncthreads();
  if (threadIdx.x == 0) block_count[blockIdx.x] = cnt;
}

__global__ void __launch_bounds__(kCollectBlock) k_abc_collect(const float2 *cur, const float2 *prev,
                                                               const float *coef, const __grid_constant__ Ghost G,
                                                               int sy, int pitch, float dx, float dy, float dz,
                                                               float dt, float keep_frac, uint32_t seed,
                                                               float min_scale, long per, const long *block_first,
                                                               float *feat, float *tgt, int4 *pos, long cap) {
  __shared__ int warp_sum[kCollectBlock / 32];
  const long n = G.off[6];
  const long lo = blockIdx.x * per, hi = min(n, lo + per);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Box all = {{0, 0, 0}, {0, 0, 0}};  // empty kept box: the whole field counts
  long next = block_first[blockIdx.x];  // slot of this block's next sample
  for (long c0 = lo; c0 < hi; c0 += kCollectBlock) {
    const long i = c0 + threadIdx.x;
    float v[kSt], s = 0.f;
    int c[3] = {0, 0, 0}, f = 0, a = 0, sgn = 1, d = 0;
    const bool keep =
        i < hi && collect_cell(cur, prev, G, i, sy, pitch, keep_frac, seed, min_scale, v, s, c, f, a, sgn, d);
    // Rank in cell order: lanes before this one in the warp, then warps before it.
    const unsigned ball = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_sum[warp] = __popc(ball);
    __syncthreads();
    int before = __popc(ball & ((1u << lane) - 1u)), total = 0;
#pragma unroll
    for (int w = 0; w < kCollectBlock / 32; ++w) {
      before += w < warp ? warp_sum[w] : 0;
      total += warp_sum[w];
    }
    __syncthreads();
    const long slot = next + before;
    next += total;
    if (!keep || slot >= cap) continue;
    pos[slot] = make_int4(c[0], c[1], c[2], f + 8 * d);
    const float inv = 1.0f / s;
    float *fr = feat + slot * kIn;
#pragma unroll
    for (int k = 0; k < kSt; ++k) fr[k] = v[k] * inv;
    const float4 m = medium_of(coef, c[0], c[1], c[2], sy, pitch);
    fr[36] = m.x * kVScale;
    fr[37] = m.y;
    fr[38] = m.z;
    fr[39] = (float)d / (float)G.L;
    int ci[3] = {c[0], c[1], c[2]};
    ci[a] -= sgn;
    const long g = cell_index(c[0], c[1], c[2], sy, pitch), gi = cell_index(ci[0], ci[1], ci[2], sy, pitch);
    const float2 ug = cur[g], ui = cur[gi], ugm = prev[g], uim = prev[gi];
    const float2 rg = outer_update(cur, coef, c[0], c[1], c[2], all, sy, pitch, dx, dy, dz, dt);
    const float2 ri = outer_update(cur, coef, ci[0], ci[1], ci[2], all, sy, pitch, dx, dy, dz, dt);
    const float ugx = 2.0f * ug.x - ugm.x + rg.x, ugy = 2.0f * ug.y - ugm.y + rg.y;
    const float uix = 2.0f * ui.x - uim.x + ri.x, uiy = 2.0f * ui.y - uim.y + ri.y;
    float *t = tgt + slot * kTgt;
    t[0] = (ug.x - uix) * inv;
    t[1] = (ug.y - uiy) * inv;
    t[2] = (ugx - ui.x) * inv;
    t[3] = (ugy - ui.y) * inv;
  }
}

// ---- inference on the tensor cores ---------------------------------------------

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_h2(float lo_v, float hi_v) {
  const __half2 h = __floats2half2_rn(lo_v, hi_v);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// tanh of two pre-activations, rounded to FP16 first, as one packed
// half2 tanh.approx (the activations feed the next MMA as FP16 anyway).
__device__ __forceinline__ uint32_t tanh_h2(float lo_v, float hi_v) {
  uint32_t x = pack_h2(lo_v, hi_v), y;
  asm("tanh.approx.f16x2 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}

// A lane's share of the network for mma.sync m16n8k16: the B fragments of
// the three layers and the biases of the output columns it holds (g = lane
// / 4 selects the row of B, t = lane % 4 the column pair).  Loaded once per
// warp, kept in registers.
struct Frags {
  uint32_t w1[4][3][2];  // layer 1: n-tile, k-step, (k 2t, k 2t+8)
  uint32_t w2[4][2][2];  // layer 2
  uint32_t w3[2][2];     // layer 3 (n-tile 0)
  float b1[4][2], b2[4][2], b3[2];
};

__device__ __forceinline__ void load_frags(const NetHalf *__restrict__ N, Frags &F) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t *w1 = reinterpret_cast<const uint32_t *>(N->w1);
  const uint32_t *w2 = reinterpret_cast<const uint32_t *>(N->w2);
  const uint32_t *w3 = reinterpret_cast<const uint32_t *>(N->w3);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int ks = 0; ks < 3; ++ks) {
      const int o = ((8 * nt + g) * kK1 + 16 * ks + 2 * t) / 2;
      F.w1[nt][ks][0] = w1[o];
      F.w1[nt][ks][1] = w1[o + 4];
    }
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) {
      const int o = ((8 * nt + g) * kHid + 16 * kt + 2 * t) / 2;
      F.w2[nt][kt][0] = w2[o];
      F.w2[nt][kt][1] = w2[o + 4];
    }
    F.b1[nt][0] = N->b1[8 * nt + 2 * t];
    F.b1[nt][1] = N->b1[8 * nt + 2 * t + 1];
    F.b2[nt][0] = N->b2[8 * nt + 2 * t];
    F.b2[nt][1] = N->b2[8 * nt + 2 * t + 1];
  }
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) {
    const int o = (g * kHid + 16 * kt + 2 * t) / 2;
    F.w3[kt][0] = w3[o];
    F.w3[kt][1] = w3[o + 4];
  }
  F.b3[0] = N->b3[2 * t];
  F.b3[1] = N->b3[2 * t + 1];
}

// The network on the warp's 16-row feature tile Xs (FP16, row stride kXs).
// Lanes with (lane & 3) == 0 return the outputs of rows lane/4 and lane/4+8.
__device__ __forceinline__ void mlp16(const __half *Xs, const Frags &F, float (&y_lo)[2], float (&y_hi)[2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint32_t a[3][4];
#pragma unroll
  for (int ks = 0; ks < 3; ++ks) {
    a[ks][0] = *reinterpret_cast<const uint32_t *>(Xs + g * kXs + 16 * ks + 2 * t);
    a[ks][1] = *reinterpret_cast<const uint32_t *>(Xs + (g + 8) * kXs + 16 * ks + 2 * t);
    a[ks][2] = *reinterpret_cast<const uint32_t *>(Xs + g * kXs + 16 * ks + 2 * t + 8);
    a[ks][3] = *reinterpret_cast<const uint32_t *>(Xs + (g + 8) * kXs + 16 * ks + 2 * t + 8);
  }
  float h[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    h[nt][0] = F.b1[nt][0]; h[nt][1] = F.b1[nt][1]; h[nt][2] = F.b1[nt][0]; h[nt][3] = F.b1[nt][1];
#pragma unroll
    for (int ks = 0; ks < 3; ++ks) mma16816(h[nt], a[ks], F.w1[nt][ks][0], F.w1[nt][ks][1]);
  }
  uint32_t a2[2][4];
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) {
    a2[kt][0] = tanh_h2(h[2 * kt][0], h[2 * kt][1]);
    a2[kt][1] = tanh_h2(h[2 * kt][2], h[2 * kt][3]);
    a2[kt][2] = tanh_h2(h[2 * kt + 1][0], h[2 * kt + 1][1]);
    a2[kt][3] = tanh_h2(h[2 * kt + 1][2], h[2 * kt + 1][3]);
  }
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    h[nt][0] = F.b2[nt][0]; h[nt][1] = F.b2[nt][1]; h[nt][2] = F.b2[nt][0]; h[nt][3] = F.b2[nt][1];
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) mma16816(h[nt], a2[kt], F.w2[nt][kt][0], F.w2[nt][kt][1]);
  }
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) {
    a2[kt][0] = tanh_h2(h[2 * kt][0], h[2 * kt][1]);
    a2[kt][1] = tanh_h2(h[2 * kt][2], h[2 * kt][3]);
    a2[kt][2] = tanh_h2(h[2 * kt + 1][0], h[2 * kt + 1][1]);
    a2[kt][3] = tanh_h2(h[2 * kt + 1][2], h[2 * kt + 1][3]);
  }
  float o[4] = {F.b3[0], F.b3[1], F.b3[0], F.b3[1]};
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) mma16816(o, a2[kt], F.w3[kt][0], F.w3[kt][1]);
  y_lo[0] = o[0];
  y_lo[1] = o[1];
  y_hi[0] = o[2];
  y_hi[1] = o[3];
}

// The same fragments in shared memory, lane-minor with a lane's two words
// side by side ([..][lane][2]: one 8-byte load per MMA operand or bias
// pair, a warp's 32 lanes reading 256 consecutive bytes, no bank conflict),
// for the boundary kernel: there the 62 registers of Frags would hold the
// SM to 16 warps.
struct FragsSmem {
  uint2 w1[4][3][32];
  uint2 w2[4][2][32];
  uint2 w3[2][32];
  float2 b1[4][32], b2[4][32], b3[32];
};

// Fills S from the network, warp 0 writing its lanes' fragments.
__device__ __forceinline__ void frags_to_smem(const NetHalf *__restrict__ N, FragsSmem &S) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  Frags F;
  load_frags(N, F);
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
#pragma unroll
    for (int ks = 0; ks < 3; ++ks) S.w1[nt][ks][lane] = make_uint2(F.w1[nt][ks][0], F.w1[nt][ks][1]);
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) S.w2[nt][kt][lane] = make_uint2(F.w2[nt][kt][0], F.w2[nt][kt][1]);
    S.b1[nt][lane] = make_float2(F.b1[nt][0], F.b1[nt][1]);
    S.b2[nt][lane] = make_float2(F.b2[nt][0], F.b2[nt][1]);
  }
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) S.w3[kt][lane] = make_uint2(F.w3[kt][0], F.w3[kt][1]);
  S.b3[lane] = make_float2(F.b3[0], F.b3[1]);
}

// mlp16 with the B fragments and biases read from shared memory.
__device__ __forceinline__ void mlp16_smem(const __half *Xs, const FragsSmem &S, float (&y_lo)[2],
                                           float (&y_hi)[2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint32_t a[3][4];
#pragma unroll
  for (int ks = 0; ks < 3; ++ks) {
    a[ks][0] = *reinterpret_cast<const uint32_t *>(Xs + g * kXs + 16 * ks + 2 * t);
    a[ks][1] = *reinterpret_cast<const uint32_t *>(Xs + (g + 8) * kXs + 16 * ks + 2 * t);
    a[ks][2] = *reinterpret_cast<const uint32_t *>(Xs + g * kXs + 16 * ks + 2 * t + 8);
    a[ks][3] = *reinterpret_cast<const uint32_t *>(Xs + (g + 8) * kXs + 16 * ks + 2 * t + 8);
  }
  float h[4][4];
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const float2 c = S.b1[nt][lane];
    h[nt][0] = c.x; h[nt][1] = c.y; h[nt][2] = c.x; h[nt][3] = c.y;
#pragma unroll
    for (int ks = 0; ks < 3; ++ks) {
      const uint2 w = S.w1[nt][ks][lane];
      mma16816(h[nt], a[ks], w.x, w.y);
    }
  }
  uint32_t a2[2][4];
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) {
    a2[kt][0] = tanh_h2(h[2 * kt][0], h[2 * kt][1]);
    a2[kt][1] = tanh_h2(h[2 * kt][2], h[2 * kt][3]);
    a2[kt][2] = tanh_h2(h[2 * kt + 1][0], h[2 * kt + 1][1]);
    a2[kt][3] = tanh_h2(h[2 * kt + 1][2], h[2 * kt + 1][3]);
  }
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const float2 c = S.b2[nt][lane];
    h[nt][0] = c.x; h[nt][1] = c.y; h[nt][2] = c.x; h[nt][3] = c.y;
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) {
      const uint2 w = S.w2[nt][kt][lane];
      mma16816(h[nt], a2[kt], w.x, w.y);
    }
  }
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) {
    a2[kt][0] = tanh_h2(h[2 * kt][0], h[2 * kt][1]);
    a2[kt][1] = tanh_h2(h[2 * kt][2], h[2 * kt][3]);
    a2[kt][2] = tanh_h2(h[2 * kt + 1][0], h[2 * kt + 1][1]);
    a2[kt][3] = tanh_h2(h[2 * kt + 1][2], h[2 * kt + 1][3]);
  }
  const float2 ob = S.b3[lane];
  float o[4] = {ob.x, ob.y, ob.x, ob.y};
#pragma unroll
  for (int kt = 0; kt < 2; ++kt) {
    const uint2 w = S.w3[kt][lane];
    mma16816(o, a2[kt], w.x, w.y);
  }
  y_lo[0] = o[0];
  y_lo[1] = o[1];
  y_hi[0] = o[2];
  y_hi[1] = o[3];
}

constexpr int kInferWarps = 4;

__device__ __forceinline__ float sigmoid(float y) { return 1.0f / (1.0f + __expf(-y)); }

// The network on given features (rows of 40 floats), raw outputs.  Bound by the
// latency of one tile a warp: with scalar feature reads and 8 warps a block it
// took 13.8 us for 8192 rows, with float4 reads and 4 warps a block 4.2 us.
__global__ void __launch_bounds__(32 * kInferWarps) k_abc_forward(const float *feat, long n, const NetHalf *net,
                                                                   float *out) {
  __shared__ __align__(16) __half Xs[kInferWarps][16 * kXs];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Frags F;
  load_frags(net, F);
  __half *X = Xs[warp];
  const long ntiles = (n + 15) / 16;
  for (long tile = blockIdx.x * (long)kInferWarps + warp; tile < ntiles; tile += (long)gridDim.x * kInferWarps) {
    // 16 rows of ten float4 (five a lane), K padded with zeros.
#pragma unroll
    for (int e = lane; e < 16 * (kIn / 4); e += 32) {
      const int r = e / (kIn / 4), k = 4 * (e % (kIn / 4));
      const long row = tile * 16 + r;
      const float4 v =
          row < n ? *reinterpret_cast<const float4 *>(feat + row * kIn + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<uint2 *>(X + r * kXs + k) = make_uint2(pack_h2(v.x, v.y), pack_h2(v.z, v.w));
    }
    if (lane < 16) *reinterpret_cast<uint4 *>(X + lane * kXs + kIn) = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    float ylo[2], yhi[2];
    mlp16(X, F, ylo, yhi);
    const int g = lane >> 2;
    if ((lane & 3) == 0) {
      const long c0 = tile * 16 + g, c1 = tile * 16 + g + 8;
      if (c0 < n) {
        out[c0 * 2] = ylo[0];
        out[c0 * 2 + 1] = ylo[1];
      }
      if (c1 < n) {
        out[c1 * 2] = yhi[0];
        out[c1 * 2 + 1] = yhi[1];
      }
    }
    __syncwarp();
  }
}

// One face pair's rays: [r0, rmid) on the low face, [rmid, r1) on the high one,
// each face in ghost-cell order (first transverse coordinate fastest, e0 of
// them).  lo and hi are the field indexes of cell d = L-3 of the faces' first
// rays, su and sv the index steps of the transverse coordinates, sn that along
// the normal.  Counts and indexes fit 32 bits (the field has fewer than 2^31
// cells, and a face pair's rays are at most 2/19 of them).  The kernels read
// it from their arguments: derived there, it holds ten registers.
struct Pass {
  int r0, rmid, r1, e0, lo, hi, su, sv, sn;
  unsigned inv;  // ceil(2^32 / e0)
};

Pass pass_of(const Ghost &G, int A, int sy, int pitch) {
  const int fa = 2 * (2 - A);  // the low face; fa + 1 is the high one
  const int t0 = A == 0 ? 1 : 0, t1 = A == 2 ? 1 : 2;
  const int plane = sy * pitch, d = G.L - kGhostD + 1;
  Pass P;
  P.r0 = (int)(G.off[fa] / kGhostD);
  P.rmid = (int)(G.off[fa + 1] / kGhostD);
  P.r1 = (int)(G.off[fa + 2] / kGhostD);
  P.e0 = G.keep.hi[t0] - G.keep.lo[t0];
  P.inv = 0xffffffffu / (unsigned)P.e0 + 1u;
  P.sn = A == 0 ? 1 : (A == 1 ? pitch : plane);
  P.su = A == 0 ? pitch : 1;
  P.sv = A == 2 ? pitch : plane;
  const int first = G.keep.lo[t0] * P.su + G.keep.lo[t1] * P.sv;
  P.lo = first + (G.in.lo[A] - d) * P.sn;
  P.hi = first + (G.in.hi[A] - 1 + d) * P.sn;
  return P;
}

// ---- the boundary step: one cooperative launch after the plain step -----------
//
// Two kernels, one launch per step: k_abc_boundary on the steps where the
// learned form evaluates its network, k_abc_rays_coop on the other steps and
// for the medium's fixed coefficients.  Both run the face pairs normal to z,
// then y, then x, with a bounded grid-wide barrier between them (a pass
// reads the next values the previous pass wrote at edge cells).
//
// k_abc_boundary: every warp takes groups of 4 consecutive rays (16 ghost
// cells):
//  1. lane 8 r + q loads point q (d = L-7+q) of ray r's outward normal line
//     at t from the current field and at t-1 from the line buffer the
//     previous launch filled; it stores the t line when the next step
//     evaluates the network too;
//  2. the 16 cells' features and the network on the tensor cores
//     (mma.sync m16n8k16), two lanes per cell building the t and t-1
//     stencils; k = sigmoid(y) stays in registers (it is written to the
//     coefficient buffer only when later steps reuse it);
//  3. lanes 4 r + j (j = 0..3: d = L-3+j) apply the box-scheme update
//     next_g = cur_i + k (cur_g - next_i) outward along ray r, an inclusive
//     scan of affine maps over the ray's 4 lanes.
// The line buffer replaces the read of the t-1 field, which the plain step
// has overwritten by the time this kernel runs.
struct BoundaryArgs {
  Pass pass[3];             // face pair normal to axis A
  int L;
  const float2 *cur;        // field at t
  float2 *next;             // field at t+1 (the plain step's result)
  const float4 *med;        // per ghost cell: vpz, epsilon, delta, field index (int bits)
  const NetHalf *net;
  const float2 *line_in;    // per ray: the 8 line points at t-1 (learned form)
  float2 *line_out;         // per ray: the 8 line points at t, for the next launch (learned form)
  float2 *k;                // per ghost cell: (k_p, k_q), read unless the network runs, written when it is kept
  int eval;                 // the network runs at this step
  int keep;                 // store the network's k for the steps that reuse it
  int save;                 // store the t lines (the next step evaluates the network)
  unsigned *bar;            // grid barrier: arrival count, generation
  unsigned *err;            // error word (bit 0: a bounded wait gave up)
  unsigned long long wait_ns;
};

constexpr int kBoundaryWarps = 8;
constexpr int kBoundaryBlocks = 4;  // resident blocks of either kernel per SM (at most 64 registers)

// Field index of cell d = L-3 of ray `ray` and the index step one cell
// outward.  The coordinates come from the ray index alone, so the field loads
// do not wait for a table lookup; the quotient by e0 is a multiplication by
// its rounded-up inverse, at most one too large, and a correction.
__device__ __forceinline__ int ray_cell(const Pass &P, int ray, int &step) {
  const bool high = ray >= P.rmid;
  const int rs = ray - (high ? P.rmid : P.r0);
  int v = (int)__umulhi((unsigned)rs, P.inv), u = rs - v * P.e0;
  if (u < 0) {
    u += P.e0;
    --v;
  }
  step = high ? P.sn : -P.sn;
  return (high ? P.hi : P.lo) + u * P.su + v * P.sv;
}

// Grid-wide barrier of a cooperative launch (every block is resident),
// bounded: false when the other blocks have not all arrived within limit_ns
// (bit 0 of the error word is then set).
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned nblocks, uint64_t limit_ns, unsigned *err) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    volatile unsigned *gen = bar + 1;
    const unsigned g0 = *gen;
    __threadfence();
    int ok = 1;
    if (atomicAdd(bar, 1u) == nblocks - 1) {
      atomicExch(bar, 0u);
      __threadfence();
      atomicAdd(bar + 1, 1u);
    } else {
      const uint64_t t0 = global_ns();
      while (*gen == g0) {
        if (global_ns() - t0 > limit_ns) {
          ok = 0;
          atomicOr(err, 1u);
          break;
        }
        __nanosleep(100);
      }
    }
    __threadfence();
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// What bounds it: issue slots (half of them used) and the chain of a group,
// lines to features to network to scan: about 550 instructions, a third of them
// the network.  256^3 (393 000 rays): 110 us with the cells' coordinates divided
// out twice a group in 64 bits and 24 warps an SM, 97 us without, 92 us with 32
// warps.
__global__ void __launch_bounds__(32 * kBoundaryWarps, kBoundaryBlocks) k_abc_boundary(const __grid_constant__ BoundaryArgs B) {
  __shared__ __align__(16) __half Xs[kBoundaryWarps][16 * kXs];
  // Lines [time: t, t-1][ray][point] (p, q).  The points past the layer stay
  // zero; strides of 12 and 56 let 16 lanes' stencil reads (2 rays, 2 times,
  // 4 cells) fall into 16 different bank pairs.
  constexpr int kLr = 12, kLt = 56;
  __shared__ float2 Ln[kBoundaryWarps][2 * kLt];
  __shared__ FragsSmem F;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  frags_to_smem(B.net, F);
  for (int i = lane; i < 2 * kLt; i += 32) Ln[warp][i] = make_float2(0.f, 0.f);
  if (lane < 16) *reinterpret_cast<uint4 *>(Xs[warp] + lane * kXs + kIn) = make_uint4(0u, 0u, 0u, 0u);  // K padding
  __syncthreads();
  const int wg = (int)blockIdx.x * kBoundaryWarps + warp, nw = (int)gridDim.x * kBoundaryWarps;
  // A group's loads (lane 8 r + q: point q of ray r at t and t-1; lane 2 c + h:
  // the medium of cell c), issued a group ahead of their use, a pass's first
  // ones before the barrier that it begins with.
  float2 pa, pb, pn;
  float4 pm;
  int pidx, pstep;  // cell d = L-3 of lane 8 r + q's ray and the step outward
  int A = 2;  // the pass of the loads and of the update (the loads' is one ahead at a barrier)
  auto load_group = [&](int grp) {
    const int ray0 = B.pass[A].r0 + 4 * grp, ray = ray0 + (lane >> 3);
    const int q = lane & 7, c = lane >> 1;
    pa = pb = make_float2(0.f, 0.f);
    pm = make_float4(0.f, 0.f, 0.f, 0.f);
    pidx = pstep = 0;
    if (grp >= (B.pass[A].r1 - B.pass[A].r0 + 3) / 4) return;
    if (ray < B.pass[A].r1) {
      pidx = ray_cell(B.pass[A], ray, pstep);  // point 4
      pa = __ldcg(B.cur + pidx + (q - kGhostD) * pstep);
      pb = __ldcg(B.line_in + (size_t)ray * 8 + q);
    }
    if (ray0 + (c >> 2) < B.pass[A].r1) pm = B.med[(size_t)ray0 * kGhostD + c];
  };
  // Lane 8 r + 3 also loads next at d = L-4, the value the update of ray r
  // starts from (no cell a pass writes: it is final when the pass begins).
  auto load_next = [&] {
    pn = make_float2(0.f, 0.f);
    if ((lane & 7) == kGhostD - 1 && pstep) pn = __ldcg(B.next + pidx - pstep);
  };
  load_group(wg);
  for (;;) {
    load_next();
    const int ngroups = (B.pass[A].r1 - B.pass[A].r0 + 3) / 4;
    for (int grp = wg; grp < ngroups; grp += nw) {
      const int ray0 = B.pass[A].r0 + 4 * grp, r1 = B.pass[A].r1;
      // 1. the rays' lines into shared memory, the t line kept for the next
      //    step when it evaluates too; then the next group's loads.
      const float4 m = pm;
      const float2 nq = pn;
      const int cidx = pidx, cstep = pstep;
      {
        const int r = lane >> 3, q = lane & 7;
        const int ray = ray0 + r;
        if (B.save && ray < r1) __stcg(B.line_out + (size_t)ray * 8 + q, pa);
        Ln[warp][r * kLr + q] = pa;
        Ln[warp][kLt + r * kLr + q] = pb;
      }
      load_group(grp + nw);
      load_next();
      __syncwarp();
      // 2. the coefficient of update lane u = 4 r + j (cell 4 r + j of the group).
      const int u = lane & 15;
      const bool live = lane < 16 && ray0 + (u >> 2) < r1;
      float2 kc;
      {
        // Features of cell c = lane / 2 (ray c / 4, d = L-3 + c % 4); the
        // lane pair builds the t (even lane) and t-1 (odd lane) stencils,
        // line points j .. j+8 (zero for a ray past the last).
        const int c = lane >> 1, half_t = lane & 1, j = c & 3;
        const float2 *line = Ln[warp] + half_t * kLt + (c >> 2) * kLr + j;
        float vv[18];
#pragma unroll
        for (int o = 0; o < 9; ++o) {
          const float2 v = line[o];
          vv[o] = v.x;
          vv[9 + o] = v.y;
        }
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 18; ++k) s = fmaxf(s, fabsf(vv[k]));
        s = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, 1));
        // Stencils this small carry no wave (the first cells a front reaches
        // hold values near the FP32 underflow, whose reciprocal overflows).
        if (!(s > kMinScale)) s = 0.f;
        const float inv = s > 0.f ? 1.0f / s : 0.f;
        __half *X = Xs[warp];
        __half *row = X + c * kXs + 18 * half_t;
#pragma unroll
        for (int k = 0; k < 18; k += 2)
          *reinterpret_cast<__half2 *>(row + k) = __floats2half2_rn(vv[k] * inv, vv[k + 1] * inv);
        if (half_t == 0) {
          const int d = B.L - kGhostD + 1 + j;
          *reinterpret_cast<__half2 *>(X + c * kXs + 36) = __floats2half2_rn(m.x * kVScale, m.y);
          *reinterpret_cast<__half2 *>(X + c * kXs + 38) = __floats2half2_rn(m.z, (float)d / (float)B.L);
        }
        __syncwarp();
        float ylo[2], yhi[2];
        mlp16_smem(X, F, ylo, yhi);
        // Rows g and g + 8 sit in lane 4 g: cell u comes from lane 4 (u % 8).
        const int src = 4 * (u & 7);
        const float a0 = __shfl_sync(0xffffffffu, ylo[0], src), a1 = __shfl_sync(0xffffffffu, ylo[1], src);
        const float b0 = __shfl_sync(0xffffffffu, yhi[0], src), b1 = __shfl_sync(0xffffffffu, yhi[1], src);
        kc = u < 8 ? make_float2(sigmoid(a0), sigmoid(a1)) : make_float2(sigmoid(b0), sigmoid(b1));
        if (B.keep && live) B.k[(size_t)ray0 * kGhostD + u] = kc;
      }
      // 3. the update along each ray (lanes 0 .. 15).
      const int r = u >> 2, j = u & 3;
      const float2 cg = Ln[warp][r * kLr + kGhostD + j];      // the cell at t
      const float2 ci = Ln[warp][r * kLr + kGhostD - 1 + j];  // its inward neighbour at t
      const int gidx = __shfl_sync(0xffffffffu, cidx, 8 * r) + j * __shfl_sync(0xffffffffu, cstep, 8 * r);
      float2 ni = make_float2(0.f, 0.f);
      {
        // next of d = L-4, loaded a group ahead by lane 8 r + 3.
        const float nx = __shfl_sync(0xffffffffu, nq.x, 8 * r + kGhostD - 1);
        const float ny = __shfl_sync(0xffffffffu, nq.y, 8 * r + kGhostD - 1);
        if (j == 0) ni = make_float2(nx, ny);
      }
      // a_d = cur_(d-1) + k_d cur_d, next_d = a_d - k_d next_(d-1): lane j
      // folds in lanes j-1 .. 0 of its ray (the first one brings next_(L-4)).
      float ax = __fmaf_rn(kc.x, cg.x, ci.x), ay = __fmaf_rn(kc.y, cg.y, ci.y);
      float mx = -kc.x, my = -kc.y;  // coefficient of next_(start-1) in the running value
      if (j == 0) {
        ax = __fmaf_rn(mx, ni.x, ax);
        ay = __fmaf_rn(my, ni.y, ay);
        mx = 0.f;
        my = 0.f;
      }
#pragma unroll
      for (int o = 1; o < kGhostD; o <<= 1) {
        const float px = __shfl_up_sync(0xffffffffu, ax, o), py = __shfl_up_sync(0xffffffffu, ay, o);
        const float qx = __shfl_up_sync(0xffffffffu, mx, o), qy = __shfl_up_sync(0xffffffffu, my, o);
        if (j >= o) {
          // value = a + m * (previous value) with the previous one = p + q * (...)
          ax = __fmaf_rn(mx, px, ax);
          ay = __fmaf_rn(my, py, ay);
          mx *= qx;
          my *= qy;
        }
      }
      if (live) __stcg(B.next + gidx, make_float2(ax, ay));
      __syncwarp();
    }
    if (A == 0) break;
    --A;
    load_group(wg);
    if (!grid_barrier(B.bar, gridDim.x, B.wait_ns, B.err)) return;
  }
}

// k_abc_rays_coop: the update with coefficients from the buffer (the
// medium's, or the network's from its last evaluation), four lanes per ray
// (j = 0..3: d = L-3+j), eight rays per warp.  Each lane loads its cell's
// coefficient and value at t, the lane of d = L-3 also the inward
// neighbour's values at t and t+1; the outward dependence is an inclusive
// scan of affine maps over the ray's 4 lanes.  SAVE: the step before an
// evaluation also stores the rays' 8 line points at t (lane j: points j
// and j+4), which the evaluating step reads as its t-1 lines.
// What bounds it: the latency of its three passes, one round of loads each up
// to 155 000 rays a pass; all loads but next's are therefore issued before the
// barrier that the pass begins with (256^3: 26 -> 24 us, SAVE 31 -> 27 us).
template <bool SAVE>
__global__ void __launch_bounds__(256, kBoundaryBlocks) k_abc_rays_coop(const __grid_constant__ BoundaryArgs B) {
  const int lane = threadIdx.x & 31, j = lane & 3;
  const int tid = (int)(blockIdx.x * blockDim.x + threadIdx.x), nth = (int)(gridDim.x * blockDim.x);
  // kU cells per thread and iteration, all their loads issued before any
  // of them is used (whether a cell lies below `total` is the same for
  // every lane of a warp, so the shuffles below see whole warps).
  constexpr int kU = 4;
  float2 kk[kU], cg[kU], ci[kU], ni[kU];
  int gidx[kU], step[kU];  // step 0: no cell
  int A = 2;  // the pass of the loads and of the update (the loads' is one ahead at a barrier)
  auto load = [&](int t0, int total) {
#pragma unroll
    for (int w = 0; w < kU; ++w) {
      const int t = t0 + w * nth;
      const int ray = B.pass[A].r0 + (t >> 2);
      kk[w] = cg[w] = ci[w] = make_float2(0.f, 0.f);
      gidx[w] = step[w] = 0;
      if (t < total && ray < B.pass[A].r1) {
        kk[w] = B.k[(size_t)ray * kGhostD + j];
        const int idx = ray_cell(B.pass[A], ray, step[w]);
        gidx[w] = idx + j * step[w];
        cg[w] = __ldcg(B.cur + gidx[w]);
        // Line point j (d = L-7+j) when saving, else lane 0's inward cell.
        if (SAVE) ci[w] = __ldcg(B.cur + gidx[w] - kGhostD * step[w]);
        else if (j == 0) ci[w] = __ldcg(B.cur + gidx[w] - step[w]);
      }
    }
  };
  auto cells = [&] { return ((B.pass[A].r1 - B.pass[A].r0) * kGhostD + 31) / 32 * 32; };  // whole warps iterate together
  int total = cells();
  load(tid, total);
  for (;;) {
    for (int t0 = tid; t0 < total; t0 += kU * nth) {
      if (t0 != tid) load(t0, total);
#pragma unroll
      for (int w = 0; w < kU; ++w) {
        ni[w] = make_float2(0.f, 0.f);
        if (j == 0 && step[w]) ni[w] = __ldcg(B.next + gidx[w] - step[w]);  // next of d = L-4
      }
      if (SAVE) {
#pragma unroll
        for (int w = 0; w < kU; ++w)
          if (step[w]) {
            float2 *line = B.line_out + (size_t)(B.pass[A].r0 + ((t0 + w * nth) >> 2)) * 8 + j;
            __stcg(line, ci[w]);
            __stcg(line + kGhostD, cg[w]);
          }
      }
#pragma unroll
      for (int w = 0; w < kU; ++w) {
        if (t0 - lane + w * nth >= total) break;  // the warp's first cell (uniform)
        // The inward cell of lanes 1 .. 3 is the cell of the lane before; that
        // of lane 0 is line point 3, which lane 3 loaded when saving.
        {
          const float ux = __shfl_up_sync(0xffffffffu, cg[w].x, 1), uy = __shfl_up_sync(0xffffffffu, cg[w].y, 1);
          const float fx = __shfl_sync(0xffffffffu, ci[w].x, lane | 3);
          const float fy = __shfl_sync(0xffffffffu, ci[w].y, lane | 3);
          if (j != 0) ci[w] = make_float2(ux, uy);
          else if (SAVE) ci[w] = make_float2(fx, fy);
        }
        float ax = __fmaf_rn(kk[w].x, cg[w].x, ci[w].x), ay = __fmaf_rn(kk[w].y, cg[w].y, ci[w].y);
        float mx = -kk[w].x, my = -kk[w].y;
        if (j == 0) {
          ax = __fmaf_rn(mx, ni[w].x, ax);
          ay = __fmaf_rn(my, ni[w].y, ay);
          mx = 0.f;
          my = 0.f;
        }
#pragma unroll
        for (int o = 1; o < kGhostD; o <<= 1) {
          const float px = __shfl_up_sync(0xffffffffu, ax, o), py = __shfl_up_sync(0xffffffffu, ay, o);
          const float qx = __shfl_up_sync(0xffffffffu, mx, o), qy = __shfl_up_sync(0xffffffffu, my, o);
          if (j >= o) {
            ax = __fmaf_rn(mx, px, ax);
            ay = __fmaf_rn(my, py, ay);
            mx *= qx;
            my *= qy;
          }
        }
        if (step[w]) __stcg(B.next + gidx[w], make_float2(ax, ay));
      }
    }
    if (A == 0) break;
    --A;
    total = cells();
    load(tid, total);
    if (!grid_barrier(B.bar, gridDim.x, B.wait_ns, B.err)) return;
  }
}

// The t-1 line points of every ray from the previous field, before the
// first boundary step (later steps carry them over themselves).
__global__ void k_abc_lines(const __grid_constant__ Ghost G, const float2 *__restrict__ prev, int sy, int pitch,
                            const float4 *__restrict__ med, float2 *__restrict__ lines) {
  const long nrays = G.off[6] / kGhostD;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < nrays * 8; i += (long)gridDim.x * blockDim.x) {
    const long ray = i >> 3;
    const int q = (int)(i & 7);
    const int f = face_of(G, ray * kGhostD);
    const int idx0 = __float_as_int(med[ray * kGhostD].w);
    lines[i] = prev[idx0 + (q - kGhostD) * normal_step(f, sy, pitch)];
  }
}

// Taper of the layer cells after the step: next *= exp(-(damping d)^2).
__global__ void k_abc_taper(const LayerCell *cells, long ncells, float2 *next, int sy, int pitch, float damping) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < ncells; i += (long)gridDim.x * blockDim.x) {
    const LayerCell c = cells[i];
    float2 *p = next + cell_index(c.x, c.y, c.z, sy, pitch);
    const float a = damping * (float)c.d;
    const float w = __expf(-a * a);
    float2 v = *p;
    v.x *= w;
    v.y *= w;
    *p = v;
  }
}

// Medium of every ghost cell (inputs of the network) with the cell's index
// in the field in .w (as int bits), and the medium's one-way coefficients.
__global__ void k_abc_fill(const __grid_constant__ Ghost G, const float *coef, int sy, int pitch, float dt, float hx, float hy, float hz,
                           float4 *med, float2 *kfix) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < G.off[6]; i += (long)gridDim.x * blockDim.x) {
    int c[3], f, a, sgn;
    ghost_cell(G, i, c, f, a, sgn);
    float4 m = medium_of(coef, c[0], c[1], c[2], sy, pitch);
    m.w = __int_as_float((int)cell_index(c[0], c[1], c[2], sy, pitch));
    med[i] = m;
    if (kfix) {
      const float kf = oneway_k(m.x, m.y, a, dt, a == 0 ? hx : (a == 1 ? hy : hz));
      kfix[i] = make_float2(kf, kf);
    }
  }
}

// ---- training -------------------------------------------------------------------

// A training block: kTB samples with kTG threads each, which take the outputs
// of a layer in kTG equal parts.  64 samples a block rather than 128 give
// 8192 samples 128 blocks (of 152 SMs).  Two blocks, a cluster, write one set of
// sums: the allocator hands out 2 MB at a time, and a call whose memory crosses
// that takes 0.1 ms more (with a set a block, 6528 to 8100 samples took 220
// instead of 112 us).
constexpr int kTB = 64, kTG = 4, kTT = kTB * kTG;
constexpr int kTO = kHid / kTG;  // a thread's outputs of a hidden layer
// More samples than kTrainOnce blocks take run on kTrainLoop blocks, several
// chunks of kTB each; fewer take a chunk a block.  (152: the GB300's SMs, and
// fixed, so that the sums and their order are the same everywhere.)
constexpr int kCluster = 2, kTrainOnce = 208, kTrainLoop = 152;
static_assert(kTrainOnce % kCluster == 0 && kTrainLoop % kCluster == 0, "whole clusters");
static_assert(kTO % 4 == 0 && kTG >= kOut && kTB % 32 == 0, "float4 stores; an output layer's row per group of warps");
constexpr int sX = 44, sH = 36;  // row strides in floats: rows 16-byte aligned, float4 reads of 8 rows conflict-free

__device__ __forceinline__ float h16(float v) { return __half2float(__float2half_rn(v)); }

// Outputs [o0, o0 + kTO) of one sample's hidden layer: z = b[o] + sum_k W[o][k] x[k] (k ascending, W's
// rows read as broadcast float4), a = tanh of z rounded to FP16 as inference
// does for its half2 tanh; h[o] = a rounded to FP16, d[o] = 1 - a^2.
template <int K>
__device__ __forceinline__ void layer(const float *W, const float *b, const float (&x)[K], int o0, float *h,
                                      float *d) {
#pragma unroll 1
  for (int o = o0; o < o0 + kTO; o += 4) {
    float z[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      z[u] = b[o + u];
#pragma unroll
      for (int k = 0; k < K; k += 4) {
        const float4 w = *reinterpret_cast<const float4 *>(W + (o + u) * K + k);
        z[u] = fmaf(w.x, x[k], z[u]);
        z[u] = fmaf(w.y, x[k + 1], z[u]);
        z[u] = fmaf(w.z, x[k + 2], z[u]);
        z[u] = fmaf(w.w, x[k + 3], z[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) z[u] = tanhf(h16(z[u]));
    *reinterpret_cast<float4 *>(h + o) = make_float4(h16(z[0]), h16(z[1]), h16(z[2]), h16(z[3]));
    *reinterpret_cast<float4 *>(d + o) =
        make_float4(1.0f - z[0] * z[0], 1.0f - z[1] * z[1], 1.0f - z[2] * z[2], 1.0f - z[3] * z[3]);
  }
}

template <int K>
__device__ __forceinline__ void load_row(const float *row, float (&x)[K]) {
#pragma unroll
  for (int k = 0; k < K; k += 4) {
    const float4 v = *reinterpret_cast<const float4 *>(row + k);
    x[k] = v.x;
    x[k + 1] = v.y;
    x[k + 2] = v.z;
    x[k + 3] = v.w;
  }
}

// Forward and backward of B samples (index b of the batch: a random sample,
// or b itself when seed is 0): each block writes its part of the loss
// sum_c (sigmoid(y_c) a_c - b_c)^2 / (2 B) and of the gradient to its cluster's
// row of partial (the gradient, then the loss).  Weights are used FP16-rounded, hidden
// pre-activations and activations are rounded to FP16 (as inference does),
// the derivatives treat the roundings as the identity.  noise > 0 perturbs the
// stencil inputs.  What bounds it: the shared-memory reads of a sample's chain
// and of the sums; with one scalar read an operand and one thread a
// sample it took 41 us for 8192 samples; float4 reads and 4 x 4 register tiles
// of the sums brought 26 us, four threads a sample 15.7 us, 16.4 with the
// cluster's exchange.
template <bool LOOP>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kTT) k_abc_train(const float *feat, const float *tgt, long nsamp, int B,
                                                    uint32_t seed, const float *P, float noise, float *partial) {
  extern __shared__ __align__(16) float sm[];
  float *X = sm, *H1 = X + kTB * sX, *D1 = H1 + kTB * sH, *H2 = D1 + kTB * sH, *D2 = H2 + kTB * sH;
  float *W1 = D2 + kTB * sH, *W2 = W1 + kHid * kIn, *W3 = W2 + kHid * kHid;
  float *b1 = W3 + kOut * kHid, *b2 = b1 + kHid, *b3 = b2 + kHid, *DY = b3 + 4;
  __shared__ long srow[kTB];
  __shared__ float wl[kOut * kTB / 32];
  const int tid = threadIdx.x;
  for (int i = tid; i < kNP; i += kTT) {
    const float v = P[i];
    if (i < oB1) W1[i] = h16(v);
    else if (i < oW2) b1[i - oB1] = v;
    else if (i < oB2) W2[i - oW2] = h16(v);
    else if (i < oW3) b2[i - oB2] = v;
    else if (i < oB3) W3[i - oW3] = h16(v);
    else b3[i - oB3] = v;
  }
  const int smp = tid % kTB, grp = tid / kTB, o0 = grp * kTO;
  constexpr int kT1 = kHid / 4 * (kIn / 4), kT2 = kHid / 4 * (kHid / 4);  // 4 x 4 tiles of the W1 and W2 sums
  constexpr int kSums = 2 * kHid + kOut * kHid + kOut, kTS = kTT - kT1 - kT2;  // the other sums and their threads
  static_assert(kTS > 0 && kSums <= 2 * kTS, "a thread takes at most one tile or two other sums");
  const bool first = tid < kT1;
  const int nk = first ? kIn : kHid, tile = first ? tid : tid - kT1;
  const int to = 4 * (tile / (nk / 4)), tk = 4 * (tile % (nk / 4));
  float l = 0.f, gs[4][4] = {};  // sums over the block's chunks
  int chunk = blockIdx.x;
  do {
    const int b = chunk * kTB + smp;
    const bool live = b < B;
    long si = 0;
    if (live)
      si = seed ? (long)((((uint64_t)mix32(seed, (uint32_t)b) << 16) ^ mix32(seed + 1u, (uint32_t)b)) % (uint64_t)nsamp)
                : b;
    if (LOOP) __syncthreads();  // the last chunk's rows have been read
    if (tid < kTB) srow[tid] = live ? si : -1;
    __syncthreads();
    for (int e = tid; e < kTB * (kIn / 4); e += kTT) {
      const int q = e / (kIn / 4), k = 4 * (e % (kIn / 4));
      const long row = srow[q];
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      if (row >= 0) {
        const float4 v = *reinterpret_cast<const float4 *>(feat + row * kIn + k);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
        if (noise > 0.f && k < kSt) {
          // Input noise (approximately normal, from four uniforms).
          for (int w = 0; w < 4; ++w) {
            float u = 0.f;
            for (int r = 0; r < 4; ++r)
              u += (float)(mix32(seed ^ (0x51ED27u * (r + 1)), (uint32_t)((chunk * kTB + q) * kIn + k + w)) >> 8);
            f[w] += noise * 1.7320508f * (u * (1.0f / 16777216.0f) - 2.0f);
          }
        }
      }
      *reinterpret_cast<float4 *>(X + q * sX + k) = make_float4(h16(f[0]), h16(f[1]), h16(f[2]), h16(f[3]));
    }
    __syncthreads();
    // D1 and D2 hold the activations' derivatives until the backward pass.
    float *h1 = H1 + smp * sH, *d1v = D1 + smp * sH, *h2 = H2 + smp * sH, *d2v = D2 + smp * sH;
    {
      float x[kIn];
      load_row(X + smp * sX, x);
      layer<kIn>(W1, b1, x, o0, h1, d1v);
    }
    __syncthreads();
    {
      float x[kHid];
      load_row(h1, x);
      layer<kHid>(W2, b2, x, o0, h2, d2v);
    }
    __syncthreads();
    if (grp < kOut) {
      const int o = grp;
      float x[kHid];
      load_row(h2, x);
      float y = b3[o];
#pragma unroll
      for (int k = 0; k < kHid; k += 4) {
        const float4 w = *reinterpret_cast<const float4 *>(W3 + o * kHid + k);
        y = fmaf(w.x, x[k], y);
        y = fmaf(w.y, x[k + 1], y);
        y = fmaf(w.z, x[k + 2], y);
        y = fmaf(w.w, x[k + 3], y);
      }
      float g = 0.f;
      if (live) {
        const float kk = 1.0f / (1.0f + expf(-y));
        const float ta = tgt[si * kTgt + o], tb = tgt[si * kTgt + 2 + o];
        const float e = fmaf(kk, ta, -tb);
        l += e * e;
        g = e * ta * kk * (1.0f - kk);
      }
      DY[smp * 2 + o] = g / (float)B;
    }
    __syncthreads();
    const float dy0 = DY[smp * 2], dy1 = DY[smp * 2 + 1];
#pragma unroll
    for (int o = o0; o < o0 + kTO; o += 4) {
      float4 d = *reinterpret_cast<float4 *>(d2v + o);
      const float4 wa = *reinterpret_cast<const float4 *>(W3 + o), wb = *reinterpret_cast<const float4 *>(W3 + kHid + o);
      d.x *= fmaf(wb.x, dy1, wa.x * dy0);
      d.y *= fmaf(wb.y, dy1, wa.y * dy0);
      d.z *= fmaf(wb.z, dy1, wa.z * dy0);
      d.w *= fmaf(wb.w, dy1, wa.w * dy0);
      *reinterpret_cast<float4 *>(d2v + o) = d;
    }
    __syncthreads();
    {
      float g1[kTO];
#pragma unroll
      for (int k = 0; k < kTO; ++k) g1[k] = 0.f;
#pragma unroll 4
      for (int o = 0; o < kHid; o += 4) {
        const float4 d = *reinterpret_cast<const float4 *>(d2v + o);
        const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int k = 0; k < kTO; k += 4) {
            const float4 w = *reinterpret_cast<const float4 *>(W2 + (o + u) * kHid + o0 + k);
            g1[k] = fmaf(w.x, dd[u], g1[k]);
            g1[k + 1] = fmaf(w.y, dd[u], g1[k + 1]);
            g1[k + 2] = fmaf(w.z, dd[u], g1[k + 2]);
            g1[k + 3] = fmaf(w.w, dd[u], g1[k + 3]);
          }
      }
#pragma unroll
      for (int k = 0; k < kTO; k += 4) {
        float4 d = *reinterpret_cast<float4 *>(d1v + o0 + k);
        d.x *= g1[k];
        d.y *= g1[k + 1];
        d.z *= g1[k + 2];
        d.w *= g1[k + 3];
        *reinterpret_cast<float4 *>(d1v + o0 + k) = d;
      }
    }
    __syncthreads();
    if (tid < kT1 + kT2) {
      const float *D = (first ? D1 : D2) + to, *A = (first ? X : H1) + tk;
      const int sA = first ? sX : sH;
#pragma unroll 4
      for (int q = 0; q < kTB; ++q) {
        const float4 d = *reinterpret_cast<const float4 *>(D + q * sH), a = *reinterpret_cast<const float4 *>(A + q * sA);
        const float dv[4] = {d.x, d.y, d.z, d.w}, av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int w = 0; w < 4; ++w) gs[u][w] = fmaf(dv[u], av[w], gs[u][w]);
      }
    } else {
      // The biases' and W3's sums.
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const int e = tid - kT1 - kT2 + v * kTS;
        float s = gs[0][v];
        if (e < kHid) {
          for (int q = 0; q < kTB; ++q) s += D1[q * sH + e];
        } else if (e < 2 * kHid) {
          for (int q = 0; q < kTB; ++q) s += D2[q * sH + e - kHid];
        } else if (e < 2 * kHid + kOut * kHid) {
          const int o = (e - 2 * kHid) / kHid, k = e % kHid;
          for (int q = 0; q < kTB; ++q) s = fmaf(DY[q * 2 + o], H2[q * sH + k], s);
        } else if (e < kSums) {
          for (int q = 0; q < kTB; ++q) s += DY[q * 2 + e - 2 * kHid - kOut * kHid];
        }
        gs[0][v] = s;
      }
    }
  } while (LOOP && (long)(chunk += gridDim.x) * kTB < B);
  // The cluster's loss and gradient sums go to its own row (summed over the
  // clusters in order by k_abc_reduce: the result does not depend on timing).
  // The second block hands its sums to the first through that one's shared
  // memory, thread by thread, where X and H1 have been read.
  static_assert(16 * kTT + 1 <= kTB * (sX + sH), "the handed sums fit X and H1");
  if (grp < kOut) {
    for (int m = 16; m > 0; m >>= 1) l += __shfl_xor_sync(0xffffffffu, l, m);
    if ((tid & 31) == 0) wl[tid >> 5] = l;
  }
  cluster_barrier();
  float bl = 0.f;
  if (tid == 0)
    for (int w = 0; w < kOut * kTB / 32; ++w) bl += wl[w];
  const bool second = blockIdx.x & 1;
  if (second) {
    const uint32_t to0 = peer_smem_addr(sm, 0);
#pragma unroll
    for (int v = 0; v < 16; ++v) st_cluster(to0 + 4u * (v * kTT + tid), gs[v / 4][v % 4]);
    if (tid == 0) st_cluster(to0 + 4u * 16 * kTT, bl);
  }
  cluster_barrier();
  if (second) return;
#pragma unroll
  for (int v = 0; v < 16; ++v) gs[v / 4][v % 4] += sm[v * kTT + tid];
  float *out = partial + (size_t)(blockIdx.x / kCluster) * (kNP + 1);
  if (tid == 0) out[kNP] = (bl + sm[16 * kTT]) / (2.0f * (float)B);
  if (tid < kT1 + kT2) {
    float *dst = out + (first ? oW1 : oW2) + to * nk + tk;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int w = 0; w < 4; ++w) dst[u * nk + w] = gs[u][w];
  } else {
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int e = tid - kT1 - kT2 + v * kTS;
      const int at = e < kHid ? oB1 + e : e < 2 * kHid ? oB2 + e - kHid : e < 2 * kHid + kOut * kHid
                         ? oW3 + e - 2 * kHid : oB3 + e - 2 * kHid - kOut * kHid;
      if (e < kSums) out[at] = gs[0][v];
    }
  }
}

// Sums of the training clusters' partial gradients and losses, in order:
// a block takes 32 parameters, its 8 warps a contiguous eighth of the
// clusters each, added up in order (5.9 us with one thread a
// parameter, 3.7 us so, 3.0 with half as many rows).
constexpr int kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps) k_abc_reduce(const float *partial, int nparts, float *grad,
                                                                   float *loss) {
  __shared__ float part[kReduceWarps][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int e = blockIdx.x * 32 + lane;  // kNP is the loss
  const int b0 = (int)((long)nparts * w / kReduceWarps), b1 = (int)((long)nparts * (w + 1) / kReduceWarps);
  float g = 0.f;
  if (e <= kNP)
    for (int b = b0; b < b1; ++b) g += partial[(size_t)b * (kNP + 1) + e];
  part[w][lane] = g;
  __syncthreads();
  if (w == 0 && e <= kNP) {
    float s = 0.f;
    for (int v = 0; v < kReduceWarps; ++v) s += part[v][lane];
    if (e < kNP) grad[e] = s;
    else *loss = s;
  }
}
constexpr int kReduceBlocks = kNP / 32 + 1;

constexpr size_t kTrainSmem = sizeof(float) * (kNP + 2 + kTB * (sX + 4 * sH + 2));

// Adam step on the master weights; clears the gradient.
__global__ void k_abc_adam(float *P, float *grad, float *m, float *v, int n, float lr, float b1, float b2, float eps,
                           float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = grad[i];
  grad[i] = 0.f;
  const float mi = b1 * m[i] + (1.f - b1) * g, vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// FP32 master weights -> inference copy.
__global__ void k_abc_pack(const float *P, NetHalf *N) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kHid * kK1) {
    const int o = i / kK1, k = i % kK1;
    N->w1[i] = __float2half_rn(k < kIn ? P[oW1 + o * kIn + k] : 0.f);
  }
  if (i < kHid * kHid) N->w2[i] = __float2half_rn(P[oW2 + i]);
  if (i < 8 * kHid) N->w3[i] = __float2half_rn(i < kOut * kHid ? P[oW3 + i] : 0.f);
  if (i < kHid) {
    N->b1[i] = P[oB1 + i];
    N->b2[i] = P[oB2 + i];
  }
  if (i < 8) N->b3[i] = i < kOut ? P[oB3 + i] : 0.f;
}

// ---- host state -------------------------------------------------------------------

namespace {

struct Trainer {
  float *P = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;  // master weights and Adam state
  NetHalf *net = nullptr;
  bool weights = false;
  long adam_t = 0;
  float *feat = nullptr, *tgt = nullptr;
  int4 *pos = nullptr;  // grid cell, face and distance of every sample
  long nsamp = 0;       // samples held (at most cap)
  long cap = 0;
  bool reserved = false;
};

struct ResidentLayer {
  bool on = false;
  int mode = 0;
  int interval = 1;  // learned form: network every `interval` steps
  long steps = 0;    // steps since SetBoundary
  float damping = 0.f;
  Ghost G;
  float4 *med = nullptr;       // medium of every ghost cell (one-way modes)
  float2 *k = nullptr;         // one-way coefficients of every ghost cell (fixed, or the network's kept ones)
  float2 *lines[2] = {nullptr, nullptr};  // learned form: t-1 line points of every ray, by step parity
  unsigned *bar = nullptr;     // the boundary kernels' grid barrier (count, generation)
  int grid_net = 0, grid_rays = 0;  // their cooperative grids
  LayerCell *cells = nullptr;  // every layer cell (taper), z, y, x order
  long ncells = 0;
};

Trainer T;
ResidentLayer R;

int err(int code, const char *msg) { return flt_record_error(code, msg); }

#define CKA(call)                                                                                       \
  do {                                                                                                  \
    cudaError_t e_ = (call);                                                                            \
    if (e_ != cudaSuccess) {                                                                            \
      cudaGetLastError(); /* not sticky: a later launch check must not see it */                        \
      char b_[256];                                                                                     \
      snprintf(b_, sizeof(b_), "%s failed: %s", #call, cudaGetErrorString(e_));                        \
      return err(e_ == cudaErrorMemoryAllocation ? FLETCHER_ERR_NOMEM : FLETCHER_ERR_CUDA, b_);         \
    }                                                                                                   \
  } while (0)

cudaStream_t stream_of() {
  const ResidentView v = resident_view();
  return v.init ? v.stream : (cudaStream_t)FLETCHER_GetStream();
}

int ensure_trainer() {
  if (T.P) return FLETCHER_OK;
  CKA(cudaMalloc(&T.P, kNP * sizeof(float)));
  CKA(cudaMalloc(&T.grad, kNP * sizeof(float)));
  CKA(cudaMalloc(&T.m, kNP * sizeof(float)));
  CKA(cudaMalloc(&T.v, kNP * sizeof(float)));
  CKA(cudaMalloc(&T.net, sizeof(NetHalf)));
  CKA(cudaMemset(T.grad, 0, kNP * sizeof(float)));
  CKA(cudaMemset(T.m, 0, kNP * sizeof(float)));
  CKA(cudaMemset(T.v, 0, kNP * sizeof(float)));
  CKA(cudaMemset(T.net, 0, sizeof(NetHalf)));
  return FLETCHER_OK;
}

int pack_net(cudaStream_t s) {
  k_abc_pack<<<(kHid * kK1 + 255) / 256, 256, 0, s>>>(T.P, T.net);
  CKA(cudaGetLastError());
  return FLETCHER_OK;
}

uint64_t splitmix(uint64_t &x) {
  uint64_t z = (x += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

int grid_of(long n, int block) {
  long b = (n + block - 1) / block;
  return (int)(b < 1 ? 1 : (b > 4096 ? 4096 : b));
}

// Clusters that n samples take, a set of sums each.
int train_parts(int n) {
  const int chunks = (n - 1) / kTB + 1;
  return (chunks <= kTrainOnce ? chunks + kCluster - 1 : kTrainLoop) / kCluster;
}

void launch_train(const float *feat, const float *tgt, long nsamp, int B, uint32_t seed, float noise, float *partial,
                  cudaStream_t s) {
  const int blocks = train_parts(B) * kCluster;
  const auto kern = (long)blocks * kTB < B ? k_abc_train<true> : k_abc_train<false>;
  kern<<<blocks, kTT, kTrainSmem, s>>>(feat, tgt, nsamp, B, seed, T.P, noise, partial);
}

int train_attr() {
  static bool done = false;
  if (!done) {
    for (auto kern : {k_abc_train<false>, k_abc_train<true>})
      CKA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
    done = true;
  }
  return FLETCHER_OK;
}

bool oneway_mode(int mode) { return mode == FLETCHER_BOUNDARY_LEARNED || mode == FLETCHER_BOUNDARY_ONEWAY; }

}  // namespace

bool abc_active() { return R.on; }

void abc_release_resident() {
  if (R.med) cudaFree(R.med);
  if (R.k) cudaFree(R.k);
  if (R.lines[0]) cudaFree(R.lines[0]);
  if (R.lines[1]) cudaFree(R.lines[1]);
  if (R.bar) cudaFree(R.bar);
  if (R.cells) cudaFree(R.cells);
  R = ResidentLayer();
}

int g_interval = 1;  // FLETCHER_AbcSetInterval

// After the plain step: the ghost zone's one-way update (with the network
// on the learned form's evaluation steps) in one cooperative launch, then
// the taper if any.
cudaError_t abc_after_step(const ResidentView &v) {
  if (!R.on) return cudaSuccess;
  if (oneway_mode(R.mode)) {
    const bool learned = R.mode == FLETCHER_BOUNDARY_LEARNED;
    BoundaryArgs a;
    memset(&a, 0, sizeof(a));
    for (int A = 0; A < 3; ++A) a.pass[A] = pass_of(R.G, A, v.sy, v.pitch);
    a.L = R.G.L;
    a.cur = v.cur;
    a.next = v.next;
    a.med = R.med;
    a.net = T.net;
    a.line_in = R.lines[R.steps & 1];
    a.line_out = R.lines[(R.steps + 1) & 1];
    a.k = R.k;
    a.eval = learned && R.steps % R.interval == 0;        // the last coefficients stay in between
    a.keep = learned && R.interval > 1;
    a.save = learned && (R.steps + 1) % R.interval == 0;  // the next step evaluates
    a.bar = R.bar;
    a.err = v.err;
    a.wait_ns = kWaitLimitNs;
    ++R.steps;
    void *args[] = {&a};
    const void *kern = a.eval ? (const void *)k_abc_boundary
                              : (a.save ? (const void *)k_abc_rays_coop<true> : (const void *)k_abc_rays_coop<false>);
    const int grid = a.eval ? R.grid_net : R.grid_rays;
    const cudaError_t e = cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(256), args, 0, v.stream);
    if (e != cudaSuccess) return e;
  }
  if (R.damping > 0.f && R.ncells)
    k_abc_taper<<<grid_of(R.ncells, 256), 256, 0, v.stream>>>(R.cells, R.ncells, v.next, v.sy, v.pitch, R.damping);
  return cudaGetLastError();
}

}  // namespace flt

using namespace flt;

// ===== Part 4: learned absorbing boundary =========================================

extern "C" int FLETCHER_AbcSetWeights(const float *params) {
  if (!params) return err(FLETCHER_ERR_ARGS, "AbcSetWeights: bad arguments");
  if (ensure_trainer()) return FLETCHER_GetLastError();
  CKA(cudaMemcpy(T.P, params, kNP * sizeof(float), cudaMemcpyHostToDevice));
  CKA(cudaMemset(T.m, 0, kNP * sizeof(float)));
  CKA(cudaMemset(T.v, 0, kNP * sizeof(float)));
  T.adam_t = 0;
  T.weights = true;
  if (pack_net(nullptr)) return FLETCHER_GetLastError();
  CKA(cudaDeviceSynchronize());
  return FLETCHER_OK;
}

extern "C" int FLETCHER_AbcInit(unsigned seed) {
  std::vector<float> p(kNP, 0.f);
  uint64_t s = 0x1234567ull ^ ((uint64_t)seed << 20);
  auto unif = [&]() { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); };
  auto fill = [&](int off, int fan_out, int fan_in) {
    const double a = sqrt(6.0 / (fan_in + fan_out));
    for (int i = 0; i < fan_out * fan_in; ++i) p[off + i] = (float)((2.0 * unif() - 1.0) * a);
  };
  fill(oW1, kHid, kIn);
  fill(oW2, kHid, kHid);
  fill(oW3, kOut, kHid);
  for (int o = 0; o < kOut; ++o) p[oB3 + o] = kInitBias;
  return FLETCHER_AbcSetWeights(p.data());
}

extern "C" int FLETCHER_AbcGetWeights(float *params) {
  if (!T.weights) return err(FLETCHER_ERR_ARGS, "AbcGetWeights: no network");
  if (!params) return err(FLETCHER_ERR_ARGS, "AbcGetWeights: bad arguments");
  CKA(cudaDeviceSynchronize());
  CKA(cudaMemcpy(params, T.P, kNP * sizeof(float), cudaMemcpyDeviceToHost));
  return FLETCHER_OK;
}

extern "C" int FLETCHER_AbcReserve(long capacity) {
  if (capacity < 0) return err(FLETCHER_ERR_ARGS, "AbcReserve: negative capacity");
  if (T.feat) cudaFree(T.feat);
  if (T.tgt) cudaFree(T.tgt);
  if (T.pos) cudaFree(T.pos);
  T.feat = T.tgt = nullptr;
  T.pos = nullptr;
  T.nsamp = 0;
  T.reserved = true;
  T.cap = capacity;
  if (capacity) {
    CKA(cudaMalloc(&T.feat, (size_t)capacity * kIn * sizeof(float)));
    CKA(cudaMalloc(&T.tgt, (size_t)capacity * kTgt * sizeof(float)));
    CKA(cudaMalloc(&T.pos, (size_t)capacity * sizeof(int4)));
  }
  return FLETCHER_OK;
}

extern "C" long FLETCHER_AbcSamples(void) { return T.nsamp; }

extern "C" int FLETCHER_AbcCollect(const int *interior_lo, const int *interior_hi, int layer, float keep_frac,
                                   unsigned seed, float min_scale) {
  const ResidentView v = resident_view();
  if (!v.init) return err(FLETCHER_ERR_ARGS, "AbcCollect needs an FP32 resident state");
  if (!T.reserved || !T.cap) return err(FLETCHER_ERR_ARGS, "AbcCollect: call FLETCHER_AbcReserve first");
  if (!interior_lo || !interior_hi || layer < kRadius + 1)
    return err(FLETCHER_ERR_ARGS, "AbcCollect: bad box or layer");
  Box in;
  const int dims[3] = {v.sx, v.sy, v.sz};
  for (int a = 0; a < 3; ++a) {
    in.lo[a] = interior_lo[a];
    in.hi[a] = interior_hi[a];
    // The next values read 4 cells beyond the kept box; all of it must be updated grid.
    if (in.hi[a] <= in.lo[a] || in.lo[a] - layer - kRadius < v.bord || in.hi[a] + layer + kRadius > dims[a] - v.bord)
      return err(FLETCHER_ERR_ARGS, "AbcCollect: the box and its layer must lie 4 cells inside the updated region");
  }
  const Ghost G = make_ghost(in, layer);
  const long n = G.off[6];
  const int nb = (int)std::max(1L, std::min(1024L, (n + kCollectBlock - 1) / kCollectBlock));
  const long per = (n + nb - 1) / nb;
  std::vector<int> cnt(nb);
  std::vector<long> first(nb);
  int *d_cnt = nullptr;
  long *d_first = nullptr;
  CKA(cudaMalloc(&d_cnt, nb * sizeof(int)));
  CKA(cudaMalloc(&d_first, nb * sizeof(long)));
  k_abc_collect_count<<<nb, kCollectBlock, 0, v.stream>>>(v.cur, v.prev, G, v.sy, v.pitch, keep_frac, seed, min_scale,
                                                          per, d_cnt);
  CKA(cudaGetLastError());
  CKA(cudaMemcpyAsync(cnt.data(), d_cnt, nb * sizeof(int), cudaMemcpyDeviceToHost, v.stream));
  CKA(cudaStreamSynchronize(v.stream));
  long total = 0;
  for (int b = 0; b < nb; ++b) {
    first[b] = T.nsamp + total;
    total += cnt[b];
  }
  CKA(cudaMemcpyAsync(d_first, first.data(), nb * sizeof(long), cudaMemcpyHostToDevice, v.stream));
  k_abc_collect<<<nb, kCollectBlock, 0, v.stream>>>(v.cur, v.prev, v.coef, G, v.sy, v.pitch, v.dx, v.dy, v.dz, v.dt,
                                                    keep_frac, seed, min_scale, per, d_first, T.feat, T.tgt, T.pos,
                                                    T.cap);
  CKA(cudaGetLastError());
  CKA(cudaStreamSynchronize(v.stream));
  cudaFree(d_cnt);
  cudaFree(d_first);
  T.nsamp = std::min(T.cap, T.nsamp + total);
  return FLETCHER_OK;
}

extern "C" int FLETCHER_AbcGetSamples(long start, long n, float *feat, float *tgt, int *pos) {
  const long have = FLETCHER_AbcSamples();
  if (start < 0 || n < 0 || start + n > have)
    return err(FLETCHER_ERR_ARGS, "AbcGetSamples: range outside the samples");
  if (feat) CKA(cudaMemcpy(feat, T.feat + start * kIn, n * kIn * sizeof(float), cudaMemcpyDeviceToHost));
  if (tgt) CKA(cudaMemcpy(tgt, T.tgt + start * kTgt, n * kTgt * sizeof(float), cudaMemcpyDeviceToHost));
  if (pos) CKA(cudaMemcpy(pos, T.pos + start, n * sizeof(int4), cudaMemcpyDeviceToHost));
  return FLETCHER_OK;
}

extern "C" int FLETCHER_AbcTrain(int iters, int batch, float lr, unsigned seed, float noise, float *loss_out) {
  const long ns = FLETCHER_AbcSamples();
  if (ns <= 0) return err(FLETCHER_ERR_ARGS, "AbcTrain: no samples");
  if (!T.weights) return err(FLETCHER_ERR_ARGS, "AbcTrain: call FLETCHER_AbcInit or AbcSetWeights first");
  if (iters < 1 || batch < 1 || !(lr > 0.f) || !(noise >= 0.f))
    return err(FLETCHER_ERR_ARGS, "AbcTrain: bad arguments");
  cudaStream_t s = stream_of();
  if (train_attr()) return FLETCHER_GetLastError();
  const int parts = train_parts(batch);
  float *loss = nullptr, *partial = nullptr;
  CKA(cudaMalloc(&loss, iters * sizeof(float)));
  CKA(cudaMalloc(&partial, (size_t)parts * (kNP + 1) * sizeof(float)));
  const float b1 = 0.9f, b2 = 0.999f;
  for (int it = 0; it < iters; ++it) {
    uint64_t st = (uint64_t)seed * 1000003ull + (uint64_t)it;
    const uint32_t sd = (uint32_t)splitmix(st) | 1u;
    launch_train(T.feat, T.tgt, ns, batch, sd, noise, partial, s);
    k_abc_reduce<<<kReduceBlocks, 32 * kReduceWarps, 0, s>>>(partial, parts, T.grad, loss + it);
    ++T.adam_t;
    const float lr_t = lr * 0.5f * (1.0f + cosf(3.14159265f * (float)it / (float)iters));
    k_abc_adam<<<(kNP + 255) / 256, 256, 0, s>>>(T.P, T.grad, T.m, T.v, kNP, lr_t, b1, b2, 1e-8f,
                                                 1.0f - powf(b1, (float)T.adam_t), 1.0f - powf(b2, (float)T.adam_t));
  }
  CKA(cudaGetLastError());
  if (pack_net(s)) return FLETCHER_GetLastError();
  if (loss_out) CKA(cudaMemcpyAsync(loss_out, loss, iters * sizeof(float), cudaMemcpyDeviceToHost, s));
  CKA(cudaStreamSynchronize(s));
  cudaFree(loss);
  cudaFree(partial);
  return FLETCHER_OK;
}

extern "C" int FLETCHER_AbcGradient(const float *feat, const float *tgt, int n, float *grad, float *loss) {
  if (!T.weights) return err(FLETCHER_ERR_ARGS, "AbcGradient: no network");
  if (!feat || !tgt || !grad || n < 1) return err(FLETCHER_ERR_ARGS, "AbcGradient: bad arguments");
  if (train_attr()) return FLETCHER_GetLastError();
  const int parts = train_parts(n);
  // The sums, then one more row: the gradient and the loss.
  float *df = nullptr, *dt = nullptr, *partial = nullptr;
  CKA(cudaMalloc(&df, (size_t)n * kIn * sizeof(float)));
  CKA(cudaMalloc(&dt, (size_t)n * kTgt * sizeof(float)));
  CKA(cudaMalloc(&partial, (size_t)(parts + 1) * (kNP + 1) * sizeof(float)));
  float *dg = partial + (size_t)parts * (kNP + 1);
  CKA(cudaMemcpy(df, feat, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice));
  CKA(cudaMemcpy(dt, tgt, (size_t)n * kTgt * sizeof(float), cudaMemcpyHostToDevice));
  launch_train(df, dt, n, n, 0u, 0.f, partial, 0);
  k_abc_reduce<<<kReduceBlocks, 32 * kReduceWarps>>>(partial, parts, dg, dg + kNP);
  CKA(cudaGetLastError());
  CKA(cudaMemcpy(grad, dg, kNP * sizeof(float), cudaMemcpyDeviceToHost));
  if (loss) CKA(cudaMemcpy(loss, dg + kNP, sizeof(float), cudaMemcpyDeviceToHost));
  cudaFree(df);
  cudaFree(dt);
  cudaFree(partial);
  return FLETCHER_OK;
}

extern "C" size_t FLETCHER_AbcGradientBytes(int n) {
  if (n < 1) return 0;
  return sizeof(float) * ((size_t)n * (kIn + kTgt) + (size_t)(train_parts(n) + 1) * (kNP + 1));
}

extern "C" int FLETCHER_AbcForward(const float *feat, int n, float *out) {
  if (!T.weights) return err(FLETCHER_ERR_ARGS, "AbcForward: no network");
  if (!feat || !out || n < 1) return err(FLETCHER_ERR_ARGS, "AbcForward: bad arguments");
  float *df = nullptr, *dout = nullptr;
  CKA(cudaMalloc(&df, (size_t)n * kIn * sizeof(float)));
  CKA(cudaMalloc(&dout, (size_t)n * kOut * sizeof(float)));
  CKA(cudaMemcpy(df, feat, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice));
  const int grid = (int)(((n + 15) / 16 + kInferWarps - 1) / kInferWarps);
  k_abc_forward<<<grid, 32 * kInferWarps>>>(df, n, T.net, dout);
  CKA(cudaGetLastError());
  CKA(cudaMemcpy(out, dout, (size_t)n * kOut * sizeof(float), cudaMemcpyDeviceToHost));
  cudaFree(df);
  cudaFree(dout);
  return FLETCHER_OK;
}

extern "C" int FLETCHER_SetBoundary(int mode, int layer, float damping) {
  const ResidentView v = resident_view();
  if (!v.init) return err(FLETCHER_ERR_ARGS, "SetBoundary needs an initialised FP32 resident state");
  abc_release_resident();
  if (mode == FLETCHER_BOUNDARY_PLAIN) return FLETCHER_OK;
  if (mode != FLETCHER_BOUNDARY_LEARNED && mode != FLETCHER_BOUNDARY_SPONGE && mode != FLETCHER_BOUNDARY_ONEWAY)
    return err(FLETCHER_ERR_ARGS, "SetBoundary: unknown mode");
  if (mode == FLETCHER_BOUNDARY_LEARNED && !T.weights)
    return err(FLETCHER_ERR_ARGS, "SetBoundary: the learned layer needs weights");
  if (layer < kRadius + 1) return err(FLETCHER_ERR_ARGS, "SetBoundary: layer must be at least 5 cells");
  if (!(damping >= 0.f) || (mode == FLETCHER_BOUNDARY_SPONGE && !(damping > 0.f)))
    return err(FLETCHER_ERR_ARGS, "SetBoundary: damping must be >= 0 (> 0 for the sponge)");
  const int dims[3] = {v.sx, v.sy, v.sz};
  Box in, keep;
  for (int a = 0; a < 3; ++a) {
    keep.lo[a] = v.bord;
    keep.hi[a] = dims[a] - v.bord;
    in.lo[a] = v.bord + layer;
    in.hi[a] = dims[a] - v.bord - layer;
    if (in.hi[a] <= in.lo[a]) return err(FLETCHER_ERR_ARGS, "SetBoundary: no interior inside the layer");
  }
  R.G = make_ghost(in, layer);
  if ((long)v.sz * v.sy * v.pitch >= (1l << 31))
    return err(FLETCHER_ERR_ARGS, "SetBoundary: the layer needs a field of fewer than 2^31 cells");
  if (oneway_mode(mode)) {
    const long n = R.G.off[6];
    CKA(cudaMalloc(&R.med, n * sizeof(float4)));
    CKA(cudaMalloc(&R.k, n * sizeof(float2)));
    k_abc_fill<<<grid_of(n, 256), 256, 0, v.stream>>>(R.G, v.coef, v.sy, v.pitch, v.dt, v.dx, v.dy, v.dz, R.med,
                                                      R.k);
    CKA(cudaGetLastError());
    if (mode == FLETCHER_BOUNDARY_LEARNED) {
      // The first step's t-1 lines from the previous field; each boundary
      // launch then stores the t lines for the next one.
      for (int b = 0; b < 2; ++b) CKA(cudaMalloc(&R.lines[b], n * 2 * sizeof(float2)));
      k_abc_lines<<<grid_of(n * 2, 256), 256, 0, v.stream>>>(R.G, v.prev, v.sy, v.pitch, R.med, R.lines[0]);
      CKA(cudaGetLastError());
    }
    CKA(cudaMalloc(&R.bar, 2 * sizeof(unsigned)));
    CKA(cudaMemsetAsync(R.bar, 0, 2 * sizeof(unsigned), v.stream));
    // Cooperative grids: every block resident at once (the grid barrier needs it).
    const int sms = v.num_sms > 0 ? v.num_sms : 1;
    int per_sm = 0;
    CKA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_abc_boundary, 256, 0));
    if (per_sm < 1) return err(FLETCHER_ERR_CUDA, "SetBoundary: the boundary kernel fits no block on an SM");
    R.grid_net = per_sm * sms;
    int per_sm_r = 0, per_sm_s = 0;
    CKA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_r, k_abc_rays_coop<false>, 256, 0));
    CKA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_s, k_abc_rays_coop<true>, 256, 0));
    per_sm_r = std::min(std::min(per_sm_r, per_sm_s), 4);
    if (per_sm_r < 1) return err(FLETCHER_ERR_CUDA, "SetBoundary: the ray kernel fits no block on an SM");
    R.grid_rays = per_sm_r * sms;
  }
  if (damping > 0.f) {
    // Layer cells in z, y, x order (coalesced).
    std::vector<LayerCell> cells;
    for (int z = keep.lo[2]; z < keep.hi[2]; ++z)
      for (int y = keep.lo[1]; y < keep.hi[1]; ++y) {
        const bool inner = z >= in.lo[2] && z < in.hi[2] && y >= in.lo[1] && y < in.hi[1];
        for (int x = keep.lo[0]; x < keep.hi[0]; x = (inner && x == in.lo[0]) ? in.hi[0] : x + 1) {
          if (inner && x >= in.lo[0] && x < in.hi[0]) continue;
          const int c[3] = {x, y, z};
          int d = 0;
          for (int a = 0; a < 3; ++a) {
            const int lo = in.lo[a] - c[a], hi = c[a] - (in.hi[a] - 1);
            d = lo > d ? lo : d;
            d = hi > d ? hi : d;
          }
          if (d > 0) cells.push_back({x, y, z, d});
        }
      }
    R.ncells = (long)cells.size();
    CKA(cudaMalloc(&R.cells, R.ncells * sizeof(LayerCell)));
    CKA(cudaMemcpyAsync(R.cells, cells.data(), R.ncells * sizeof(LayerCell), cudaMemcpyHostToDevice, v.stream));
  }
  CKA(cudaStreamSynchronize(v.stream));
  R.mode = mode;
  R.damping = damping;
  R.interval = g_interval;
  R.steps = 0;
  R.on = true;
  return FLETCHER_OK;
}

extern "C" int FLETCHER_AbcSetInterval(int steps) {
  if (steps < 1) return err(FLETCHER_ERR_ARGS, "AbcSetInterval: steps must be >= 1");
  g_interval = steps;
  if (R.on) R.interval = steps;
  return FLETCHER_OK;
}

extern "C" long FLETCHER_AbcLayerCells(void) { return (R.on && oneway_mode(R.mode)) ? R.G.off[6] : 0; }

extern "C" void FLETCHER_AbcRelease(void) {
  abc_release_resident();
  if (T.P) cudaFree(T.P);
  if (T.grad) cudaFree(T.grad);
  if (T.m) cudaFree(T.m);
  if (T.v) cudaFree(T.v);
  if (T.net) cudaFree(T.net);
  if (T.feat) cudaFree(T.feat);
  if (T.tgt) cudaFree(T.tgt);
  if (T.pos) cudaFree(T.pos);
  T = Trainer();
}
